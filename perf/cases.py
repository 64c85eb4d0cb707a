"""The work that a user of this package has it do, as cases that can be timed: the Mega-MoE layer from one decoded token
to a long prefill in its three number formats, the stand-alone grouped, masked and dense GEMMs, the weight-gradient GEMM
and the activation quantiser. Sizes are those of this repository's benchmark and tests, or generic ones around them.

Inputs are quantised here with plain tensor expressions and made from the seed alone; ``exact`` computes the same
operation from the same inputs in 64 bits. What a number format itself rounds (the BF16 gate / up values and the FP8 or
NVFP4 activations between the two GEMMs of a layer, the BF16 output row of each slot) is part of the operation there too.
"""
import torch

import deepgemm_b200 as dg

_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
_E2M1_THRESHOLDS = (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0)  # a value on a threshold goes down
_DEV = 'cuda'


# ---------------------------------------------------------------------------------------------------------------- cases

def _moe(name, mma, tokens, experts=256, topk=8, hidden=7168, inter=2048, shared=0, fused=True):
    return dict(name=name, kind='moe', mma=mma, tokens=tokens, experts=experts, topk=topk, hidden=hidden, inter=inter,
                shared=shared, fused=fused)


def listed():
    return [
        # A few sequences being decoded on one GPU: one token each, router and quantisation inside the call.
        _moe('moe_fp8_decode_4', 'fp8xfp4', 4),
        # Decode with a full batch: every expert receives a handful of rows.
        _moe('moe_fp8_decode_256', 'fp8xfp4', 256),
        # The headline workload: 4096 tokens through a 256-expert layer.
        _moe('moe_fp8_4096', 'fp8xfp4', 4096),
        # A ragged chunk of a prefill on a smaller layer with a shared expert; the caller has quantised and routed already
        # and a few of its slots are masked.
        _moe('moe_fp8_shared_1999', 'fp8xfp4', 1999, experts=32, shared=1, fused=False),
        # Prefill of 16384 tokens in NVFP4.
        _moe('moe_nvfp4_16384', 'nvfp4xnvfp4', 16384),
        # The layer as it is trained or served without quantisation.
        _moe('moe_bf16_4096', 'bf16xbf16', 4096, experts=64, fused=False),
        # A small expert-parallel shard: four experts, 64 to 256 rows each.
        dict(name='contiguous_fp8_small', kind='contiguous', mma='fp8xfp4', groups=4, rows_lo=64, rows_hi=256, n=512, k=1024,
             psum=False),
        # Decode GEMM over 32 local experts whose row counts only the device knows.
        dict(name='masked_fp8_decode', kind='masked', mma='fp8xfp4', groups=32, max_m=256, mean=64, n=4096, k=7168),
        # A projection around the experts while decoding: few rows, a long K.
        dict(name='dense_bf16_decode', kind='dense', mma='bf16', m=128, n=7168, k=16384),
        # The same kind of projection in a prefill, in FP8, with a row count that no tile divides.
        dict(name='dense_fp8_prefill', kind='dense', mma='fp8xfp8', m=4000, n=7168, k=2048),
        # Weight gradient of an expert layer (the backward direction): accumulates into FP32 gradients.
        dict(name='kgrouped_fp8_wgrad', kind='kgrouped', mma='fp8', groups=8, mean_k=4096, m=4096, n=7168),
        # What every caller of the GEMMs runs on its activations first.
        dict(name='cast_fp8_4096', kind='cast', mma='fp8', m=4096, k=7168, gran=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(['moe', 'moe', 'moe', 'contiguous', 'masked', 'dense', 'dense', 'kgrouped', 'cast'])
    if kind == 'moe':
        mma = rng.choice(['fp8xfp4', 'fp8xfp4', 'nvfp4xnvfp4', 'bf16xbf16'])
        experts = rng.choice([16, 32, 64] if mma == 'bf16xbf16' else [32, 64, 128, 256])
        fused = mma != 'bf16xbf16' and rng.random() < 0.6
        shared = rng.choice([0, 1]) if mma == 'fp8xfp4' and not fused else 0
        case = _moe('', mma, _log_int(rng, 1, 8192), experts=experts, topk=rng.choice([4, 6, 8]),
                    hidden=rng.choice([2048, 4096, 7168]), inter=rng.choice([1024, 1536, 2048]), shared=shared, fused=fused)
        del case['name']
        return case
    if kind == 'contiguous':
        mma = rng.choice(['fp8xfp4', 'fp8xfp8', 'bf16', 'nvfp4'])
        lo = _log_int(rng, 16, 2048)
        return dict(kind=kind, mma=mma, groups=rng.choice([3, 4, 8, 16]), rows_lo=lo, rows_hi=lo * 2,
                    n=128 * _log_int(rng, 4, 56) if mma != 'nvfp4' else 256 * _log_int(rng, 2, 28), k=256 * _log_int(rng, 4, 28),
                    psum=rng.random() < 0.5)
    if kind == 'masked':
        return dict(kind=kind, mma=rng.choice(['fp8xfp4', 'fp8xfp8', 'bf16']), groups=_log_int(rng, 4, 48), max_m=256,
                    mean=_log_int(rng, 2, 160), n=256 * _log_int(rng, 4, 28), k=128 * _log_int(rng, 8, 56))
    if kind == 'dense':
        m, mma = _log_int(rng, 1, 8192), rng.choice(['bf16', 'fp8xfp8', 'fp8xfp4'])
        return dict(kind=kind, mma=mma, m=m, n=128 * _log_int(rng, 4, 64), k=128 * _log_int(rng, 4, 128))
    if kind == 'kgrouped':
        return dict(kind=kind, mma=rng.choice(['fp8', 'bf16']), groups=rng.choice([4, 8, 16]), mean_k=128 * _log_int(rng, 1, 32),
                    m=rng.choice([1024, 2000, 2048, 4096]), n=rng.choice([1024, 1536, 4096, 7168]))
    return dict(kind='cast', mma=rng.choice(['fp8', 'fp8', 'fp4', 'nvfp4']), m=_log_int(rng, 1, 16384),
                k=128 * _log_int(rng, 8, 56), gran=rng.choice([32, 128]))


# ----------------------------------------------------------------------------------------------------- number formats

def _ceil_div(a, b):
    return -(-a // b)


def _align(a, b):
    return _ceil_div(a, b) * b


def _ue8m0_ceil(x):
    """Smallest power of two >= x."""
    bits = x.float().contiguous().view(torch.int32)
    e = ((bits >> 23) & 0xFF) + ((bits & 0x7FFFFF) != 0).to(torch.int32)
    return (e.clamp_(1, 254) << 23).view(torch.float32)


def _pack_ue8m0(sf):
    pad = _align(sf.shape[-1], 4) - sf.shape[-1]
    if pad:
        sf = torch.nn.functional.pad(sf, (0, pad), value=1.0)
    return (sf.contiguous().view(torch.int32) >> 23).to(torch.uint8).view(torch.int32)


def _e2m1_codes(x):
    mag = torch.zeros(x.shape, dtype=torch.uint8, device=x.device)
    ax = x.abs()
    for t in _E2M1_THRESHOLDS:
        mag += ax > t
    return mag | ((x < 0) & (mag != 0)).to(torch.uint8) << 3


def _pack_codes(codes):
    return (codes[..., 0::2] | (codes[..., 1::2] << 4)).view(torch.int8)


def _unpack_codes(packed):
    table = torch.tensor(_E2M1 + (0.0,) + tuple(-v for v in _E2M1[1:]), dtype=torch.float64, device=packed.device)
    raw = packed.contiguous().view(torch.uint8)
    out = torch.empty(raw.shape[:-1] + (raw.shape[-1] * 2,), dtype=torch.float64, device=packed.device)
    out[..., 0::2] = table[(raw & 0xF).int()]
    out[..., 1::2] = table[(raw >> 4).int()]
    return out


def _blocks(x, gran):
    pad = _align(x.shape[-1], gran) - x.shape[-1]
    if pad:
        x = torch.nn.functional.pad(x, (0, pad))
    return x.float().view(x.shape[:-1] + (-1, gran))


def _fp8(x, gran):
    """[..., K] -> (E4M3, FP32 power-of-two scale per ``gran`` along K)."""
    k, b = x.shape[-1], _blocks(x, gran)
    sf = _ue8m0_ceil(b.abs().amax(-1).clamp(min=1e-4) / 448.0)
    q = (b * (1.0 / sf).unsqueeze(-1)).to(torch.float8_e4m3fn).flatten(-2)
    return q[..., :k].contiguous(), sf


def _fp4(x, gran):
    k, b = x.shape[-1], _blocks(x, gran)
    sf = _ue8m0_ceil(b.abs().amax(-1).clamp(min=1e-4) / 6.0)
    return _pack_codes(_e2m1_codes(b * (1.0 / sf).unsqueeze(-1)).flatten(-2))[..., :k // 2].contiguous(), sf


def _nvfp4(x, scale):
    """[..., K] -> (packed E2M1, UE4M3 scale per 16) against the FP32 scalar ``scale``."""
    b = x.float().unflatten(-1, (-1, 16))
    sf = (b.abs().amax(-1) / 6.0 / scale).clamp(max=448.0).to(torch.float8_e4m3fn)
    f = (sf.float() * scale).unsqueeze(-1)
    return _pack_codes(_e2m1_codes(torch.where(f > 0, b / f, torch.zeros_like(b))).flatten(-2)), sf


def _spread(sf, gran, k):
    return sf.double().repeat_interleave(gran, dim=-1)[..., :k]


def _from_fp8(q, sf, gran):
    return q.double() * _spread(sf, gran, q.shape[-1])


def _from_fp4(q, sf, gran):
    return _unpack_codes(q) * _spread(sf, gran, q.shape[-1] * 2)


def _from_nvfp4(q, sf, scale):
    return _unpack_codes(q) * _spread(sf.float(), 16, q.shape[-1] * 2) * scale.double()


def _gen(seed):
    return torch.Generator(device=_DEV).manual_seed(int(seed) * 7919 + 17)


def _randn(g, *shape, std=1.0):
    return (torch.randn(*shape, generator=g, device=_DEV) * std).bfloat16()


# ------------------------------------------------------------------------------------------------------------- MoE layer

_CHUNK = 8  # experts whose weights are drawn and quantised together


def _moe_weights(c, g):
    """[(W1 [gate | up], W2)] of all experts in the layer's format, as the quantiser leaves them: tuples of tensors."""
    parts = ([], [])
    for lo in range(0, c['experts'], _CHUNK):
        e = min(_CHUNK, c['experts'] - lo)
        for out, shape in zip(parts, ((e, 2 * c['inter'], c['hidden']), (e, c['hidden'], c['inter']))):
            w = _randn(g, *shape, std=0.02)
            if c['mma'] == 'bf16xbf16':
                out.append((w,))
            elif c['mma'] == 'fp8xfp4':
                out.append(_fp4(w, 32))
            else:
                scale = w.abs().flatten(1).amax(1).float() / (6.0 * 448.0)
                out.append(_nvfp4(w, scale.view(e, 1, 1)) + (scale,))
    return [tuple(torch.cat(t) for t in zip(*p)) for p in parts]


def _moe_inputs(c, g):
    x = _randn(g, c['tokens'], c['hidden'])
    logits = torch.randn(c['tokens'], c['experts'], generator=g, device=_DEV)
    drop = torch.rand(c['tokens'], c['topk'], generator=g, device=_DEV) < 0.02
    return x, logits, drop


def _route(logits, topk):
    """Sigmoid scores, the topk largest (ties to the lower expert), weights renormalised to sum 1."""
    idx = torch.sort(logits, dim=1, descending=True, stable=True).indices[:, :topk].contiguous()
    s = torch.sigmoid(logits.double()).gather(1, idx)
    return idx, s / s.sum(1, keepdim=True)


def _moe_scales(c):
    """Calibrated NVFP4 scales: tokens stay below 6, the weighted activations between the GEMMs below about 25 s^2 / k."""
    act = 0.02 ** 2 * c['hidden'] * 40.0 / c['topk']
    return [torch.tensor(v / (6.0 * 448.0), dtype=torch.float32, device=_DEV) for v in (6.0, act)]


def _shared_weights(c, g):
    si = c['inter'] * c['shared']
    return _fp8(_randn(g, 2 * si, c['hidden'], std=0.02), 32), _fp8(_randn(g, c['hidden'], si, std=0.02), 32)


def _routing(c, logits, drop):
    idx, w = _route(logits, c['topk'])
    if not c['fused']:
        idx, w = idx.masked_fill(drop, -1), w.masked_fill(drop, 0.0)
    return idx, w


def _prepare_moe(c, seed):
    g = _gen(seed)
    x, logits, drop = _moe_inputs(c, g)
    w1, w2 = _moe_weights(c, g)
    e, h, i, t = c['experts'], c['hidden'], c['inter'], c['tokens']
    s = dict(case=c)
    if c['mma'] == 'bf16xbf16':
        s['l1'], s['l2'] = dg.transform_weights_for_mega_moe(w1[0], w2[0])
    elif c['mma'] == 'fp8xfp4':
        s['l1'], s['l2'] = dg.transform_weights_for_mega_moe(
            (w1[0], dg.transform_sf_into_required_layout(w1[1], 2 * i, h, (1, 32), e)),
            (w2[0], dg.transform_sf_into_required_layout(w2[1], h, i, (1, 32), e)))
    else:
        s['l1'], s['l2'] = dg.transform_weights_for_mega_moe((w1[0], dg.pack_nvfp4_sf_mn_major(w1[1]), w1[2]),
                                                             (w2[0], dg.pack_nvfp4_sf_mn_major(w2[1]), w2[2]))
    del w1, w2
    s['shared'] = {}
    if c['shared']:
        (a, a_sf), (b, b_sf) = _shared_weights(c, g)
        si = i * c['shared']
        s1, s2 = dg.transform_weights_for_mega_moe((a, dg.transform_sf_into_required_layout(a_sf, 2 * si, h, (1, 32))),
                                                   (b, dg.transform_sf_into_required_layout(b_sf, h, si, (1, 32))))
        s['shared'] = dict(shared_l1_weights=s1, shared_l2_weights=s2)
    buf = dg.get_symm_buffer_for_mega_moe(None, e, t, c['topk'], h, i, c['shared'], mma_type=c['mma'])
    s['buf'], s['y'] = buf, torch.empty(t, h, dtype=torch.bfloat16, device=_DEV)
    if c['mma'] == 'nvfp4xnvfp4':
        s['x_scale'], s['act_scale'] = _moe_scales(c)
    if c['fused']:
        s['x'], s['logits'] = x, logits
        return s
    # the caller's own quantiser and router have filled the buffer
    idx, w = _routing(c, logits, drop)
    buf.topk_idx[:t].copy_(idx)
    buf.topk_weights[:t].copy_(w)
    if c['mma'] == 'bf16xbf16':
        buf.x[:t].copy_(x)
    elif c['mma'] == 'fp8xfp4':
        q, sf = _fp8(x, 32)
        buf.x[:t].copy_(q)
        buf.x_sf[:t].copy_(_pack_ue8m0(sf))
    else:
        q, sf = _nvfp4(x, s['x_scale'])
        buf.x[:t].copy_(q)
        buf.x_sf[:t].copy_(sf.view(torch.uint8).view(torch.int32))
    return s


def _run_moe(s):
    c, buf = s['case'], s['buf']
    if c['mma'] == 'bf16xbf16':
        dg.bf16_mega_moe(s['y'], s['l1'], s['l2'], buf)
    elif c['mma'] == 'fp8xfp4':
        if c['fused']:
            dg.fp8_fp4_mega_moe_bf16_input(s['y'], s['x'], s['l1'], s['l2'], buf, logits=s['logits'])
        else:
            dg.fp8_fp4_mega_moe(s['y'], s['l1'], s['l2'], buf, **s['shared'])
    elif c['fused']:
        dg.nvfp4_mega_moe_bf16_input(s['y'], s['x'], s['l1'], s['l2'], buf, s['x_scale'], s['act_scale'], logits=s['logits'])
    else:
        dg.nvfp4_mega_moe(s['y'], s['l1'], s['l2'], buf, s['x_scale'], s['act_scale'])
    if c['fused']:  # the router's answer comes with the layer's
        return s['y'], buf.topk_idx[:c['tokens']], buf.topk_weights[:c['tokens']]
    return s['y']


def _exact_moe(c, seed):
    g = _gen(seed)
    x, logits, drop = _moe_inputs(c, g)
    idx, w = _routing(c, logits, drop)
    if c['mma'] == 'bf16xbf16':
        xd = x.double()
    elif c['mma'] == 'fp8xfp4':
        xd = _from_fp8(*_fp8(x, 32), 32)
    else:
        x_scale, act_scale = _moe_scales(c)
        xd = _from_nvfp4(*_nvfp4(x, x_scale), x_scale)

    def act_of(acc, weight):
        half = acc.shape[1] // 2
        gate, up = acc[:, :half].bfloat16().double(), acc[:, half:].bfloat16().double()
        a = gate / (1.0 + torch.exp(-gate)) * up * weight.double().unsqueeze(1)
        if c['mma'] == 'bf16xbf16':
            return a.bfloat16().double()
        if c['mma'] == 'fp8xfp4':
            b = a.float().unflatten(1, (-1, 32))
            sf = _ue8m0_ceil(b.abs().amax(-1) * (1.0 / 448.0))
            return _from_fp8((b * (1.0 / sf).unsqueeze(-1)).to(torch.float8_e4m3fn).flatten(1), sf, 32)
        return _from_nvfp4(*_nvfp4(a, act_scale), act_scale)

    slots = torch.zeros(c['tokens'], c['topk'], c['hidden'], dtype=torch.bfloat16, device=_DEV)
    for lo in range(0, c['experts'], _CHUNK):
        one = dict(c, experts=min(_CHUNK, c['experts'] - lo))
        w1, w2 = _moe_weights(one, g)
        for j in range(one['experts']):
            tok, slot = torch.nonzero(idx == lo + j, as_tuple=True)
            if tok.numel() == 0:
                continue
            if c['mma'] == 'bf16xbf16':
                d1, d2 = w1[0][j].double(), w2[0][j].double()
            elif c['mma'] == 'fp8xfp4':
                d1, d2 = _from_fp4(w1[0][j], w1[1][j], 32), _from_fp4(w2[0][j], w2[1][j], 32)
            else:
                d1, d2 = _from_nvfp4(w1[0][j], w1[1][j], w1[2][j]), _from_nvfp4(w2[0][j], w2[1][j], w2[2][j])
            slots[tok, slot] = (act_of(xd[tok] @ d1.T, w[tok, slot].float()) @ d2.T).bfloat16()
    y = torch.zeros(c['tokens'], c['hidden'], dtype=torch.float64, device=_DEV)
    for k in range(c['topk']):
        y += slots[:, k].double()
    if c['shared']:
        (a, a_sf), (b, b_sf) = _shared_weights(c, g)
        acc = xd @ _from_fp8(a, a_sf, 32).T
        y += (act_of(acc, torch.ones(c['tokens'], device=_DEV)) @ _from_fp8(b, b_sf, 32).T).bfloat16().double()
    return (y, idx, w) if c['fused'] else y


def _work_moe(c):
    t, h, i, e, k = c['tokens'], c['hidden'], c['inter'], c['experts'], c['topk']
    rows = t * k * (1.0 if c['fused'] else 0.98)
    per_weight = {'fp8xfp4': 0.5 + 1 / 32, 'nvfp4xnvfp4': 0.5 + 1 / 16, 'bf16xbf16': 2.0}[c['mma']]
    touched = e * (1.0 - (1.0 - k / e) ** t)  # experts that some token chose, whose weights have to be read
    x_bytes = t * h * (2.0 if c['fused'] or c['mma'] == 'bf16xbf16' else 1.0 + 1 / 32 if c['mma'] == 'fp8xfp4' else 0.5625)
    route = t * e * 4 + t * k * 12 if c['fused'] else t * k * 12
    n_bytes = touched * 3 * h * i * per_weight + x_bytes + route + t * h * 2
    flops = rows * 6.0 * h * i
    if c['shared']:
        si = i * c['shared']
        n_bytes += 3 * h * si * (1 + 1 / 32)
        flops += t * 6.0 * h * si
    return dict(bytes=n_bytes, flops=flops)


# ------------------------------------------------------------------------------------------------------- stand-alone GEMMs

def _weights(mma, g, *shape):
    """A weight operand ~ N(0, 0.02) in its format: (values, scales, ...) as a quantiser leaves it."""
    w = _randn(g, *shape, std=0.02)
    if mma == 'bf16':
        return (w,)
    if mma == 'fp8xfp4':
        return _fp4(w, 32)
    if mma == 'fp8xfp8':
        return _fp8(w, 128)
    scale = w.abs().flatten(1).amax(1).float() / (6.0 * 448.0)
    return _nvfp4(w, scale.view(-1, 1, 1)) + (scale,)


def _acts(mma, a):
    """Activations in the format that goes with ``mma``: E4M3 with one scale per 128, NVFP4 against a calibrated scale, BF16."""
    if mma == 'bf16':
        return (a,)
    if mma == 'nvfp4':
        scale = torch.tensor(6.0 / (6.0 * 448.0), dtype=torch.float32, device=_DEV)
        return _nvfp4(a, scale) + (scale,)
    return _fp8(a, 128)


def _weight_gran(mma):
    return 32 if mma == 'fp8xfp4' else 128


def _weight_exact(mma, w):
    if mma == 'bf16':
        return w[0].double()
    if mma == 'fp8xfp4':
        return _from_fp4(w[0], w[1], 32)
    if mma == 'fp8xfp8':
        return _from_fp8(w[0], w[1], 128)
    return _from_nvfp4(*w)


def _acts_exact(mma, a):
    if mma == 'bf16':
        return a[0].double()
    return _from_nvfp4(*a) if mma == 'nvfp4' else _from_fp8(a[0], a[1], 128)


def _operand_bytes(mma, rows, cols, weight):
    if mma == 'bf16':
        return rows * cols * 2.0
    if mma == 'nvfp4':
        return rows * cols * (0.5 + 1 / 16)
    if mma == 'fp8xfp4' and weight:
        return rows * cols * (0.5 + 1 / 32)
    return rows * cols * (1.0 + 1 / 32)


def _group_rows(c, seed):
    """Rows of each group, from the seed: uniform in [rows_lo, rows_hi]."""
    r = torch.randint(c['rows_lo'], c['rows_hi'] + 1, (c['groups'],), generator=torch.Generator().manual_seed(int(seed)))
    return r.tolist()


def _contiguous_inputs(c, seed):
    g, rows = _gen(seed), _group_rows(c, seed)
    m = c['groups'] * _align(c['rows_hi'], 128)  # the caller's buffer holds the most rows that can come
    a = _randn(g, m, c['k'])
    ids = torch.full((m,), -1, dtype=torch.int32)
    ends, at = [], 0
    for j, r in enumerate(rows):
        ids[at:at + r] = j
        ends.append(at + r)
        a[at + r:at + _align(r, 128)] = 0
        at += _align(r, 128)
    a[at:] = 0
    layout = torch.tensor(ends, dtype=torch.int32) if c['psum'] else ids
    return rows, m, _acts(c['mma'], a), _weights(c['mma'], g, c['groups'], c['n'], c['k']), layout.to(_DEV)


def _layout_weights(mma, w, n, k, groups=None):
    """A weight operand with its scales in the layout the kernels read, laid out once when the model is loaded."""
    if mma in ('fp8xfp4', 'fp8xfp8'):
        return (w[0], dg.transform_sf_into_required_layout(w[1], n, k, (1, _weight_gran(mma)), groups))
    if mma == 'nvfp4':
        return (w[0], dg.pack_nvfp4_sf_mn_major(w[1]), w[2])
    return w[0]


def _prepare_contiguous(c, seed):
    _, m, a, w, layout = _contiguous_inputs(c, seed)
    return dict(case=c, a=a if c['mma'] != 'bf16' else a[0], b=_layout_weights(c['mma'], w, c['n'], c['k'], c['groups']),
                layout=layout, d=torch.zeros(m, c['n'], dtype=torch.bfloat16, device=_DEV))


def _run_contiguous(s):
    c = s['case']
    if c['mma'] == 'bf16':
        dg.m_grouped_bf16_gemm_nt_contiguous(s['a'], s['b'], s['d'], s['layout'], use_psum_layout=c['psum'])
    elif c['mma'] == 'nvfp4':
        dg.m_grouped_nvfp4_gemm_nt_contiguous(s['a'], s['b'], s['d'], s['layout'], use_psum_layout=c['psum'])
    else:
        dg.m_grouped_fp8_fp4_gemm_nt_contiguous(s['a'], s['b'], s['d'], s['layout'], recipe_a=(1, 128),
                                                recipe_b=(1, _weight_gran(c['mma'])), use_psum_layout=c['psum'])
    return s['d']


def _exact_contiguous(c, seed):
    rows, m, a, w, _ = _contiguous_inputs(c, seed)
    ad = _acts_exact(c['mma'], a)
    d = torch.zeros(m, c['n'], dtype=torch.float64, device=_DEV)
    at = 0
    for j, r in enumerate(rows):
        d[at:at + r] = ad[at:at + r] @ _weight_exact(c['mma'], tuple(t[j] for t in w)).T
        at += _align(r, 128)
    return d


def _work_contiguous(c):
    rows = c['groups'] * (c['rows_lo'] + c['rows_hi']) / 2
    n, k = c['n'], c['k']
    return dict(bytes=_operand_bytes(c['mma'], rows, k, False) + _operand_bytes(c['mma'], c['groups'] * n, k, True) + rows * n * 2,
                flops=2.0 * rows * n * k)


def _masked_inputs(c, seed):
    g = _gen(seed)
    rows = torch.poisson(torch.full((c['groups'],), float(c['mean'])), generator=torch.Generator().manual_seed(int(seed)))
    rows = rows.clamp(0, c['max_m']).to(torch.int32)
    a = _acts(c['mma'], _randn(g, c['groups'], c['max_m'], c['k']))
    return rows, a, _weights(c['mma'], g, c['groups'], c['n'], c['k'])


def _prepare_masked(c, seed):
    rows, a, w = _masked_inputs(c, seed)
    if c['mma'] != 'bf16':  # a fused dispatch leaves packed scales in the layout the GEMM reads
        a = (a[0], dg.transform_sf_into_required_layout(a[1], c['max_m'], c['k'], (1, 128), c['groups']))
    return dict(case=c, a=a if c['mma'] != 'bf16' else a[0], b=_layout_weights(c['mma'], w, c['n'], c['k'], c['groups']),
                rows=rows.to(_DEV), d=torch.zeros(c['groups'], c['max_m'], c['n'], dtype=torch.bfloat16, device=_DEV))


def _run_masked(s):
    c = s['case']
    if c['mma'] == 'bf16':
        dg.m_grouped_bf16_gemm_nt_masked(s['a'], s['b'], s['d'], s['rows'], c['mean'])
    else:
        dg.m_grouped_fp8_fp4_gemm_nt_masked(s['a'], s['b'], s['d'], s['rows'], c['mean'], recipe_a=(1, 128),
                                            recipe_b=(1, _weight_gran(c['mma'])))
    return s['d']


def _exact_masked(c, seed):
    rows, a, w = _masked_inputs(c, seed)
    d = torch.zeros(c['groups'], c['max_m'], c['n'], dtype=torch.float64, device=_DEV)
    for j, r in enumerate(rows.tolist()):
        if r:
            d[j, :r] = _acts_exact(c['mma'], tuple(t[j, :r] for t in a)) @ _weight_exact(c['mma'], tuple(t[j] for t in w)).T
    return d


def _work_masked(c):
    rows = c['groups'] * c['mean']
    n, k = c['n'], c['k']
    return dict(bytes=_operand_bytes(c['mma'], rows, k, False) + _operand_bytes(c['mma'], c['groups'] * n, k, True) + rows * n * 2,
                flops=2.0 * rows * n * k)


def _dense_inputs(c, seed):
    g = _gen(seed)
    return _acts(c['mma'], _randn(g, c['m'], c['k'])), _weights(c['mma'], g, c['n'], c['k'])


def _prepare_dense(c, seed):
    a, w = _dense_inputs(c, seed)
    return dict(case=c, a=a if c['mma'] != 'bf16' else a[0], b=_layout_weights(c['mma'], w, c['n'], c['k']),
                d=torch.empty(c['m'], c['n'], dtype=torch.bfloat16, device=_DEV))


def _run_dense(s):
    c = s['case']
    if c['mma'] == 'bf16':
        dg.bf16_gemm_nt(s['a'], s['b'], s['d'])
    else:
        dg.fp8_fp4_gemm_nt(s['a'], s['b'], s['d'], recipe_a=(1, 128), recipe_b=(1, _weight_gran(c['mma'])))
    return s['d']


def _exact_dense(c, seed):
    a, w = _dense_inputs(c, seed)
    return _acts_exact(c['mma'], a) @ _weight_exact(c['mma'], w).T


def _work_dense(c):
    m, n, k = c['m'], c['n'], c['k']
    return dict(bytes=_operand_bytes(c['mma'], m, k, False) + _operand_bytes(c['mma'], n, k, True) + m * n * 2, flops=2.0 * m * n * k)


# ------------------------------------------------------------------------------------------------- weight-gradient GEMM

def _group_ks(c, seed):
    """K rows of each group: multiples of 128 around ``mean_k``, the sum fixed."""
    r = torch.Generator().manual_seed(int(seed))
    ks, mean = [c['mean_k']] * c['groups'], c['mean_k'] // 128
    for j in range(0, c['groups'] - 1, 2):
        move = 128 * int(torch.randint(0, mean // 2 + 1, (1,), generator=r))
        ks[j], ks[j + 1] = ks[j] - move, ks[j + 1] + move
    return ks


def _per_channel_fp8(x):
    b = x.float().unflatten(0, (-1, 128))
    sf = _ue8m0_ceil(b.abs().amax(1).clamp(min=1e-4) / 448.0)
    return (b * (1.0 / sf).unsqueeze(1)).to(torch.float8_e4m3fn).flatten(0, 1), sf


def _kgrouped_inputs(c, seed):
    g, ks = _gen(seed), _group_ks(c, seed)
    a, b = _randn(g, sum(ks), c['m']), _randn(g, sum(ks), c['n'])
    acc = torch.randn(c['groups'], c['m'], c['n'], generator=g, device=_DEV)
    if c['mma'] == 'fp8':
        a, b = _per_channel_fp8(a), _per_channel_fp8(b)
    return ks, a, b, acc


def _prepare_kgrouped(c, seed):
    ks, a, b, acc = _kgrouped_inputs(c, seed)
    return dict(case=c, ks=ks, a=a, b=b, c=acc, layout=torch.tensor(ks, dtype=torch.int32, device=_DEV), d=torch.empty_like(acc))


def _run_kgrouped(s):
    # c and d are two tensors, so that a pass can be repeated
    entry = dg.k_grouped_fp8_gemm_tn_contiguous if s['case']['mma'] == 'fp8' else dg.k_grouped_bf16_gemm_tn_contiguous
    entry(s['a'], s['b'], s['d'], s['ks'], s['layout'], s['c'])
    return s['d']


def _exact_kgrouped(c, seed):
    ks, a, b, acc = _kgrouped_inputs(c, seed)

    def rows(t, lo, k):
        if c['mma'] == 'bf16':
            return t[lo:lo + k].double()
        return t[0][lo:lo + k].double() * t[1][lo // 128:(lo + k) // 128].double().repeat_interleave(128, dim=0)

    d, at = acc.double(), 0
    for j, k in enumerate(ks):
        d[j] += rows(a, at, k).T @ rows(b, at, k)
        at += k
    return d


def _work_kgrouped(c):
    sum_k, m, n = c['groups'] * c['mean_k'], c['m'], c['n']
    per = 2.0 if c['mma'] == 'bf16' else 1.0 + 4 / 128
    return dict(bytes=sum_k * (m + n) * per + 8.0 * c['groups'] * m * n, flops=2.0 * sum_k * m * n)


# ---------------------------------------------------------------------------------------------------------- quantisers

def _prepare_cast(c, seed):
    return dict(case=c, x=_randn(_gen(seed), c['m'], c['k']),
                scale=torch.tensor(6.0 / (6.0 * 448.0), dtype=torch.float32, device=_DEV))


def _run_cast(s):
    c = s['case']
    if c['mma'] == 'fp8':
        q, sf = dg.utils.math.per_token_cast_to_fp8(s['x'], True, c['gran'])
        return q.view(torch.uint8), sf
    if c['mma'] == 'fp4':
        return dg.utils.math.per_token_cast_to_fp4(s['x'], True, c['gran'])
    q, sf, _ = dg.per_token_cast_to_nvfp4(s['x'], s['scale'])
    return q, sf.view(torch.uint8)


def _work_cast(c):
    per = {'fp8': 1.0 + 4 / c['gran'], 'fp4': 0.5 + 4 / c['gran'], 'nvfp4': 0.5 + 1 / 16}[c['mma']]
    return dict(bytes=c['m'] * c['k'] * (2.0 + per), flops=0.0)


# -------------------------------------------------------------------------------------------------------------- the file

_PREPARE = dict(moe=_prepare_moe, contiguous=_prepare_contiguous, masked=_prepare_masked, dense=_prepare_dense,
                kgrouped=_prepare_kgrouped, cast=_prepare_cast)
_RUN = dict(moe=_run_moe, contiguous=_run_contiguous, masked=_run_masked, dense=_run_dense, kgrouped=_run_kgrouped, cast=_run_cast)
_EXACT = dict(moe=_exact_moe, contiguous=_exact_contiguous, masked=_exact_masked, dense=_exact_dense, kgrouped=_exact_kgrouped)
_WORK = dict(moe=_work_moe, contiguous=_work_contiguous, masked=_work_masked, dense=_work_dense, kgrouped=_work_kgrouped,
             cast=_work_cast)


def prepare(case, seed):
    return _PREPARE[case['kind']](case, seed)


def run(state):
    return _RUN[state['case']['kind']](state)


def exact(case, seed):
    return _EXACT[case['kind']](case, seed) if case['kind'] in _EXACT else None


def work(case):
    return _WORK[case['kind']](case)


def tolerance(case):
    """About four times what the present code differs from ``exact``, which is what another order of the 32-bit sums shows at
    most: 1.7e-3 to 1.9e-3 for BF16 results (a rounding of up to 2^-9, and in a layer also the BF16 and FP8 / FP4 values
    between its GEMMs that fall on the other side of a rounding boundary), 3e-7 to 3e-6 for FP32 ones. Quantisers are
    exact, the router's choice is but for ties."""
    if case['kind'] == 'cast':
        return 'exact'
    if case['kind'] == 'kgrouped':
        return dict(rel=1.2e-5)
    if case['kind'] == 'moe':
        return dict(rel=7e-3, differ=1e-3)
    return dict(rel=7e-3)
