"""The GEMM kernel on CTA pairs (256 x 256 tiles), and the forms that stay on single CTAs although pairs are asked for, against
the oracle at the sizes where its tiles can go wrong: rows around multiples of 128 and 256 (the second CTA of the last pair with no, one or all of its rows), groups that leave a remainder to
the single-CTA kernel, K around the depth of the operand ring, empty groups. Tolerances as for the single-CTA kernel:
calc_diff <= 2e-3 (FP4 weights), <= 1e-3 (FP8 x FP8), < 1e-5 (BF16)."""
import pytest
import torch

from oracle import gemm as ogemm
from oracle import moe as omoe
from oracle import nvfp4 as onv
from oracle import quant
from tests.helpers import gemm_kernels_of, moe_case, moe_case_nvfp4, quantize_groups

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    return deepgemm_b200


@pytest.fixture(autouse=True)
def _pairs_everywhere():
    from deepgemm_b200 import _lib
    _lib.check(_lib.lib().dgb200_set_tuning(b'pair', 1))
    yield
    _lib.check(_lib.lib().dgb200_set_tuning(b'pair', -1))
    assert _lib.device_status()[0] == 0


ROWS = [(1, 256, 128), (127, 512, 768), (129, 256, 896), (256, 512, 1024), (257, 256, 128), (385, 512, 640), (700, 768, 2048)]


@pytest.mark.parametrize('kind', ['fp8xfp8', 'fp8xfp4', 'nvfp4', 'masked', 'bf16', 'k_grouped_fp8', 'k_grouped_bf16'])
def test_which_forms_run_on_pairs(dg, kind):
    """Scale factors in plain row order stay on single CTAs, whatever the knob says: no CTA of a pair hands the other one shared
    memory that its threads have written. The K-grouped form packs its scales in the order the tensor cores read."""
    m, n, k = 512, 512, 512
    ints = lambda rows, gran, groups=None: dg.transform_sf_into_required_layout(
        torch.ones(*([groups] if groups else []), rows, k // gran, device='cuda'), rows, k, (1, gran), groups)
    fp8 = lambda *shape: torch.ones(*shape, device='cuda').to(torch.float8_e4m3fn)
    fp4 = lambda *shape: torch.zeros(*shape[:-1], shape[-1] // 2, dtype=torch.int8, device='cuda')
    bf16 = lambda *shape: torch.ones(*shape, dtype=torch.bfloat16, device='cuda')
    if kind in ('fp8xfp8', 'fp8xfp4'):
        gran = 32 if kind == 'fp8xfp4' else 128
        a, b = (fp8(m, k), ints(m, gran)), ((fp8 if kind == 'fp8xfp8' else fp4)(n, k), ints(n, gran))
        call = lambda: dg.fp8_fp4_gemm_nt(a, b, bf16(m, n), recipe_a=(1, gran), recipe_b=(1, gran))
    elif kind == 'nvfp4':
        a = dg.per_token_cast_to_nvfp4(bf16(m, k))
        sf = dg.pack_nvfp4_sf_mn_major(torch.ones(1, n, k // 16, device='cuda').to(torch.float8_e4m3fn))
        layout = torch.tensor([m], dtype=torch.int32, device='cuda')
        call = lambda: dg.m_grouped_nvfp4_gemm_nt_contiguous(a, (fp4(1, n, k), sf, torch.ones(1, device='cuda')), bf16(m, n), layout,
                                                             use_psum_layout=True)
    elif kind == 'masked':
        counts = torch.tensor([m, m], dtype=torch.int32, device='cuda')
        call = lambda: dg.m_grouped_fp8_fp4_gemm_nt_masked((fp8(2, m, k), ints(m, 128, 2)), (fp8(2, n, k), ints(n, 128, 2)), bf16(2, m, n),
                                                           counts, m, recipe_a=(1, 128), recipe_b=(1, 128))
    elif kind == 'bf16':
        call = lambda: dg.bf16_gemm_nt(bf16(m, k), bf16(n, k), bf16(m, n))
    else:
        ks, d = torch.tensor([k], dtype=torch.int32, device='cuda'), torch.zeros(1, m, n, device='cuda')
        if kind == 'k_grouped_fp8':
            a, b = dg.utils.per_channel_cast_to_fp8(bf16(k, m), True), dg.utils.per_channel_cast_to_fp8(bf16(k, n), True)
            call = lambda: dg.k_grouped_fp8_gemm_tn_contiguous(a, b, d, [k], ks, c=d)
        else:
            call = lambda: dg.k_grouped_bf16_gemm_tn_contiguous(bf16(k, m), bf16(k, n), d, [k], ks, c=d)
    assert gemm_kernels_of(call) == {(256, kind in ('bf16', 'k_grouped_fp8', 'k_grouped_bf16'), False)}


@pytest.mark.parametrize('m,n,k', ROWS)
@pytest.mark.parametrize('b_fp4', [True, False])
def test_dense_fp8(dg, m, n, k, b_fp4):
    torch.manual_seed(m + n + k)
    a_q, a_sf = quant.quantize_fp8_per_token(torch.randn(m, k).bfloat16(), 128)
    b = (torch.randn(n, k) * 0.02).bfloat16()
    b_q, b_sf = (quant.quantize_fp4_per_token if b_fp4 else quant.quantize_fp8_per_token)(b, 32)
    want = quant.dequantize_fp8(a_q, a_sf, 128) @ (quant.dequantize_fp4(b_q, b_sf, 32) if b_fp4 else quant.dequantize_fp8(b_q, b_sf, 32)).T
    d = torch.full((m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    dg.fp8_fp4_gemm_nt((a_q.cuda(), a_sf.cuda()), (b_q.cuda(), b_sf.cuda()), d, recipe_a=(1, 128), recipe_b=(1, 32))
    assert quant.calc_diff(d.cpu(), want) <= (2e-3 if b_fp4 else 1e-3)


@pytest.mark.parametrize('m,n,k', ROWS)
@pytest.mark.parametrize('form', ['nt', 'nn', 'tn'])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
def test_dense_bf16(dg, m, n, k, form, dtype):
    torch.manual_seed(m + n + k)
    m = m if form != 'tn' else -(-m // 8) * 8  # what a transposed a needs
    a, b = torch.randn(m, k).bfloat16(), torch.randn(n, k).bfloat16()
    want = a.float() @ b.float().T
    a_in = a.T.contiguous() if form == 'tn' else a
    b_in = b if form == 'nt' else b.T.contiguous()
    d = torch.full((m, n), float('nan'), dtype=dtype, device='cuda')
    getattr(dg, f'bf16_gemm_{form}')(a_in.cuda(), b_in.cuda(), d)
    assert quant.calc_diff(d.cpu(), want) < 1e-5


@pytest.mark.parametrize('kind', ['fp8', 'bf16'])
def test_masked(dg, kind):
    """Two groups' tiles never touch rows past their own count, nor each other's."""
    rows, max_m, n, k = [0, 1, 128, 129, 256, 300, 384], 384, 256, 512
    torch.manual_seed(5)
    a, b = torch.randn(len(rows), max_m, k).bfloat16(), (torch.randn(len(rows), n, k) * 0.02).bfloat16()
    masked = torch.tensor(rows, dtype=torch.int32)
    d = torch.full((len(rows), max_m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    if kind == 'bf16':
        want, mask = ogemm.bf16_grouped_gemm_masked(a, b, masked)
        dg.m_grouped_bf16_gemm_nt_masked(a.cuda(), b.cuda(), d, masked.cuda(), 200)
    else:
        (a_q, a_sf), (b_q, b_sf) = quantize_groups(a, 128, False), quantize_groups(b, 32, True)
        want, mask = ogemm.grouped_gemm_masked(a_q, a_sf, b_q, b_sf, masked, gran_k_a=128, gran_k_b=32)
        dg.m_grouped_fp8_fp4_gemm_nt_masked((a_q.cuda(), a_sf.cuda()), (b_q.cuda(), b_sf.cuda()), d, masked.cuda(), 200,
                                            recipe_a=(1, 128), recipe_b=(1, 32))
    got = d.cpu()
    assert torch.isnan(got.float())[~mask].all() and not torch.isnan(got.float())[mask].any()
    assert quant.calc_diff(got[mask], want[mask]) <= (1e-5 if kind == 'bf16' else 2e-3)


@pytest.mark.parametrize('alignment', [16, 128])
@pytest.mark.parametrize('zero_padding', [False, True])
@pytest.mark.parametrize('mn_major', [False, True])
def test_psum_bf16(dg, alignment, zero_padding, mn_major):
    """Groups that start off the 128-row grid: the second CTA's rows may lie in the next group. Padding rows as asked."""
    rows, n, k = [128, 0, 1, 129, 255, 256, 257, 385, 40], 512, 320
    torch.manual_seed(alignment)
    starts, ends, at = [], [], 0
    for r in rows:
        starts.append(at)
        ends.append(at + r)
        at += -(-r // alignment) * alignment
    a = torch.zeros(at + 64, k).bfloat16()  # ... and rows no group owns at the end
    for s, e in zip(starts, ends):
        a[s:e] = torch.randn(e - s, k).bfloat16()
    b, psum = (torch.randn(len(rows), n, k) * 0.05).bfloat16(), torch.tensor(ends, dtype=torch.int32)
    want, mask = ogemm.bf16_grouped_gemm_contiguous(a, b, psum, use_psum_layout=True, alignment=alignment)
    d = torch.full((a.size(0), n), float('nan'), dtype=torch.bfloat16, device='cuda')
    b_in = b.cuda().transpose(1, 2).contiguous().transpose(1, 2) if mn_major else b.cuda()
    before = dg.get_mk_alignment_for_contiguous_layout()
    dg.set_mk_alignment_for_contiguous_layout(alignment)
    try:
        forms = gemm_kernels_of(lambda: dg.m_grouped_bf16_gemm_nt_contiguous(a.cuda(), b_in, d, psum.cuda(), use_psum_layout=True,
                                                                             ensure_zero_padding=zero_padding))
    finally:
        dg.set_mk_alignment_for_contiguous_layout(before)
    assert forms == {(256, True, False)}
    got = d.cpu().float()
    padding = torch.zeros_like(mask)
    for s, e in zip(starts, ends):
        padding[e:s + -(-(e - s) // alignment) * alignment] = True
    assert quant.calc_diff(got[mask], want[mask]) < 1e-5
    assert (got[padding] == 0).all() if zero_padding else torch.isnan(got[padding]).all()
    assert torch.isnan(got[~mask & ~padding]).all()


@pytest.mark.parametrize('rows,k,pairs', [([800, 801, 1023], 5376, True), ([800, 801, 1023], 256, False), ([300, 200, 500], 5376, False)])
def test_psum_bf16_takes_pairs_by_itself(dg, rows, k, pairs):
    """Only with many rows per group and enough work in all."""
    from deepgemm_b200 import _lib
    _lib.check(_lib.lib().dgb200_set_tuning(b'pair', -1))
    n = 512
    torch.manual_seed(1)
    ends, at = [], 0
    for r in rows:
        ends.append(at + r)
        at += -(-r // 128) * 128
    a, b, psum = torch.randn(at, k).bfloat16(), (torch.randn(3, n, k) * 0.05).bfloat16(), torch.tensor(ends, dtype=torch.int32)
    want, mask = ogemm.bf16_grouped_gemm_contiguous(a, b, psum, use_psum_layout=True)
    d = torch.zeros(at, n, dtype=torch.bfloat16, device='cuda')
    forms = gemm_kernels_of(lambda: dg.m_grouped_bf16_gemm_nt_contiguous(a.cuda(), b.cuda(), d, psum.cuda(), use_psum_layout=True))
    assert forms == {(256, pairs, False)}
    assert quant.calc_diff(d.cpu()[mask], want[mask]) < 1e-5


@pytest.mark.parametrize('m,n,k,pairs', [(4096, 4096, 1024, True), (1024, 512, 8192, True), (512, 512, 1024, False), (100, 4096, 8192, False)])
def test_dense_and_k_grouped_take_pairs_by_themselves(dg, m, n, k, pairs):
    from deepgemm_b200 import _lib
    for name, value in ((b'pair', -1), (b'split_k', 0)):
        _lib.check(_lib.lib().dgb200_set_tuning(name, value))
    bf16 = lambda *shape: torch.ones(*shape, dtype=torch.bfloat16, device='cuda')
    try:
        assert gemm_kernels_of(lambda: dg.bf16_gemm_nt(bf16(m, k), bf16(n, k), bf16(m, n))) == {(256, pairs, False)}
    finally:
        _lib.check(_lib.lib().dgb200_set_tuning(b'split_k', -1))
    m = -(-m // 8) * 8
    ks, d = torch.tensor([k], dtype=torch.int32, device='cuda'), torch.zeros(1, m, n, device='cuda')
    forms = gemm_kernels_of(lambda: dg.k_grouped_bf16_gemm_tn_contiguous(bf16(k, m), bf16(k, n), d, [k], ks, c=d))
    assert forms == {(256, pairs, False)}


@pytest.mark.parametrize('m', [16, 144, 256, 272, 400])
@pytest.mark.parametrize('kind', ['fp8', 'bf16'])
@pytest.mark.parametrize('alias', [True, False])
def test_k_grouped(dg, m, kind, alias):
    ks, n = [128, 0, 896, 640], 512
    torch.manual_seed(m)
    a, b = torch.randn(sum(ks), m).bfloat16(), torch.randn(sum(ks), n).bfloat16()
    c = torch.randn(len(ks), m, n)
    c_dev = c.cuda()
    d = c_dev if alias else torch.full_like(c_dev, float('nan'))
    layout = torch.tensor(ks, dtype=torch.int32, device='cuda')
    if kind == 'fp8':
        (a_q, a_sf), (b_q, b_sf) = quant.quantize_fp8_per_channel(a), quant.quantize_fp8_per_channel(b)
        want = ogemm.k_grouped_gemm(a_q, a_sf, b_q, b_sf, c, ks)
        dg.k_grouped_fp8_gemm_tn_contiguous((a_q.cuda(), a_sf.cuda()), (b_q.cuda(), b_sf.cuda()), d, ks, layout, c=c_dev)
    else:
        want, at = c.clone(), 0
        for g, k in enumerate(ks):
            want[g] += a[at:at + k].float().T @ b[at:at + k].float()
            at += k
        dg.k_grouped_bf16_gemm_tn_contiguous(a.cuda(), b.cuda(), d, ks, layout, c=c_dev)
    got = d.cpu()
    assert torch.equal(got[1], c[1]), 'an empty group must pass c through'
    for g in (0, 2, 3):
        assert quant.calc_diff(got[g] - c[g], want[g] - c[g]) <= (1e-3 if kind == 'fp8' else 1e-5)


@pytest.mark.parametrize('kind', ['fp8', 'bf16', 'nvfp4'])
def test_layer_with_remainders(dg, kind):
    """Experts whose rows leave every kind of remainder: whole pair tiles, 1 and 128 rows for the single-CTA kernel, 129 rows
    that make a pair tile of their own, and experts that are only one of the two."""
    rows = [0, 1, 128, 129, 255, 256, 257, 384, 385, 512, 513, 300]
    experts, topk, hidden, inter, tokens = len(rows), 1, 512, 256, sum(rows)
    make = moe_case_nvfp4 if kind == 'nvfp4' else moe_case
    c = make(tokens, hidden, inter, experts, topk, seed=3)
    order = torch.repeat_interleave(torch.arange(experts), torch.tensor(rows))
    idx = order[torch.randperm(tokens)].view(tokens, 1)
    w = torch.rand(tokens, 1) + 0.5
    mma = {'fp8': 'fp8xfp4', 'bf16': 'bf16xbf16', 'nvfp4': 'nvfp4xnvfp4'}[kind]
    buf = dg.get_symm_buffer_for_mega_moe(None, experts, tokens, topk, hidden, inter, mma_type=mma)
    buf.topk_idx[:tokens].copy_(idx.cuda())
    buf.topk_weights[:tokens].copy_(w.cuda())
    y = torch.full((tokens, hidden), float('nan'), dtype=torch.bfloat16, device='cuda')
    if kind == 'fp8':
        want = omoe.moe_layer(c['x_q'], c['x_sf'], idx, w, c['l1_q'], c['l1_sf'], c['l2_q'], c['l2_sf'])
        l1, l2 = dg.transform_weights_for_mega_moe(
            (c['l1_q'].cuda(), dg.transform_sf_into_required_layout(c['l1_sf'].cuda(), 2 * inter, hidden, (1, 32), experts)),
            (c['l2_q'].cuda(), dg.transform_sf_into_required_layout(c['l2_sf'].cuda(), hidden, inter, (1, 32), experts)))
        buf.x[:tokens].copy_(c['x_q'].cuda())
        buf.x_sf[:tokens].copy_(quant.pack_ue8m0(c['x_sf']).cuda())
        dg.fp8_fp4_mega_moe(y, l1, l2, buf)
    elif kind == 'bf16':
        w1, w2 = (torch.randn(experts, 2 * inter, hidden) * 0.05).bfloat16(), (torch.randn(experts, hidden, inter) * 0.05).bfloat16()
        want = omoe.moe_layer_bf16(c['x'], idx, w, w1, w2)
        l1, l2 = dg.transform_weights_for_mega_moe(w1.cuda(), w2.cuda())
        buf.x[:tokens].copy_(c['x'].cuda())
        dg.bf16_mega_moe(y, l1, l2, buf)
    else:
        scale = onv.calibrate_act_scale(c['x_q'], c['x_sf'], c['x_scale'], idx, w, c['l1_q'], c['l1_sf'], c['l1_scales'])
        want = onv.moe_layer_nvfp4(c['x_q'], c['x_sf'], c['x_scale'], idx, w, c['l1_q'], c['l1_sf'], c['l1_scales'], c['l2_q'],
                                   c['l2_sf'], c['l2_scales'], scale)
        l1, l2 = dg.transform_weights_for_mega_moe((c['l1_q'].cuda(), dg.pack_nvfp4_sf_mn_major(c['l1_sf'].cuda()), c['l1_scales'].cuda()),
                                                   (c['l2_q'].cuda(), dg.pack_nvfp4_sf_mn_major(c['l2_sf'].cuda()), c['l2_scales'].cuda()))
        buf.x[:tokens].copy_(c['x_q'].cuda())
        buf.x_sf[:tokens].copy_(c['x_sf'].view(torch.uint8).contiguous().view(torch.int32).cuda())
        dg.nvfp4_mega_moe(y, l1, l2, buf, c['x_scale'].cuda(), scale.cuda(), fast_math=False)
    got = y.cpu()
    assert not torch.isnan(got.float()).any()
    per_expert = [quant.calc_diff(got[idx[:, 0] == e], want[idx[:, 0] == e]) for e in range(experts) if rows[e]]
    assert max(per_expert) <= (1e-4 if kind == 'bf16' else 2e-3), per_expert
