"""The layer's GEMMs that run side by side on the library's own streams: which launches do, what an SM limit makes of them, CUDA
graphs, and callers on several streams at once. The bits never depend on where a GEMM ran."""
import pytest
import torch

from oracle import quant
from tests.helpers import kernel_launches, moe_case, quantize_groups

pytestmark = pytest.mark.gpu
HIDDEN, INTER, TOPK = 512, 256, 2


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    yield deepgemm_b200
    from deepgemm_b200 import _lib
    assert _lib.device_status()[0] == 0


def _layer(dg, tokens, experts, shared, seed=7):
    """(call, output) of a layer on a buffer of its own, quantised rows and routes already in it."""
    c = moe_case(tokens, HIDDEN, INTER, experts, TOPK, seed=seed)
    ints = lambda sf, rows, k, groups=None: dg.transform_sf_into_required_layout(sf.cuda(), rows, k, (1, 32), groups)
    l1, l2 = dg.transform_weights_for_mega_moe((c['l1_q'].cuda(), ints(c['l1_sf'], 2 * INTER, HIDDEN, experts)),
                                               (c['l2_q'].cuda(), ints(c['l2_sf'], HIDDEN, INTER, experts)))
    extra = {}
    if shared:
        torch.manual_seed(seed + 1)
        (q1, f1), (q2, f2) = (quantize_groups((torch.randn(1, *s) * 0.02).bfloat16(), 32, False) for s in ((2 * INTER, HIDDEN), (HIDDEN, INTER)))
        s1, s2 = dg.transform_weights_for_mega_moe((q1[0].cuda(), ints(f1[0], 2 * INTER, HIDDEN)), (q2[0].cuda(), ints(f2[0], HIDDEN, INTER)))
        extra = dict(shared_l1_weights=s1, shared_l2_weights=s2)
    buf = dg.get_symm_buffer_for_mega_moe(None, experts, tokens, TOPK, HIDDEN, INTER, num_shared_experts=int(shared))
    buf.x[:tokens].copy_(c['x_q'].cuda())
    buf.x_sf[:tokens].copy_(quant.pack_ue8m0(c['x_sf']).cuda())
    buf.topk_idx[:tokens].copy_(c['topk_idx'].cuda())
    buf.topk_weights[:tokens].copy_(c['topk_weights'].cuda())
    y = torch.full((tokens, HIDDEN), float('nan'), dtype=torch.bfloat16, device='cuda')
    return (lambda: dg.fp8_fp4_mega_moe(y, l1, l2, buf, **extra)), y


# rows per expert: all GEMMs swapped; split by group size (about 150); whole pair tiles and remainders (about 300)
CASES = [(8, 8, True), (300, 4, False), (300, 4, True), (600, 4, False), (600, 4, True)]


@pytest.mark.parametrize('tokens,experts,shared', CASES)
def test_an_sm_limit_holds(dg, tokens, experts, shared, tmp_path):
    call, y = _layer(dg, tokens, experts, shared)
    call()
    torch.cuda.synchronize()
    want = y.clone()
    gemms = lambda: [k for k in kernel_launches(call, tmp_path / 'trace.json') if 'gemm' in k[0]]
    assert len({k[1] for k in gemms()}) > 1, 'nothing runs on a side stream: the case no longer tests the limit'
    limit = 40
    dg.set_num_sms(limit)
    try:
        call()  # the profiler leaves launches alone that it has not seen the kernel of before
        y.fill_(float('nan'))
        launches = gemms()
    finally:
        dg.set_num_sms(0)
    assert len({k[1] for k in launches}) == 1 and max(k[2] for k in launches) <= limit
    assert torch.equal(y, want)
