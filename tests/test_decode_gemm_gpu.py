"""The decode-sized GEMMs (of the FP8 x MXFP4 layer, and masked) against the oracle where the kernel's operand ring changes its layout:
experts just below and above the small token slots (16 and 80 rows), in every order, beside empty experts and experts of more
than one token tile; K extents shorter and longer than the ring. calc_diff <= 2e-3 (FP4 weights), per expert."""
import pytest
import torch

from oracle import gemm as ogemm
from oracle import moe as omoe
from oracle import quant
from tests.helpers import moe_case, quantize_groups

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    return deepgemm_b200


@pytest.mark.parametrize('rows', [
    [1, 16, 17, 2, 0, 40, 3, 16, 1, 170, 5, 15] + [1] * 20,  # about 9 rows per expert: slots of 16
    [80, 81, 1, 0, 79, 160, 2, 161, 64, 300, 80, 10],        # more: slots of 80
    [0, 0, 3],
], ids=['slots16', 'slots80', 'few'])
@pytest.mark.parametrize('hidden,inter', [(512, 256), (1280, 1152)])
def test_ring_layouts(dg, rows, hidden, inter):
    from deepgemm_b200 import _lib
    experts, tokens = len(rows), sum(rows)
    c = moe_case(tokens, hidden, inter, experts, 1, seed=tokens + hidden)
    idx = torch.repeat_interleave(torch.arange(experts), torch.tensor(rows))[torch.randperm(tokens)].view(tokens, 1)
    w = torch.rand(tokens, 1) + 0.5
    want = omoe.moe_layer(c['x_q'], c['x_sf'], idx, w, c['l1_q'], c['l1_sf'], c['l2_q'], c['l2_sf'])
    l1, l2 = dg.transform_weights_for_mega_moe(
        (c['l1_q'].cuda(), dg.transform_sf_into_required_layout(c['l1_sf'].cuda(), 2 * inter, hidden, (1, 32), experts)),
        (c['l2_q'].cuda(), dg.transform_sf_into_required_layout(c['l2_sf'].cuda(), hidden, inter, (1, 32), experts)))
    buf = dg.get_symm_buffer_for_mega_moe(None, experts, tokens, 1, hidden, inter)
    buf.x[:tokens].copy_(c['x_q'].cuda())
    buf.x_sf[:tokens].copy_(quant.pack_ue8m0(c['x_sf']).cuda())
    buf.topk_idx[:tokens].copy_(idx.cuda())
    buf.topk_weights[:tokens].copy_(w.cuda())
    y = torch.full((tokens, hidden), float('nan'), dtype=torch.bfloat16, device='cuda')
    _lib.check(_lib.lib().dgb200_set_tuning(b'swap_ab', 1))
    try:
        dg.fp8_fp4_mega_moe(y, l1, l2, buf)
        torch.cuda.synchronize()
    finally:
        _lib.check(_lib.lib().dgb200_set_tuning(b'swap_ab', -1))
    assert _lib.device_status()[0] == 0
    got = y.cpu()
    assert not torch.isnan(got.float()).any()
    per_expert = [quant.calc_diff(got[idx[:, 0] == e], want[idx[:, 0] == e]) for e in range(experts) if rows[e]]
    assert max(per_expert) <= 2e-3, per_expert


@pytest.mark.parametrize('expected,rows', [(5, [0, 1, 16, 17, 3, 0, 128, 2, 160, 8]), (64, [80, 0, 81, 1, 160, 161, 256, 129, 80, 300])])
@pytest.mark.parametrize('gran_a,gran_b,b_fp4', [(128, 32, True), (32, 32, True), (128, 128, False), (32, 128, False)])
@pytest.mark.parametrize('n,k', [(256, 384), (512, 1280)])
def test_masked(dg, expected, rows, gran_a, gran_b, b_fp4, n, k):
    """The masked GEMM on the same kernel: plain scale factors per 32 and per 128; rows past a group's count stay untouched and a
    count above the buffer is clipped."""
    from deepgemm_b200 import _lib
    max_m = 260
    torch.manual_seed(n + k + expected)
    a, b = torch.randn(len(rows), max_m, k).bfloat16(), (torch.randn(len(rows), n, k) * 0.02).bfloat16()
    (a_q, a_sf), (b_q, b_sf) = quantize_groups(a, gran_a, False), quantize_groups(b, gran_b, b_fp4)
    masked = torch.tensor(rows, dtype=torch.int32)
    want, mask = ogemm.grouped_gemm_masked(a_q, a_sf, b_q, b_sf, masked.clamp(max=max_m), gran_k_a=gran_a, gran_k_b=gran_b)
    d = torch.full((len(rows), max_m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    dg.m_grouped_fp8_fp4_gemm_nt_masked((a_q.cuda(), a_sf.cuda()), (b_q.cuda(), b_sf.cuda()), d, masked.cuda(), expected,
                                        recipe_a=(1, gran_a), recipe_b=(1, gran_b))
    got = d.cpu()
    assert _lib.device_status()[0] == 0
    assert torch.isnan(got.float())[~mask].all() and not torch.isnan(got.float())[mask].any()
    per_group = [quant.calc_diff(got[g][mask[g]], want[g][mask[g]]) for g in range(len(rows)) if rows[g]]
    assert max(per_group) <= (2e-3 if b_fp4 else 1e-3), per_group
