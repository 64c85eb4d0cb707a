"""The decode-sized GEMMs of the FP8 x MXFP4 layer against the layer oracle where the kernel's operand ring changes its layout:
experts just below and above the small token slots (16 and 64 rows), in every order, beside empty experts and experts of more
than one token tile; K extents shorter and longer than the ring. calc_diff <= 2e-3 (FP4 weights), per expert."""
import pytest
import torch

from oracle import moe as omoe
from oracle import quant
from tests.helpers import moe_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    return deepgemm_b200


@pytest.mark.parametrize('rows', [
    [1, 16, 17, 2, 0, 40, 3, 16, 1, 170, 5, 15] + [1] * 20,  # about 9 rows per expert: slots of 16
    [64, 65, 1, 0, 63, 160, 2, 161, 64, 300, 64, 10],        # more: slots of 64
    [0, 0, 3],
], ids=['slots16', 'slots64', 'few'])
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
