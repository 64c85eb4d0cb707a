"""Router and dispatch plan around the size up to which one CTA makes both: bit-exact against the oracle for either kernel, logits
with ties, signed zeros, infinities and NaN included."""
import pytest
import torch

from oracle import moe as omoe
from oracle import quant

pytestmark = pytest.mark.gpu
SEGMENT = 128


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    return deepgemm_b200


@pytest.mark.parametrize('tokens,experts,topk', [(1, 1, 1), (3, 300, 5), (128, 64, 8), (129, 64, 8), (31, 768, 32), (31, 769, 32), (32, 40, 32), (33, 40, 32), (600, 513, 3)])
def test_route_and_plan(dg, tokens, experts, topk):
    from deepgemm_b200 import _lib
    hidden, inter = 256, 128
    torch.manual_seed(tokens + experts)
    logits = (torch.randn(tokens, experts) * 4).round() / 4  # many ties
    logits[0, experts // 2] = -0.0
    want_idx, want_w = omoe.route_sigmoid_topk(logits, topk)
    w1 = torch.zeros(experts, 2 * inter, hidden // 2, dtype=torch.int8, device='cuda')
    w2 = torch.zeros(experts, hidden, inter // 2, dtype=torch.int8, device='cuda')
    s1 = dg.transform_sf_into_required_layout(torch.ones(experts, 2 * inter, hidden // 32, device='cuda'), 2 * inter, hidden, (1, 32), experts)
    s2 = dg.transform_sf_into_required_layout(torch.ones(experts, hidden, inter // 32, device='cuda'), hidden, inter, (1, 32), experts)
    l1, l2 = dg.transform_weights_for_mega_moe((w1, s1), (w2, s2))
    buf = dg.get_symm_buffer_for_mega_moe(None, experts, tokens, topk, hidden, inter)
    lay = buf.layout
    word = lambda name, n: buf.buffer[lay[name]:lay[name] + 4 * n].view(torch.int32)
    stats = torch.full((experts,), 7, dtype=torch.int32, device='cuda')
    y = torch.empty(tokens, hidden, dtype=torch.bfloat16, device='cuda')
    x = torch.randn(tokens, hidden, device='cuda').bfloat16()
    word('src_of_row', lay['max_rows']).fill_(12345)  # what an earlier call with more rows left
    dg.fp8_fp4_mega_moe_bf16_input(y, x, l1, l2, buf, logits=logits.cuda(), cumulative_local_expert_recv_stats=stats)
    assert _lib.device_status()[0] == 0
    assert torch.equal(buf.topk_idx[:tokens].cpu(), want_idx)
    assert (buf.topk_weights[:tokens].cpu() - want_w).abs().max() <= 1e-6
    dest, src, start, end = omoe.dispatch_plan(want_idx, experts, SEGMENT)
    assert torch.equal(word('dest_row', tokens * topk).cpu(), dest)
    assert torch.equal(word('expert_start', experts).cpu(), start) and torch.equal(word('expert_end', experts).cpu(), end)
    assert torch.equal(word('src_of_row', src.numel()).cpu(), src)
    assert torch.equal(stats.cpu(), 7 + end - start)
    rows = src >= 0
    got_w = buf.buffer[lay['row_weight']:lay['row_weight'] + 4 * src.numel()].view(torch.float32).cpu()
    assert torch.equal(got_w[rows], buf.topk_weights[:tokens].cpu().reshape(-1)[src[rows].long()])
    # the caller's own routes, masked slots and ids that are no expert among them
    own = want_idx.clone()
    own[::2, 0] = -1
    own[-1, -1] = experts + 5
    buf.topk_idx[:tokens].copy_(own.cuda())
    dg.fp8_fp4_mega_moe_bf16_input(y, x, l1, l2, buf)
    dest, src, start, end = omoe.dispatch_plan(own, experts, SEGMENT)
    assert torch.equal(word('dest_row', tokens * topk).cpu(), dest) and torch.equal(word('expert_end', experts).cpu(), end)
    assert torch.equal(word('src_of_row', src.numel()).cpu(), src)
    assert _lib.device_status()[0] == 0


def test_route_of_special_logits(dg):
    inf, nan = float('inf'), float('nan')
    rows = [[1.0, inf, 2.0, -inf, nan, 0.0, -0.0, 3.0], [-inf] * 8, [nan] * 8, [-1.0, -1.0, nan, -inf, -2.0, -1.0, -inf, -3.0],
            [0.0, -0.0, -0.0, 0.0, -5.0, -5.0, -6.0, -7.0]]
    idx, w = dg.route_sigmoid_topk(torch.tensor(rows, device='cuda'), 4)
    none = 0x7fffffff  # no logit above -infinity is left
    assert idx.cpu().tolist() == [[1, 7, 2, 0], [none] * 4, [none] * 4, [0, 1, 5, 4], [0, 1, 2, 3]]
    s = torch.sigmoid(torch.tensor([inf, 3.0, 2.0, 1.0]))
    assert (w[0].cpu() - s / s.sum()).abs().max() <= 1e-6
