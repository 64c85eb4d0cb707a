"""The layer's GEMMs that run side by side on the library's own streams: which launches do, what an SM limit makes of them, CUDA
graphs, and callers on several streams at once. The bits never depend on where a GEMM ran."""
import os
import subprocess
import sys
import threading

import pytest
import torch

from oracle import quant
from tests.helpers import kernel_launches, moe_case, quantize_groups

pytestmark = pytest.mark.gpu
HIDDEN, INTER, TOPK = 512, 256, 2
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


# rows per expert: all GEMMs swapped; split by group size (about 150); whole pair tiles and remainders (about 300, so few experts only
# with the knob)
CASES = [(8, 8, True), (300, 4, False), (300, 4, True), (600, 4, False), (600, 4, True)]


@pytest.fixture(autouse=True)
def _pairs_and_remainders():
    from deepgemm_b200 import _lib
    _lib.check(_lib.lib().dgb200_set_tuning(b'pair', 1))
    yield
    _lib.check(_lib.lib().dgb200_set_tuning(b'pair', -1))


@pytest.mark.parametrize('tokens,experts,shared', CASES)
def test_an_sm_limit_holds(dg, tokens, experts, shared):
    call, y = _layer(dg, tokens, experts, shared)
    call()
    torch.cuda.synchronize()
    want = y.clone()
    streams = set()
    for _ in range(5):  # the profiler may miss some launches
        streams |= {stream for _, stream, _ in kernel_launches(call, 'gemm_kernel')}
    assert len(streams) > 1, 'nothing runs on a side stream: the case no longer tests the limit'
    limit = 40
    dg.set_num_sms(limit)
    try:
        y.fill_(float('nan'))
        launches = kernel_launches(call, 'gemm_kernel')
    finally:
        dg.set_num_sms(0)
    assert len({stream for _, stream, _ in launches}) == 1 and max(ctas for _, _, ctas in launches) <= limit
    assert torch.equal(y, want)


@pytest.mark.parametrize('tokens,experts,shared', CASES)
def test_inside_a_cuda_graph(dg, tokens, experts, shared):
    call, y = _layer(dg, tokens, experts, shared)
    call()
    torch.cuda.synchronize()
    want = y.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for _ in range(2):
        y.fill_(float('nan'))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


def test_first_call_of_a_process_inside_a_capture():
    """The side streams and their events are made while the caller's stream is being captured."""
    code = ('import torch, deepgemm_b200 as dg\n'
            'from deepgemm_b200 import _lib\n'
            'from tests.test_side_streams_gpu import _layer\n'
            '_lib.check(_lib.lib().dgb200_set_tuning(b"pair", 1))\n'
            'call, y = _layer(dg, 600, 4, True)\n'
            'torch.cuda.synchronize()\n'
            'graph = torch.cuda.CUDAGraph()\n'
            'with torch.cuda.graph(graph):\n'
            '    call()\n'
            'graph.replay()\n'
            'torch.cuda.synchronize()\n'
            'replayed = y.clone()\n'
            'y.fill_(float("nan"))\n'
            'call()\n'
            'torch.cuda.synchronize()\n'
            'assert torch.equal(y, replayed) and not y.isnan().any()\n')
    done = subprocess.run([sys.executable, '-c', code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


def test_two_threads_on_two_streams(dg):
    """Two callers share the side streams: their forks and joins must not mix. One layer of each kind of split."""
    layers = [_layer(dg, 600, 4, True, seed=11), _layer(dg, 300, 4, True, seed=12)]
    want = []
    for call, y in layers:
        call()
        torch.cuda.synchronize()
        want.append(y.clone())
        y.fill_(float('nan'))
    got, errors = [[], []], []

    def work(i):
        try:
            call, y = layers[i]
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(20):
                    call()
                    got[i].append(y.clone())
                    y.fill_(float('nan'))
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for i in range(2):
        assert len(got[i]) == 20 and all(torch.equal(y, want[i]) for y in got[i])
