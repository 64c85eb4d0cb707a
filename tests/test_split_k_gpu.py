"""The dense GEMMs with a tile's K split over a cluster, against the oracle: fewer rows than a tile and a little more than one,
K parts of unequal length, both tile widths (the wide one from 10 tiles on), FP32 outputs with and without an accumulator input.
Every call must have run the split form. Tolerances as for the
unsplit kernel: calc_diff <= 2e-3 (FP4 weights), <= 1e-3 (FP8 x FP8), < 1e-5 (BF16)."""
import pytest
import torch

from oracle import quant
from tests.helpers import gemm_kernels_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    return deepgemm_b200


@pytest.fixture(params=[2, 4, 8])
def split(request):
    from deepgemm_b200 import _lib
    _lib.check(_lib.lib().dgb200_set_tuning(b'split_k', request.param))
    yield request.param
    _lib.check(_lib.lib().dgb200_set_tuning(b'split_k', -1))
    assert _lib.device_status()[0] == 0


@pytest.mark.parametrize('m,n,k,block_n', [(1, 128, 4096, 128), (17, 256, 4224, 128), (128, 384, 8192, 128), (129, 512, 4992, 128),
                                           (200, 256, 5120, 128), (100, 2560, 4096, 256), (130, 1536, 4224, 256)])
@pytest.mark.parametrize('kind', ['bf16', 'fp8xfp8', 'fp8xfp4'])
def test_split_k(dg, split, m, n, k, block_n, kind):
    torch.manual_seed(m + n + k)
    a, b = torch.randn(m, k).bfloat16(), (torch.randn(n, k) * 0.02).bfloat16()
    if kind == 'bf16':
        want, tol = a.double() @ b.double().T, 1e-5
        run = lambda d, c=None: dg.bf16_gemm_nt(a.cuda(), b.cuda(), d, c)
    else:
        fp4 = kind == 'fp8xfp4'
        gran_a, gran_b = (128, 32) if fp4 else (32, 128)
        a_q, a_sf = quant.quantize_fp8_per_token(a, gran_a)
        b_q, b_sf = (quant.quantize_fp4_per_token if fp4 else quant.quantize_fp8_per_token)(b, gran_b)
        b_f = quant.dequantize_fp4(b_q, b_sf, gran_b) if fp4 else quant.dequantize_fp8(b_q, b_sf, gran_b)
        want, tol = quant.dequantize_fp8(a_q, a_sf, gran_a).double() @ b_f.double().T, 2e-3 if fp4 else 1e-3
        run = lambda d, c=None: dg.fp8_fp4_gemm_nt((a_q.cuda(), a_sf.cuda()), (b_q.cuda(), b_sf.cuda()), d, c, recipe_a=(1, gran_a),
                                                   recipe_b=(1, gran_b))
    d = torch.full((m, n), float('nan'), dtype=torch.bfloat16, device='cuda')
    assert gemm_kernels_of(lambda: run(d)) == {(block_n, False, True)}
    assert quant.calc_diff(d.cpu(), want) <= tol
    f = torch.full((m, n), float('nan'), dtype=torch.float32, device='cuda')
    assert gemm_kernels_of(lambda: run(f)) == {(block_n, False, True)}
    # FP32 partial sums of K products each: the relative error is far below the BF16 bound
    assert quant.calc_diff(f.cpu(), want) <= 1e-8
    c = torch.randn(m, n, device='cuda')
    out = torch.full_like(c, float('nan'))
    run(out, c)
    assert quant.calc_diff(out.cpu().double() - c.cpu().double(), want) <= 1e-8
    again = torch.full_like(f, float('nan'))
    run(again)
    assert torch.equal(f, again), 'the order of the sums is fixed'


@pytest.mark.parametrize('m,n,k,form', [(128, 7168, 16384, (256, False, True)), (33, 1536, 7168, (128, False, True)),
                                        (8, 1024, 2048, (128, False, True)), (128, 4096, 1024, (256, False, False))])
def test_the_rule_splits_by_itself(dg, m, n, k, form):
    """Without the knob: long K and few tiles split, short K does not."""
    a, b = torch.randn(m, k, device='cuda').bfloat16(), torch.randn(n, k, device='cuda').bfloat16()
    d = torch.empty(m, n, dtype=torch.bfloat16, device='cuda')
    assert gemm_kernels_of(lambda: dg.bf16_gemm_nt(a, b, d)) == {form}


def test_rows_do_not_depend_on_the_batch_without_the_split(dg):
    """With split_k 0 a row's bits are the same in every batch: K is summed in one order whatever the tile."""
    from deepgemm_b200 import _lib
    torch.manual_seed(3)
    n, k = 1536, 7168
    a, b = torch.randn(1000, k, device='cuda').bfloat16(), torch.randn(n, k, device='cuda').bfloat16()
    _lib.check(_lib.lib().dgb200_set_tuning(b'split_k', 0))
    try:
        outs = []
        for m in (1, 33, 128, 129, 300, 1000):
            d = torch.empty(m, n, dtype=torch.float32, device='cuda')
            dg.bf16_gemm_nt(a[:m], b, d)
            outs.append(d)
    finally:
        _lib.check(_lib.lib().dgb200_set_tuning(b'split_k', -1))
    assert all(torch.equal(d, outs[-1][:d.size(0)]) for d in outs)
