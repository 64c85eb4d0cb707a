"""The quantisers' paths for blocks that hold infinities or NaN, and for scales whose reciprocal is no ordinary number, against the
arithmetic they stand for: the block maximum passes over NaN, values are divided by the scale in FP32, E2M1 thresholds round
down, a NaN has code 0."""
import pytest
import torch

from oracle import quant

pytestmark = pytest.mark.gpu
INF, NAN = float('inf'), float('nan')


@pytest.fixture(scope='module')
def dg():
    import deepgemm_b200
    return deepgemm_b200


def _rows():
    torch.manual_seed(0)
    x = torch.randn(12, 512)
    x[1, 3], x[2, 40], x[3, 5], x[4, 100] = INF, -INF, NAN, -NAN
    x[5, 64:96] = NAN
    x[6, 7], x[6, 8] = INF, NAN
    x[7] = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0, -0.25, -0.75, -1.25, -1.75, -2.5, -3.5, -5.0, -6.0]).repeat(32)
    x[8] = -0.0
    x[9, ::2] = 0.0
    x[10] *= 1e-30
    x[11] *= 1e30
    return x.bfloat16()


def _amax(blocks):
    a = blocks.abs()
    return torch.where(a.isnan(), torch.zeros(()), a).amax(-1)


def _codes(q):
    mag = torch.zeros(q.shape, dtype=torch.int64)
    for t in quant.E2M1_THRESHOLDS:
        mag += q.abs() > t
    codes = (mag | ((q < 0) & (mag != 0)).long() << 3).to(torch.uint8).flatten(1)
    return (codes[:, 0::2] | (codes[:, 1::2] << 4)).view(torch.int8)


@pytest.mark.parametrize('gran', [32, 128])
def test_fp4(dg, gran):
    x = _rows()
    blocks = x.float().view(12, -1, gran)
    sf = quant.ue8m0_ceil(_amax(blocks).clamp(min=1e-4) / 6.0)
    q, got_sf = dg.utils.per_token_cast_to_fp4(x.cuda(), use_ue8m0=True, gran_k=gran)
    assert torch.equal(got_sf.cpu(), sf)
    assert torch.equal(q.cpu(), _codes(blocks * (1.0 / sf).unsqueeze(-1)))


@pytest.mark.parametrize('gran', [32, 128])
def test_fp8(dg, gran):
    x = _rows()
    blocks = x.float().view(12, -1, gran)
    sf = quant.ue8m0_ceil(_amax(blocks).clamp(min=1e-4) / 448.0)
    q, got_sf = dg.utils.per_token_cast_to_fp8(x.cuda(), use_ue8m0=True, gran_k=gran)
    assert torch.equal(got_sf.cpu(), sf)
    v = (blocks * (1.0 / sf).unsqueeze(-1)).flatten(1)
    want = v.clamp(-448.0, 448.0).to(torch.float8_e4m3fn)  # the conversion saturates
    finite = ~v.isnan()
    assert torch.equal(q.cpu().view(torch.uint8)[finite], want.view(torch.uint8)[finite])
    assert (q.cpu().float()[~finite].isnan()).all()


# 1e-13 and 1e-15: the scale itself has an ordinary reciprocal, the quotients of the 1e30 row overflow
@pytest.mark.parametrize('scale', [1.0 / 448, 0.00371, 1e-13, 1e-15, 1e-25, 1e-40, 1e22])
def test_nvfp4(dg, scale):
    x = _rows()
    s = torch.tensor(scale, dtype=torch.float32)
    blocks = x.float().view(12, -1, 16)
    sf = (_amax(blocks) / 6.0 / s).clamp(max=448.0).to(torch.float8_e4m3fn)
    factor = (sf.float() * s).unsqueeze(-1)
    want = _codes(torch.where(factor > 0, blocks / factor, torch.zeros(())))
    q, got_sf, _ = dg.per_token_cast_to_nvfp4(x.cuda(), s.cuda())
    assert torch.equal(got_sf.cpu().view(torch.uint8), sf.view(torch.uint8))
    assert torch.equal(q.cpu(), want)
