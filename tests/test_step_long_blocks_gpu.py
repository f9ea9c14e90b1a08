"""Blocks of 2048 to 8192 elements (from 6832, fp32 4104, the step forms their momenta twice): the longest ones, every codebook density, values that are not finite, lr = 0 and GefenMuon's momentum, against the oracle
bit for bit."""
import pytest
import torch

from tests.test_step_chunks import _codebooks, _run
from tests.test_step_kernels_gpu import _assert_codes, _state
from tests.util import reference_like_codebook

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nb,period", [(9, 2048), (4, 2056), (5, 3072), (1, 3080), (7, 4096), (3, 6152), (2, 8184), (161, 8192)])
def test_long_blocks(oracle, cuda_device, dtype, nb, period):
    _run(oracle, cuda_device, nb, period, dtype, reference_like_codebook())


@pytest.mark.parametrize("name", sorted(_codebooks()))
def test_codebooks(oracle, cuda_device, name):
    _run(oracle, cuda_device, 5, 4104, torch.bfloat16, _codebooks()[name])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lr", [0.0, 1e-3])
def test_values_that_are_not_finite(oracle, cuda_device, dtype, lr):
    from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_fused_update_from_vmean_cuda

    cb = reference_like_codebook()
    p, g, codes, mag, v = _state(6, 4096, dtype, dtype, seed=8)
    g[1, 5], g[3, 7], g[4, 0], g[4, 9], g[5, 4095] = (float(x) for x in ("nan", "inf", "-inf", "nan", "nan"))
    g[2].zero_()
    mag[2] = 0
    dp, dg, dc, dm, dv = (t.to(cuda_device) for t in (p, g, codes, mag, v))
    args = dict(beta1=0.9, lr=lr, bias_correction_1=0.1, bias_correction_2=0.001, eps=1e-8)
    oracle.automatic_gefen_fused_update_from_vmean(p, g, codes, mag, v, cb, False, **args)
    automatic_gefen_fused_update_from_vmean_cuda(dp, dg, dc, dm, dv, cb.to(cuda_device), False, **args)
    _assert_codes(dc, codes)
    assert torch.equal(dm.cpu(), mag)
    assert torch.equal(torch.nan_to_num(dp.cpu(), nan=7.0), torch.nan_to_num(p, nan=7.0))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nb,period", [(3, 4096), (2, 8192)])
def test_momentum(oracle, cuda_device, dtype, nb, period):
    from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_muon_momentum_cuda

    cb = reference_like_codebook()
    _, g, codes, mag, _ = _state(nb, period, dtype, dtype, seed=period)
    out = torch.empty_like(g)
    dg, dc, dm = (t.to(cuda_device) for t in (g, codes, mag))
    dout = torch.empty_like(dg)
    for _ in range(2):
        oracle.automatic_gefen_muon_momentum(g, codes, mag, cb, out, False, 0.95)
        automatic_gefen_muon_momentum_cuda(dg, dc, dm, cb.to(cuda_device), dout, False, 0.95)
        _assert_codes(dc, codes)
        assert torch.equal(dm.cpu(), mag) and torch.equal(dout.cpu(), out)
