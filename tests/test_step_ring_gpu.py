"""The step kernel whose inputs arrive in shared memory by bulk copies and whose momenta wait in tensor memory: both sides
of its size limit, more units than warps, copies that start and end between 16-byte boundaries, and tables in which a
warp's next unit belongs to another tensor. Bit for bit against the oracle, or against the same tensors one by one."""
import numpy as np
import pytest
import torch

from tests.test_step_chunks import _codebooks, _run
from tests.test_step_kernels_gpu import _assert_codes, _state
from tests.util import make_grad, make_param, reference_like_codebook

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,nb,period", [
    (torch.bfloat16, 3, 6824), (torch.bfloat16, 3, 6832), (torch.float32, 3, 4096), (torch.float32, 3, 4104),     # chunks of 8
    (torch.float16, 3, 6820), (torch.float16, 3, 6828), (torch.float32, 3, 4092), (torch.float32, 3, 4100),       # of 4
    (torch.bfloat16, 3, 6822), (torch.bfloat16, 3, 6826), (torch.bfloat16, 3, 6825), (torch.bfloat16, 3, 6827),   # of 2 and 1
])
def test_largest_units(oracle, cuda_device, dtype, nb, period):
    _run(oracle, cuda_device, nb, period, dtype, reference_like_codebook())


# every warp of a full grid comes to several units; blocks of an odd number of chunks move the codes off 16 bytes
@pytest.mark.parametrize("dtype,nb,period", [(torch.bfloat16, 9001, 1032), (torch.float32, 9001, 520), (torch.float16, 200001, 24),
                                             (torch.bfloat16, 9001, 300), (torch.bfloat16, 70001, 27)])
def test_many_units(oracle, cuda_device, dtype, nb, period):
    _run(oracle, cuda_device, nb, period, dtype, reference_like_codebook())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset,periods", [(0, (8, 24, 64, 72, 512, 1000, 1024)), (0, (1032, 2048, 4000)), (4, (60, 12, 300, 512, 1500)),
                                            (1, (27, 63, 64))])
def test_tables_of_small_tensors(cuda_device, dtype, offset, periods):
    from gefen_b200 import _lib

    lib, tag = _lib.load(), _lib.dtype_tag(dtype)
    cb = reference_like_codebook().to(cuda_device)
    ws = _lib.codebook_workspace(cb)
    count = 300
    blocks = [1 + (7 * i) % 5 + (3000 if i % 97 == 0 else 0) for i in range(count)]
    shapes = [(nb, periods[i % len(periods)]) for i, nb in enumerate(blocks)]

    def state():
        flat = []
        for i, (nb, period) in enumerate(shapes):
            one = {"g": make_grad((nb, period), 3, i, 0, dtype), "p": make_param((nb, period), 3, i, dtype),
                   "codes": ((torch.arange(nb * period) * 37 + i) % 256).to(torch.uint8),
                   "mag": torch.full((nb,), 1e-3 + i * 1e-5).to(dtype), "v": torch.full((nb,), 1e-6).to(dtype)}
            flat.append({k: torch.cat([torch.zeros(offset, dtype=t.dtype), t.reshape(-1)]).to(cuda_device)[offset:] for k, t in one.items()})
        return flat

    def step(tensors, which):
        host = np.zeros(len(which), dtype=_lib.STEP_TENSOR_DTYPE)
        for r, i in enumerate(which):
            for k in ("g", "p", "codes", "mag", "v"):
                host[k][r] = tensors[i][k].data_ptr()
            host["num_blocks"][r], host["period"][r] = shapes[i]
            host["flags"][r] = _lib.STEP_FUSE_VMEAN | (_lib.STEP_WEIGHT_DECAY if i % 2 else 0)
        host["mag_dtype"] = host["v_dtype"] = tag
        for k, value in (("beta1", 0.9), ("beta2", 0.999), ("lr", 3e-4), ("bc1", 0.3), ("bc2", 0.003), ("eps", 1e-8), ("wd_mul", 0.99997)):
            host[k] = value
        table = torch.empty(host.nbytes, dtype=torch.uint8, device=cuda_device)
        _lib.check(lib.gefen_b200_multi_tensor_step(host.ctypes.data, _lib.ptr(table), len(which), tag, _lib.ptr(ws), _lib.current_stream(cuda_device)))
        torch.cuda.synchronize()

    together, alone = state(), state()
    for _ in range(2):
        step(together, list(range(count)))
        for i in range(count):
            step(alone, [i])
    for a, b in zip(together, alone):
        for k in a:
            assert torch.equal(a[k], b[k]), k


# blocks too long for the buffers, whose momenta are formed twice
@pytest.mark.parametrize("name", sorted(_codebooks()))
def test_codebooks_of_long_blocks(oracle, cuda_device, name):
    _run(oracle, cuda_device, 5, 8184, torch.bfloat16, _codebooks()[name])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("period,lr", [(8192, 1e-3), (8192, 0.0), (512, 1e-3), (300, 1e-3), (300, 0.0)])
def test_values_that_are_not_finite(oracle, cuda_device, dtype, period, lr):
    from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_fused_update_from_vmean_cuda

    cb = reference_like_codebook()
    p, g, codes, mag, v = _state(6, period, dtype, dtype, seed=9)
    g[1, 5], g[3, 7], g[4, 0], g[4, 9], g[5, period - 1] = (float(x) for x in ("nan", "inf", "-inf", "nan", "nan"))
    g[2].zero_()
    mag[2] = 0
    dp, dg, dc, dm, dv = (t.to(cuda_device) for t in (p, g, codes, mag, v))
    args = dict(beta1=0.9, lr=lr, bias_correction_1=0.1, bias_correction_2=0.001, eps=1e-8)
    oracle.automatic_gefen_fused_update_from_vmean(p, g, codes, mag, v, cb, False, **args)
    automatic_gefen_fused_update_from_vmean_cuda(dp, dg, dc, dm, dv, cb.to(cuda_device), False, **args)
    _assert_codes(dc, codes)
    assert torch.equal(dm.cpu(), mag)
    assert torch.equal(torch.nan_to_num(dp.cpu(), nan=7.0), torch.nan_to_num(p, nan=7.0))
