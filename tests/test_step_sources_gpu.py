"""The step with gradients averaged over several buffers (here: the same buffer on this GPU, given once or several times)
and parameters stored to further copies against the plain step of the same gradients: bit for bit, second moments
included, whatever kernel the blocks' length and alignment choose."""
import numpy as np
import pytest
import torch

from tests.util import make_grad, make_param, reference_like_codebook

pytestmark = pytest.mark.gpu


def _step(device, dtype, nb, period, sources, copies, steps=2, wd=0.1):
    """Parameters (all copies), codes, magnitudes and second moments after `steps` steps."""
    from gefen_b200 import _lib

    lib = _lib.load()
    n = nb * period
    pad = (n + 127) // 128 * 128     # a copy starts on a multiple of 16 bytes behind the first
    params = torch.zeros(1 + copies, pad, dtype=dtype, device=device)
    params[:, :n] = make_param((n,), period, 0, dtype).to(device)
    gen = torch.Generator().manual_seed(nb)
    codes = torch.randint(0, 256, (n,), dtype=torch.uint8, generator=gen).to(device)
    mag = (torch.rand(nb, generator=gen) * 2e-3).to(device)
    v = (torch.rand(nb, generator=gen) * 1e-6 + 1e-7).to(device)
    cb = reference_like_codebook().to(device)
    ws = _lib.codebook_workspace(cb)
    rows = np.zeros(1, dtype=_lib.STEP_TENSOR_DTYPE)
    table = torch.empty(rows.nbytes, dtype=torch.uint8, device=device)
    peers = np.array([(r + 1) * pad * params.element_size() for r in range(copies)], dtype=np.int64)
    grads = np.zeros(max(sources, 1), dtype=np.int64)
    for step in range(steps):
        # 8 significant bits (fp16: 11): the sum of up to eight equal values takes three more, exact in fp32
        g = make_grad((nb, period), period, 0, step, dtype if dtype == torch.float16 else torch.bfloat16).to(dtype).to(device)
        rows["p"], rows["g"], rows["codes"], rows["mag"], rows["v"] = (t.data_ptr() for t in (params, g, codes, mag, v))
        rows["num_blocks"], rows["period"], rows["mag_dtype"], rows["v_dtype"] = nb, period, _lib.F32, _lib.F32
        rows["flags"] = _lib.STEP_FUSE_VMEAN | (_lib.STEP_WEIGHT_DECAY if wd else 0)
        for key, value in (("beta1", 0.9), ("beta2", 0.999), ("lr", 3e-4), ("bc1", 0.3), ("bc2", 0.003), ("eps", 1e-8),
                           ("wd_mul", 1 - 3e-4 * wd)):
            rows[key] = value
        _lib.check(lib.gefen_b200_multi_tensor_step_peers(
            rows.ctypes.data, _lib.ptr(table), 1, _lib.dtype_tag(dtype), _lib.ptr(ws), peers.ctypes.data if copies else None, copies,
            grads.ctypes.data if sources else None, sources, 1.0 / max(sources, 1), _lib.current_stream(device)))
    torch.cuda.synchronize()
    return params[:, :n].clone(), codes, mag, v


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nb,period", [(6, 2048), (37, 512), (65, 64), (5, 1664),
                                       (9, 300), (5, 1500), (33, 12), (11, 514), (33, 18), (21, 147), (50, 27), (3, 2047),
                                       (2, 8188), (2, 8191), (3, 4096), (2, 8192)])
def test_averaged_gradients_and_copies(cuda_device, dtype, nb, period):
    plain = _step(cuda_device, dtype, nb, period, 0, 0)
    # powers of two: the average of equal gradients is the gradient itself
    for sources, copies in ((1, 0), (2, 0), (4, 1), (8, 3), (0, 2)):
        got = _step(cuda_device, dtype, nb, period, sources, copies)
        for copy in got[0]:
            assert torch.equal(copy, plain[0][0]), (sources, copies)
        for a, b in zip(got[1:], plain[1:]):
            assert torch.equal(a, b), (sources, copies)
