"""Several launches of one step overlap; what the program launches next does not. Steps of tables that need every kernel of
the library, each followed at once by products that take tensor memory and start programmatically, against the same calls
with the device idle in between: the same bits."""
import numpy as np
import pytest
import torch

from tests.util import make_grad, make_param, reference_like_codebook

pytestmark = pytest.mark.gpu

# (blocks, period, kind): rows of one kind of launch lie together, and the last row has no blocks
ROWS = [(300, 2048, "fuse"), (7, 1032, "fuse"), (5000, 64, "fuse"), (90, 300, "fuse"), (3, 8192, "fuse"), (2, 10000, "fuse"),
        (40, 256, "one"), (2000, 520, "fuse"), (12, 27, "fuse"), (0, 2048, "fuse")]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_launches_of_a_step_and_products_after_it(cuda_device, dtype):
    from gefen_b200 import _lib
    from gefen_b200 import newton_schulz as ns

    lib, tag = _lib.load(), _lib.dtype_tag(dtype)
    ws = _lib.codebook_workspace(reference_like_codebook().to(cuda_device))
    matrix = torch.randn(300, 500, generator=torch.Generator().manual_seed(1)).to(cuda_device)

    def run(idle):
        tensors, host = [], np.zeros(len(ROWS), dtype=_lib.STEP_TENSOR_DTYPE)
        for r, (nb, period, kind) in enumerate(ROWS):
            n = max(nb, 1) * period
            one = {"g": make_grad((n,), 5, r, 0, dtype), "p": make_param((n,), 5, r, dtype), "codes": (torch.arange(n) * 37 % 256).to(torch.uint8),
                   "mag": torch.full((max(nb, 1),), 1e-3), "v": torch.full((n if kind == "one" else max(nb, 1),), 1e-6)}
            tensors.append({k: t.to(cuda_device) for k, t in one.items()})
            for k, t in tensors[-1].items():
                host[k][r] = t.data_ptr()
            host["num_blocks"][r], host["period"][r] = nb, period
            host["flags"][r] = _lib.STEP_PERIOD1 if kind == "one" else _lib.STEP_FUSE_VMEAN
        host["mag_dtype"] = host["v_dtype"] = _lib.F32
        for k, value in (("beta1", 0.9), ("beta2", 0.999), ("lr", 3e-4), ("bc1", 0.3), ("bc2", 0.003), ("eps", 1e-8), ("wd_mul", 1.0)):
            host[k] = value
        table = torch.empty(host.nbytes, dtype=torch.uint8, device=cuda_device)
        out = []
        for _ in range(10):
            _lib.check(lib.gefen_b200_multi_tensor_step(host.ctypes.data, _lib.ptr(table), len(ROWS), tag, _lib.ptr(ws),
                                                        _lib.current_stream(cuda_device)))
            if idle:
                torch.cuda.synchronize()
            out.append(ns.zeropower_via_newtonschulz(matrix, (3.4445, -4.7750, 2.0315), 5, 1e-7).clone())
            if idle:
                torch.cuda.synchronize()
        _lib.check_step_status(cuda_device)
        ns.check_status(cuda_device)
        return [t for one in tensors for t in one.values()] + out

    for a, b in zip(run(False), run(True)):
        assert torch.equal(a, b)
