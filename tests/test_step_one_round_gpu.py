"""fp32 launches whose units make one round of the staged kernel's warps and two of the ring kernel's: both sides of both
ends of that range. A launch in the range against the same blocks in two launches outside it, second moments included, and
against the oracle."""
import numpy as np
import pytest
import torch

from tests.test_step_chunks import _run
from tests.test_step_sources_gpu import _step
from tests.util import make_grad, make_param, reference_like_codebook

pytestmark = pytest.mark.gpu


def _units(device, which):
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    return {"two rounds of twelve": 12 * sms + 1, "one of sixteen": 16 * sms, "one of twelve": 12 * sms, "two of sixteen": 16 * sms + 1}[which]


@pytest.mark.parametrize("which", ["two rounds of twelve", "one of sixteen", "one of twelve", "two of sixteen"])
@pytest.mark.parametrize("period,blocks", [(2048, 1), (512, 4)])
def test_against_the_oracle(oracle, cuda_device, period, blocks, which):
    _run(oracle, cuda_device, _units(cuda_device, which) * blocks - blocks // 2, period, torch.float32, reference_like_codebook())


@pytest.mark.parametrize("which", ["two rounds of twelve", "one of sixteen"])
@pytest.mark.parametrize("period,blocks", [(2048, 1), (512, 4), (1992, 1), (1000, 2)])
@pytest.mark.parametrize("muon", [False, True])
def test_against_two_launches(cuda_device, period, blocks, which, muon):
    from gefen_b200 import _lib

    lib = _lib.load()
    ws = _lib.codebook_workspace(reference_like_codebook().to(cuda_device))
    nb = _units(cuda_device, which) * blocks
    n = nb * period

    def run(cuts):
        gen = torch.Generator().manual_seed(nb)
        one = {"g": make_grad((n,), 2, 0, 0), "p": make_param((n,), 2, 0), "codes": torch.randint(0, 256, (n,), dtype=torch.uint8, generator=gen),
               "mag": torch.rand(nb, generator=gen) * 2e-3, "v": torch.rand(nb, generator=gen) * 1e-6}
        one = {k: t.to(cuda_device) for k, t in one.items()}
        table = torch.empty(256, dtype=torch.uint8, device=cuda_device)
        for b0, b1 in zip(cuts, cuts[1:]):
            host = np.zeros(1, dtype=_lib.STEP_TENSOR_DTYPE)
            for k, t in one.items():
                host[k] = t[b0 if k in ("mag", "v") else b0 * period:].data_ptr()
            host["num_blocks"], host["period"], host["mag_dtype"], host["v_dtype"] = b1 - b0, period, _lib.F32, _lib.F32
            host["flags"] = _lib.STEP_MUON | _lib.STEP_NESTEROV if muon else _lib.STEP_FUSE_VMEAN | _lib.STEP_WEIGHT_DECAY
            for k, value in (("beta1", 0.9), ("beta2", 0.999), ("lr", 3e-4), ("bc1", 0.3), ("bc2", 0.003), ("eps", 1e-8), ("wd_mul", 0.99997)):
                host[k] = value
            _lib.check(lib.gefen_b200_multi_tensor_step(host.ctypes.data, _lib.ptr(table), 1, _lib.F32, _lib.ptr(ws), _lib.current_stream(cuda_device)))
            torch.cuda.synchronize()
        return one

    together, apart = run([0, nb]), run([0, nb // 2, nb])
    for k in together:
        assert torch.equal(together[k], apart[k]), k


@pytest.mark.parametrize("period,blocks", [(2048, 1), (512, 4)])
def test_copies_of_the_parameters(cuda_device, period, blocks):
    nb = _units(cuda_device, "one of sixteen") * blocks
    plain = _step(cuda_device, torch.float32, nb, period, 0, 0)
    got = _step(cuda_device, torch.float32, nb, period, 0, 2)
    for copy in got[0]:
        assert torch.equal(copy, plain[0][0])
    for a, b in zip(got[1:], plain[1:]):
        assert torch.equal(a, b)
