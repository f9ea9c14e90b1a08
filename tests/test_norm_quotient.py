"""The quotient of a matrix by its norm: the IEEE quotient, also where it is taken through the norm's reciprocal."""
import subprocess
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def test_every_pair_of_bf16_values(tmp_path):
    exe = tmp_path / "sweep"
    subprocess.run(["/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++", "-O2", "-fopenmp", "-ffp-contract=off", "-mfma", "-mavx2",
                    "-std=c++17", "-o", str(exe), str(ROOT / "tests" / "native" / "norm_divider_sweep.cpp")], check=True)
    bad, checked, reciprocal = (int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0
    assert checked > 1_000_000_000 and 200_000_000 < reciprocal < checked


# norms given by eps, which the matrix stays below: the ends of the range of the reciprocal (2^-100, 2^100), values between
# powers of two, the usual one
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("eps", [2.0 ** -101, 2.0 ** -100 * 0.996, 2.0 ** -100, 2.0 ** -100 * 1.008, 1e-25, 1e-7, 0.7, 1.0, 3.0, 1.9921875, 1e9, 1e18,
                                 2.0 ** 99 * 1.9921875, 2.0 ** 100, 2.0 ** 100 * 1.008, 2.0 ** 120])
def test_against_torch_on_the_gpu(cuda_device, dtype, eps):
    from gefen_b200 import newton_schulz as ns

    norm = torch.tensor(eps).bfloat16().float()
    gen = torch.Generator().manual_seed(1)
    for shape in ((64, 512), (72, 33), (513, 24)):   # wide and unpadded, padded, tall
        n = shape[0] * shape[1]
        # mantissas of 8 bits over all scales below the norm that leave its sum of squares alone; values around the least
        # that takes the reciprocal; zeros and the smallest subnormals
        top = min(float(norm) * 2.0 ** -14, 2.0 ** 50)
        v = (1 + torch.rand(n, generator=gen)) * top * torch.exp2(-torch.randint(0, 120, (n,), generator=gen).float())
        edge = 1e-18 * max(float(norm), 1.0)
        if edge < top:
            v[::7] = edge * (1 + (torch.rand(v[::7].numel(), generator=gen) - 0.5) / 16)
        v[::11], v[5::101] = 0.0, 9.2e-41
        v = (v * (torch.randint(0, 2, (n,), generator=gen) * 2 - 1)).bfloat16().reshape(shape)
        got = ns.zeropower_via_newtonschulz(v.to(cuda_device, dtype), (3.4445, -4.7750, 2.0315), 0, eps)
        want = (v.to(cuda_device).float() / norm.to(cuda_device)).bfloat16()
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), shape
