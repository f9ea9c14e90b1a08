"""The cap on the warps of a CTA (GEFEN_B200_STEP_WARPS, read once by a process): with one to three warps the buffers of the
ring kernel lie where eighteen warps keep their descriptors. The same bits as without it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import hashlib, torch
from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_fused_update_from_vmean_cuda
from tests.util import make_grad, make_param, reference_like_codebook
for dtype, nb, period in [(torch.bfloat16, 900, 2048), (torch.float32, 700, 512), (torch.bfloat16, 3000, 300), (torch.float32, 9, 64)]:
    gen = torch.Generator().manual_seed(nb)
    one = [make_param((nb, period), 1, 0, dtype), make_grad((nb, period), 1, 0, 0, dtype),
           torch.randint(0, 256, (nb, period), dtype=torch.uint8, generator=gen), torch.full((nb, 1), 1e-3, dtype=dtype),
           torch.full((nb, 1), 1e-6, dtype=dtype)]
    one = [t.cuda() for t in one]
    for _ in range(2):
        automatic_gefen_fused_update_from_vmean_cuda(*one, reference_like_codebook().cuda(), False, 0.9, 3e-4, 0.1, 0.001, 1e-8)
    for t in one:
        print(hashlib.sha1(t.cpu().view(torch.uint8).numpy().tobytes()).hexdigest())
"""


def test_capped_warps(cuda_device):
    def run(**env):
        return subprocess.run([sys.executable, "-c", SCRIPT], env={**os.environ, **env}, capture_output=True, text=True, check=True, timeout=300,
                              cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__)))).stdout

    plain = run()
    assert len(plain.split()) == 20
    for warps in ("1", "3"):
        assert run(GEFEN_B200_STEP_WARPS=warps) == plain
