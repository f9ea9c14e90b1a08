"""Waits of the step kernels that run out, kernel by kernel: nothing is half done, the status says so, and the next call
works. The waits run out because they are granted no polls; nothing faults, traps or hangs."""
import pytest
import torch

from tests.util import make_grad, make_param, reference_like_codebook

pytestmark = pytest.mark.gpu


@pytest.fixture
def limits():
    from gefen_b200 import _lib

    lib = _lib.load()
    set_limit = {"tables": lib.gefen_b200_debug_set_stage_spin_limit, "inputs": lib.gefen_b200_debug_set_input_spin_limit}
    yield lambda wait, limit: _lib.check(set_limit[wait](limit))
    for one in set_limit.values():
        _lib.check(one(-1))


def _call(device, dtype, nb, period, kind):
    from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_step_cuda

    gen = torch.Generator().manual_seed(nb)
    p = make_param((nb, period), 1, 0, dtype).to(device)
    g = make_grad((nb, period), 1, 0, 0, dtype).to(device)
    codes = torch.randint(0, 256, (nb, period), dtype=torch.uint8, generator=gen).to(device)
    mag = (torch.rand(nb, 1, generator=gen) * 2e-3).to(device)
    v = (torch.rand(nb * period if kind == "one" else nb, 1, generator=gen) * 1e-6 + 1e-9).to(device)
    cb = reference_like_codebook().to(device)

    def step():
        automatic_gefen_step_cuda(p, g, codes, mag, v, cb, kind == "one", 0.9, 0.999, 3e-4, 0.99997, 0.1, 0.001, 1e-8)
        torch.cuda.synchronize()   # the kernel came back by itself
        return [t.clone() for t in (p, codes, mag, v)]

    return step, [t.clone() for t in (p, codes, mag, v)]


# the ring kernel (whole-warp and shared-warp blocks, small chunks, more units than warps, a single one)
RING = [(torch.bfloat16, 64, 2048, ""), (torch.float32, 30001, 512, ""), (torch.bfloat16, 9001, 1032, ""), (torch.bfloat16, 90, 300, ""),
        (torch.float16, 50, 27, ""), (torch.float32, 1, 8, "")]
# momenta formed twice, staged (one round of sixteen warps per SM), one-element moments in registers, the generic kernel by
# warp (float64) and by CTA
OTHERS = [(torch.bfloat16, 3, 8192, ""), (torch.float32, 9001, 512, ""), (torch.bfloat16, 40, 256, "one"), (torch.float64, 33, 768, ""), (torch.bfloat16, 2, 10007, "")]


@pytest.mark.parametrize("wait,dtype,nb,period,kind", [("inputs",) + c for c in RING] + [("tables",) + c for c in RING + OTHERS])
def test_wait_runs_out(cuda_device, limits, wait, dtype, nb, period, kind):
    from gefen_b200 import _lib

    step, before = _call(cuda_device, dtype, nb, period, kind)
    assert _lib.step_status(cuda_device) == 0
    limits(wait, 0)
    for was, now in zip(before, step()):
        assert torch.equal(was, now)
    with pytest.raises(_lib.GefenB200Error, match="gave up waiting"):
        _lib.check_step_status(cuda_device)
    limits(wait, -1)
    after = step()
    assert _lib.step_status(cuda_device) == 0
    again, _ = _call(cuda_device, dtype, nb, period, kind)   # the same call without a time-out before it
    for a, b in zip(after, again()):
        assert torch.equal(a, b)
    assert not torch.equal(before[1], after[1])


@pytest.mark.parametrize("dtype,nb,period,kind", OTHERS)
def test_other_kernels_wait_for_no_inputs(cuda_device, limits, dtype, nb, period, kind):
    from gefen_b200 import _lib

    step, before = _call(cuda_device, dtype, nb, period, kind)
    limits("inputs", 0)
    assert not torch.equal(before[1], step()[1])
    assert _lib.step_status(cuda_device) == 0
