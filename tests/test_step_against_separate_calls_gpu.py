"""Whole steps (one table, or one call per tensor) against the separate entry points: second moment, weight decay by torch,
and the update from the second moment. Codes and magnitudes do not depend on the second moment and are the same bits. It is
added up in another order there, so parameters may differ by what one rounding of a block's second moment moves: 2^-9 of an
update of lr at most for the types of 8 and 11 bits, a hundredth of the bound (1e-4 of the parameters, relative L2)."""
import pytest
import torch

from gefen_b200 import workloads
from tests.util import rel_l2

pytestmark = pytest.mark.gpu


class Separate:
    """One tensor stepped with the separate entry points, from a zero state."""

    def __init__(self, p, period, divisor, state_dtype):
        n, device = p.numel(), p.device
        self.period, self.divisor, self.t = period, divisor, 0
        self.codes = torch.zeros(n // period, period, dtype=torch.uint8, device=device)
        self.mag = torch.zeros(n // (divisor if period == 1 else period), 1, dtype=state_dtype, device=device)
        self.v = torch.zeros(n // period, 1, dtype=state_dtype, device=device)

    def step(self, p, g, codebook, lr, wd):
        from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_fused_update_from_vmean_cuda, automatic_gefen_period1_update_cuda
        from gefen_b200.kernels.automatic_vmean import automatic_vmean_update_cuda

        self.t += 1
        bc1, bc2 = 1 - 0.9 ** self.t, 1 - 0.999 ** self.t
        if self.period != 1:
            automatic_vmean_update_cuda(self.v, g.reshape(-1, self.period), 0.999)
        if wd:
            p.mul_(1 - lr * wd)
        if self.period == 1:
            automatic_gefen_period1_update_cuda(p, g.reshape(-1), self.codes, self.mag, self.v, codebook, self.divisor, 0.9, 0.999, lr, bc1, bc2, 1e-8)
        else:
            automatic_gefen_fused_update_from_vmean_cuda(p, g.reshape(-1, self.period), self.codes, self.mag, self.v, codebook, False, 0.9, lr, bc1,
                                                         bc2, 1e-8)


def _compare(device, dtype, params, grads_of_step, fused, lr, wd, steps):
    from gefen_b200 import Gefen

    others = [p.clone() for p in params]
    params = [torch.nn.Parameter(p) for p in params]
    opt = Gefen(params, lr=lr, weight_decay=wd, fused=fused)
    separate = None
    for step in range(steps):
        for p, g in zip(params, grads_of_step(step)):
            p.grad = g
        opt.step()
        if separate is None:
            states = [opt.state[p] for p in params]
            separate = [Separate(p, s["automatic_period"], s.get("period_one_divisor"), s["m_magnitude"].dtype) for p, s in zip(others, states)]
        for one, p, mine in zip(separate, others, params):
            one.step(p, mine.grad, opt._gefen_codebook, lr, wd)
    opt.check()
    for one, p, mine in zip(separate, others, params):
        state = opt.state[mine]
        assert torch.equal(state["m_codebook"], one.codes)
        assert torch.equal(state["m_magnitude"], one.mag)
        assert rel_l2(mine.detach().float().cpu(), p.float().cpu()) <= 1e-4
    return {one.period for one in separate}


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("which", ["1.5b", "32b"])
def test_llama_layers(cuda_device, which, fused):
    shapes = [("embed", (8192, 2048))] + workloads.llama_1_5b()[1:10] if which == "1.5b" else workloads.llama_32b()[1:10]
    params = [workloads.init_param(n, s, i, torch.bfloat16, cuda_device) for i, (n, s) in enumerate(shapes)]
    _compare(cuda_device, torch.bfloat16, params,
             lambda step: [workloads.make_grad(s, i, step, torch.bfloat16, cuda_device) for i, (_, s) in enumerate(shapes)], fused, 3e-4, 0.1, 2)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("wd", [0.0, 0.1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_small_shapes(cuda_device, dtype, wd, fused):
    shapes = [(40, 512), (16, 9000), (50, 300), (1,), (77,), (24, 2056)]
    gen = torch.Generator().manual_seed(5)
    params = [(torch.randn(s, generator=gen) * 0.02).to(cuda_device, dtype) for s in shapes]
    # (gradients whose squares fp16 still holds in the second moment)
    grads = [[(torch.randn(s, generator=gen) * 0.3).to(cuda_device, dtype) for s in shapes] for _ in range(3)]
    _compare(cuda_device, dtype, params, lambda step: grads[step], fused, 3e-4, wd, 3)


@pytest.mark.parametrize("wd", [0.0, 0.1])
def test_float64_one_call_per_tensor(cuda_device, monkeypatch, wd):
    """float64 has a state only where it is forced to fp32; the call per tensor keeps the separate launches for it."""
    from gefen_b200 import gefen

    monkeypatch.setattr(gefen, "F_FP32", True)
    shapes = [(40, 512), (50, 300), (77,), (4, 9000)]
    gen = torch.Generator().manual_seed(6)
    params = [(torch.randn(s, generator=gen) * 0.02).to(cuda_device, torch.float64) for s in shapes]
    grads = [[(torch.randn(s, generator=gen) * 1e-3).to(cuda_device, torch.float64) for s in shapes] for _ in range(3)]
    _compare(cuda_device, torch.float64, params, lambda step: grads[step], False, 3e-4, wd, 3)


def test_second_moment_per_element_takes_any_beta2(cuda_device):
    """Only the second moment of blocks wants beta2 in [0, 1]."""
    from gefen_b200 import Gefen

    g = (torch.randn(77, generator=torch.Generator().manual_seed(7)) * 1e-3).to(cuda_device)
    params = [torch.nn.Parameter(torch.zeros(77, device=cuda_device)) for _ in range(2)]
    for p, fused in zip(params, (True, False)):
        opt = Gefen([p], lr=1e-3, fused=fused)
        opt.param_groups[0]["beta2"] = -0.5
        opt.state[p]["automatic_period"] = 1
        p.grad = g.clone()
        opt.step()
        assert bool(p.detach().any())
    assert torch.equal(params[0], params[1])
