"""Period-1 tensors on their own kernel: run lengths from one element to 256 in every type, many vectors in one launch,
and a step whose launches overlap followed at once by work that reads all of its results."""
import pytest
import torch

from tests.util import make_grad, make_param, reference_like_codebook

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("numel,divisor", [(1, 1), (2, 2), (31, 31), (32, 32), (33, 33), (255, 255), (256, 256), (2048, 256), (1000, 250), (7 * 254, 254)])
def test_vectors(oracle, cuda_device, dtype, numel, divisor):
    from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_period1_update_cuda

    cb = reference_like_codebook()
    g = make_grad((numel,), numel, 0, 0, dtype) * 100
    p = make_param((numel,), numel, 0, dtype)
    gen = torch.Generator().manual_seed(numel)
    codes = torch.randint(0, 256, (numel, 1), dtype=torch.uint8, generator=gen)
    mag = (torch.rand(numel // divisor, 1, generator=gen) * 1e-1).to(dtype)
    v = (torch.rand(numel, 1, generator=gen) * 1e-3 + 1e-4).to(dtype)
    if numel > 40:
        g[3], g[35] = float("nan"), float("inf")
    dp, dg, dc, dm, dv = (t.to(cuda_device) for t in (p, g, codes, mag, v))
    args = (divisor, 0.9, 0.999, 1e-3, 0.3, 0.003, 1e-8)
    oracle.automatic_gefen_period1_update(p, g, codes, mag, v, cb, *args)
    automatic_gefen_period1_update_cuda(dp, dg, dc, dm, dv, cb.to(cuda_device), *args)
    assert torch.equal(dc.cpu(), codes)
    for got, want in ((dm, mag), (dv, v), (dp, p)):
        assert torch.equal(torch.nan_to_num(got.cpu().float(), nan=7.0), torch.nan_to_num(want.float(), nan=7.0))


def test_overlapping_launches_are_complete_for_what_follows(cuda_device):
    """Every launch class in one step; copies enqueued right behind it must see all of them. Against a step with one
    synchronised launch per class."""
    from gefen_b200 import Gefen

    shapes = [(4096, 2048), (3000, 512), (2000, 300), (1000, 1030), (500, 147), (2048,), (77,), (3, 8209)]
    gen = torch.Generator(device=cuda_device).manual_seed(0)
    data = [torch.randn(s, generator=gen, device=cuda_device) * 0.02 for s in shapes]
    grads = [torch.randn(s, generator=gen, device=cuda_device) * 1e-3 *
             (torch.exp(torch.randn(s[0], 1, generator=gen, device=cuda_device)) if len(s) == 2 else 1.0) for s in shapes]
    runs = []
    for together in (True, False):
        params = [torch.nn.Parameter(d.bfloat16()) for d in data]
        opt = Gefen(params, lr=1e-3, weight_decay=0.1)
        for p, g in zip(params, grads):
            p.grad = g.bfloat16()
        opt.step()
        for _ in range(5):
            if together:
                opt.step()
                seen = [p.detach().clone() for p in params]
            else:
                for i, p in enumerate(params):
                    opt._step_multi_tensor(only={id(p)})
                    torch.cuda.synchronize()
        runs.append((seen if together else [p.detach().clone() for p in params],
                     [opt.state[p]["m_codebook"].clone() for p in params]))
    for a, b in zip(runs[0][0] + runs[0][1], runs[1][0] + runs[1][1]):
        assert torch.equal(a, b)
