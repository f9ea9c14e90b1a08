"""The histograms of many tensors in one launch against the single-tensor kernel."""
import pytest
import torch

from tests.util import make_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.float64])
@pytest.mark.parametrize("bins", [4096, 1000, 1])
def test_histograms_of_many_tensors(cuda_device, dtype, bins):
    from gefen_b200.kernels.exact_histogram_fused import gefen_exact_histogram_cuda, gefen_exact_histogram_many_cuda

    flats, periods = [], []
    for i, (nb, period) in enumerate([(5000, 64), (1, 8), (70, 2048), (33, 147), (9, 8192), (3, 9001), (40000, 1), (7, 300), (1, 262144)]):
        g = make_grad((nb, period), 5, i, 0, torch.float32).reshape(-1)
        g[: min(period, 50)] = 0.0
        buffer = torch.zeros(g.numel() + 1, dtype=dtype, device=cuda_device)
        view = buffer[i % 2:i % 2 + g.numel()]
        view.copy_(g)
        if i == 3:
            view[5] = float("nan")
        flats.append(view)
        periods.append(period)
    want = torch.zeros(bins, dtype=torch.float32)
    for flat, period in zip(flats, periods):
        row = torch.zeros(bins, dtype=torch.int64, device=cuda_device)
        gefen_exact_histogram_cuda(flat, period, row)
        want.add_(row.cpu().to(torch.float32))
    assert torch.equal(gefen_exact_histogram_many_cuda(flats, periods, bins).cpu(), want)
