"""The scan of many tensors' candidate periods against plain fp64, on inputs that reach every branch: bases of all
lengths and alignments, values outside the range of the product form."""
import math

import pytest
import torch


def _scores(flat, periods, squared, eps):
    x = flat.double().cpu()
    logs = ((x if squared else x * x) + eps).log()
    out = []
    for p in periods:
        means = logs.view(-1, p).mean(1)
        out.append(float((means[1:] - means[:-1]).abs().mean()))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.float64])
@pytest.mark.parametrize("squared", [False, True])
def test_many_scan_against_fp64(cuda_device, dtype, squared):
    from gefen_b200 import partitioning
    from gefen_b200.kernels.period_variance import period_scan_many_async

    gen = torch.Generator(device=cuda_device).manual_seed(3)
    lengths = [36, 1024, 768 * 96, 9 * 11 * 13 * 4, 300 * 77, 4 * 1733, 4 * 20011, 64 * 8192 * 4, 17 * 64]
    flats = []
    for i, n in enumerate(lengths):
        x = torch.randn(n, generator=gen, device=cuda_device) * 1e-3 * torch.exp(torch.randn(n, generator=gen, device=cuda_device))
        if i % 3 == 1 and dtype not in (torch.float16,):
            x[n // 3] = 1e30       # takes its own logarithm
        if i % 3 == 2:
            x[: n // 2] = 0.0
        x = x.abs() if squared else x
        buffer = torch.zeros(n + 1, device=cuda_device, dtype=dtype)
        view = buffer[i % 2:i % 2 + n]      # every second tensor starts out of line
        view.copy_(x)
        flats.append(view)
    cands = [[p for p in partitioning.native_divisors(n) if n // p >= 4] for n in lengths]
    got = torch.cat([s.cpu() for s in period_scan_many_async(flats, cands, input_is_squared=squared, epsilon=1e-12)])
    cursor = 0
    for flat, cand in zip(flats, cands):
        # scores are means of differences between means of about -25: n roundings of 2^-53 relative to those
        for want, row in zip(_scores(flat, cand, squared, 1e-12), got[cursor:cursor + len(cand)]):
            assert abs(float(row[0]) - want) <= 1e-12 * (1 + abs(want)), (flat.numel(), want, float(row[0]))
            assert float(row[1]) == 0.0
        cursor += len(cand)


@pytest.mark.gpu
def test_scan_counts_invalid_inputs_and_follows_nan(cuda_device):
    from gefen_b200.kernels.period_variance import period_scan_async

    x = torch.full((4096,), 1e-3, device=cuda_device)
    x[5], x[4000] = -1.0, -2.0
    stats = period_scan_async(x, [8, 16, 64], input_is_squared=True, epsilon=1e-12).cpu()
    assert stats[:, 1].tolist() == [2.0, 2.0, 2.0]
    y = torch.full((4096,), 1e-3, device=cuda_device)
    y[7] = float("nan")
    assert all(math.isnan(v) for v in period_scan_async(y, [8, 64], input_is_squared=False, epsilon=1e-12).cpu()[:, 0].tolist())
    tiny = period_scan_async(x.abs(), [8, 64], input_is_squared=False, epsilon=1e-300).cpu()   # below the product form's range
    assert bool(torch.isfinite(tiny).all())


@pytest.mark.gpu
@pytest.mark.parametrize("squared", [False, True])
@pytest.mark.parametrize("eps", [2.0 ** -121, 2.0 ** -119, 2.0 ** -71, 2.0 ** -69, 1.0, 2.0 ** 99, 2.0 ** 101, 2.0 ** 130, 1e300])
def test_epsilon_on_both_sides_of_the_product_form(cuda_device, squared, eps):
    from gefen_b200.kernels.period_variance import period_scan_async

    gen = torch.Generator(device=cuda_device).manual_seed(1)
    x = torch.exp2(torch.rand(64 * 96, generator=gen, device=cuda_device) * 122.5 - 60)
    got = period_scan_async(x, [8, 64, 512], input_is_squared=squared, epsilon=eps).cpu()
    for want, row in zip(_scores(x, [8, 64, 512], squared, eps), got):
        # means of logarithms of up to 700: 2^-53 of those per term
        assert abs(float(row[0]) - want) <= 1e-12 * (1 + abs(want)), (want, float(row[0]))


@pytest.mark.gpu
def test_blocks_whose_logarithms_leave_32_bits(cuda_device):
    """Two blocks of 2^29 + 2^20 elements, zeros and ones: the binary exponent of the first block's product is -40 times
    its length, about five times what 32 bits hold."""
    from gefen_b200.kernels.period_variance import period_scan_async

    period = (1 << 29) + (1 << 20)
    x = torch.zeros(2 * period, dtype=torch.bfloat16, device=cuda_device)
    x[period:] = 1.0
    want = math.log(1.0 + 1e-12) - math.log(1e-12)
    got = float(period_scan_async(x, [period], input_is_squared=False, epsilon=1e-12).cpu()[0, 0])
    # one rounding of 2^-53 per factor (relative), and the logarithm itself
    assert abs(got - want) <= 1e-12 * want


def test_native_divisors():
    from gefen_b200 import partitioning

    for n in list(range(2, 400)) + [768 * 2304, 128256 * 2048, 50257 * 768, 1000003, 999983 * 4, 2 ** 30, 17920 * 6656]:
        assert partitioning.native_divisors(n) == partitioning.divisors(n)
