"""The pruned exact-DP fit against the oracle, on histograms from flat to concentrated in a few bins."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["bell", "flat", "spikes", "steep", "two ends"])
@pytest.mark.parametrize("k,active", [(256, 4096), (256, 300), (16, 1000), (2, 50), (255, 256)])
def test_pruned_dp_is_bit_exact(oracle, cuda_device, shape, k, active):
    from gefen_b200 import quantization

    gen = torch.Generator().manual_seed(k + active)
    centers = torch.sort(torch.rand(active, generator=gen) * 2 - 1).values
    counts = {"bell": torch.exp(-0.5 * (centers / 0.28) ** 2) * 1e6, "flat": torch.full((active,), 1000.0),
              "spikes": torch.where(torch.rand(active, generator=gen) < 0.02, 1e8, 1.0),
              "steep": torch.exp(-centers.abs() * 40) * 1e9, "two ends": torch.where(centers.abs() > 0.95, 1e6, 1.0)}[shape]
    counts = torch.floor(counts) + 1
    for force in (True, False):
        want = oracle.exact_dp(centers, counts, k, force)
        got = quantization.exact_dp({"active_centers": centers, "active_counts": counts}, k, force, device=cuda_device)
        assert torch.equal(got, want)
