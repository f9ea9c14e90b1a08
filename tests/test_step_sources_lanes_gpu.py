"""Averaged gradients in short blocks, where the lanes of a block depend on the number of buffers: the same bits
as the plain step, second moments included, over several units per warp and a ragged last one."""
import pytest
import torch

from tests.test_step_sources_gpu import _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nb,period", [(300001, 8), (200003, 16), (150001, 24), (150001, 32), (90001, 40), (90007, 48), (90001, 56), (90003, 64), (70001, 72)])
def test_short_blocks(cuda_device, dtype, nb, period):
    plain = _step(cuda_device, dtype, nb, period, 0, 0)
    # (the average of three or five equal values of 8 or 11 bits is the value itself after rounding to its type)
    for sources in (1, 2, 3, 4, 5, 8):
        got = _step(cuda_device, dtype, nb, period, sources, 0)
        assert torch.equal(got[0][0], plain[0][0]), sources
        for a, b in zip(got[1:], plain[1:]):
            assert torch.equal(a, b), sources
