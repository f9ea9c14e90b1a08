"""The ring kernel with three and more units for every warp of a full grid, for every chunk length: the buffers are filled
again, the barrier's phase turns, units lie side by side. The number of units is asserted. Bit for bit against the oracle."""
import pytest
import torch

from tests.test_step_chunks import _run
from tests.util import reference_like_codebook

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,nb,period,blocks_per_unit", [
    (torch.bfloat16, 9001, 1032, 1), (torch.float32, 7201, 1032, 1), (torch.float32, 30001, 520, 2), (torch.float16, 300001, 24, 16),   # chunks of 8
    (torch.bfloat16, 40001, 300, 4), (torch.float32, 30001, 300, 4),       # of 4
    (torch.bfloat16, 300001, 18, 32), (torch.bfloat16, 10001, 514, 1),     # of 2
    (torch.bfloat16, 160001, 27, 16), (torch.float32, 40001, 147, 2),      # of 1
])
def test_three_units_per_warp(oracle, cuda_device, dtype, nb, period, blocks_per_unit):
    warps = (16 if dtype == torch.float32 else 20) * torch.cuda.get_device_properties(cuda_device).multi_processor_count
    assert nb // blocks_per_unit >= 3 * warps
    _run(oracle, cuda_device, nb, period, dtype, reference_like_codebook())
