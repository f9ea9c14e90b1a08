"""The ring kernel where the work on one chunk takes lanes apart before the warp reads the next chunk's momenta from tensor
memory: codebooks whose quantiser searches (its early exit depends on the value), blocks whose last rounds ask for
parameters in some lanes only. Every warp of a full grid comes to several units. Bit for bit against the oracle."""
import pytest
import torch

from tests.test_step_chunks import _codebooks, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["ends below one", "all in one cell", "five per cell"])
@pytest.mark.parametrize("dtype,nb,period", [(torch.bfloat16, 9001, 1112), (torch.float32, 7201, 1040), (torch.float16, 20001, 520),
                                             (torch.bfloat16, 40001, 300), (torch.bfloat16, 300001, 18), (torch.float32, 120001, 27)])
def test_lanes_that_branch_between_rounds(oracle, cuda_device, dtype, nb, period, name):
    _run(oracle, cuda_device, nb, period, dtype, _codebooks()[name])


@pytest.mark.parametrize("dtype,nb,period", [(torch.bfloat16, 9001, 1336), (torch.bfloat16, 9001, 2040), (torch.float32, 7201, 1848)])
def test_last_rounds_that_ask_in_some_lanes(oracle, cuda_device, dtype, nb, period):
    _run(oracle, cuda_device, nb, period, dtype, _codebooks()["fit"])
