"""The fused Lloyd-Max update against the plain formula."""
import pytest
import torch

from tests.util import reference_like_codebook

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 37, 256])
@pytest.mark.parametrize("force", [True, False])
def test_lloyd_update(cuda_device, k, force):
    from gefen_b200 import _lib

    gen = torch.Generator().manual_seed(k)
    cb = reference_like_codebook(k=max(k, 2))[:k].to(cuda_device).contiguous()
    sums = (torch.randn(k, generator=gen) * 1e3).to(cuda_device)
    counts = torch.randint(0, 4, (k,), generator=gen).to(cuda_device) * 1000
    want = torch.where(counts > 0, sums / counts.clamp(min=1).float(), cb)
    if force:
        want[0] = -1.0
        want[-1] = 1.0
    want = want.sort().values
    ws = torch.empty(_lib.CODEBOOK_WS_BYTES, dtype=torch.uint8, device=cuda_device)
    _lib.check(_lib.load().gefen_b200_lloyd_update(_lib.ptr(cb), k, int(force), _lib.ptr(sums), _lib.ptr(counts), _lib.ptr(ws),
                                                   _lib.current_stream(cuda_device)))
    assert torch.equal(cb, want)
    assert not bool(sums.any()) and not bool(counts.any())
    assert torch.equal(ws[:32784], _lib.codebook_workspace(want.contiguous())[:32784])
