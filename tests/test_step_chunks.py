"""The staged step kernel on blocks and pointers that are multiples of 4, 2 or 1 elements only, and its quantiser on
codebooks that put one, several or very many thresholds into one table cell. Same inputs, oracle and bit-exactness
as the tests of the usual blocks."""
import pytest
import torch

from tests.util import make_grad, make_param, reference_like_codebook

# (blocks, period): a chunk and one more, less than a lane's share, a ragged last unit, the longest staged blocks
BLOCKS = [(5, 4), (67, 12), (9, 300), (5, 1500), (3, 2044), (2, 8188),     # chunks of four
          (7, 2), (33, 18), (11, 514), (3, 2042), (2, 8190),               # of two
          (9, 1), (35, 3), (50, 27), (21, 147), (5, 513), (3, 2047), (2, 8191)]


def _codebooks():
    return {
        "fit": reference_like_codebook(),
        "two per cell": torch.linspace(-1, 1, 256).sign() * torch.linspace(-1, 1, 256).abs().pow(1.6),
        "five per cell": torch.cat([torch.tensor([-1.0]), torch.linspace(-0.05, 0.05, 254), torch.tensor([1.0])]),
        "all in one cell": torch.cat([torch.tensor([-1.0]), 0.3 + torch.arange(254) * 1e-6, torch.tensor([1.0])]),
        "ends below one": torch.linspace(-0.9, 0.7, 200),
    }


def _run(oracle, device, nb, period, dtype, codebook, offset=0):
    from gefen_b200.kernels.automatic_gefen_fused import automatic_gefen_fused_update_from_vmean_cuda

    g = make_grad((nb, period), period, 0, 0, dtype)
    p = make_param((nb, period), period, 0, dtype)
    gen = torch.Generator().manual_seed(nb)
    codes = torch.randint(0, codebook.numel(), (nb, period), dtype=torch.uint8, generator=gen)
    mag = (torch.rand(nb, 1, generator=gen) * 2e-3).to(dtype)
    v = (torch.rand(nb, 1, generator=gen) * 1e-6 + 1e-7).to(dtype)
    cb = codebook.float().contiguous()

    def on_device(t):   # `offset` elements into a larger allocation: every pointer is that much out of line
        flat = torch.zeros(t.numel() + offset, dtype=t.dtype, device=device)
        view = flat[offset:].view(t.shape)
        view.copy_(t)
        return view

    dp, dg, dc = (on_device(t) for t in (p, g, codes))
    dm, dv = mag.to(device), v.to(device)
    args = dict(beta1=0.9, lr=3e-4, bias_correction_1=0.3, bias_correction_2=0.003, eps=1e-8)
    for _ in range(2):
        oracle.automatic_gefen_fused_update_from_vmean(p, g, codes, mag, v, cb, False, **args)
        automatic_gefen_fused_update_from_vmean_cuda(dp, dg, dc, dm, dv, cb.to(device), False, **args)
    assert torch.equal(dc.cpu(), codes)
    assert torch.equal(dm.cpu(), mag)
    assert torch.equal(dp.cpu(), p)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nb,period", BLOCKS)
def test_small_chunks(oracle, cuda_device, dtype, nb, period):
    _run(oracle, cuda_device, nb, period, dtype, reference_like_codebook())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [1, 2, 4])
@pytest.mark.parametrize("nb,period", [(9, 512), (3, 2048), (40, 24)])
def test_pointers_out_of_line(oracle, cuda_device, dtype, offset, nb, period):
    _run(oracle, cuda_device, nb, period, dtype, reference_like_codebook(), offset)


@pytest.mark.gpu
@pytest.mark.parametrize("period", [2048, 256, 64, 32, 300, 147])
@pytest.mark.parametrize("name", sorted(_codebooks()))
def test_codebooks_of_every_density(oracle, cuda_device, period, name):
    _run(oracle, cuda_device, 21, period, torch.float32, _codebooks()[name])


def test_launch_class_follows_length_and_alignment():
    """The chunk of a launch class divides the block and the alignment of every pointer, and is the largest such."""
    import numpy as np

    from gefen_b200 import _lib

    lib = _lib.load()
    chunk = {1: 8, 2: 8, 3: 4, 4: 2, 5: 1}
    for size, dtype in ((4, _lib.F32), (2, _lib.BF16), (2, _lib.F16)):
        for period in list(range(1, 70)) + [147, 300, 513, 1024, 1032, 1500, 2048, 8192, 8193, 10000]:
            for shift in (0, 1, 2, 3, 4, 8, 16):
                row = np.zeros(1, dtype=_lib.STEP_TENSOR_DTYPE)
                row["g"], row["p"], row["codes"] = 4096 + shift * size, 8192, 16384 + shift
                row["period"], row["num_blocks"] = period, 3
                cls = lib.gefen_b200_step_launch_class(row.ctypes.data, dtype)
                if period > 8192:
                    assert cls == -1
                    continue
                fits = [v for v in (8, 4, 2, 1) if period % v == 0 and shift * size % min(16, v * size) == 0 and shift % v == 0]
                assert chunk[cls] == fits[0], (period, shift, size, cls)
                assert cls != 1 or period > 1024


def test_classes_of_a_whole_table():
    import numpy as np

    from gefen_b200 import _lib

    lib = _lib.load()
    rows = np.zeros(60, dtype=_lib.STEP_TENSOR_DTYPE)
    rows["num_blocks"], rows["period"] = 3, [1 + 7 * i * i for i in range(60)]
    rows["g"], rows["p"], rows["codes"] = 4096 + 4 * np.arange(60), 8192, 16384
    rows["flags"] = np.where(np.arange(60) % 5 == 0, _lib.STEP_PERIOD1, 0)
    for tag in (_lib.F32, _lib.BF16, _lib.F64):
        tensor, launch = _lib.step_classes(rows, tag)
        assert tensor == [lib.gefen_b200_step_tensor_class(rows[i:i + 1].ctypes.data, tag) for i in range(60)]
        assert launch == [lib.gefen_b200_step_launch_class(rows[i:i + 1].ctypes.data, tag) for i in range(60)]
    assert _lib.step_classes(rows[:0], _lib.F32) == [[], []]
