"""Newton-Schulz orthogonalisation used by GefenMuon (reference: gefen_muon.py:16-51).

X <- X / max(||X||_F, eps); then `steps` times: A = X X^T, B = b*A + c*A*A, X <- a*X + B*X, all in
bf16 with fp32 accumulation, on the wide orientation (rows <= cols; taller inputs are transposed).
Each product rounds its result to bf16 once, as the reference's torch.addmm / `@` calls do.

The products run on the library's tcgen05 GEMMs, all matrices of a group in one launch per product
(`gefen_b200_ns_group`: K-major and MN-major operands, so no transposed copy is made between
products). The kernels take dimensions that are multiples of 8 (16-byte rows); any other matrix is
padded with zero rows and columns, which the iteration maps to zero rows and columns (they add
nothing to X X^T), and the result is cut back. There is no library GEMM behind this module.
"""
from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from . import _lib

_STATUS = {}


# Elements of all matrices that go through the iteration together: enough tiles for several waves of the GPU's SMs
# (two layers of a 1.7 B model), and a bound on the iterates' memory (4 bytes per element, the Gram matrices on top).
GROUP_ELEMENTS = 1 << 27
# Matrices that one group may hold (GEFEN_B200_NS_GROUP_MATRICES of the library).
GROUP_MATRICES = 4096


def _status(device) -> torch.Tensor:
    t = _STATUS.get(device.index)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=device)
        _STATUS[device.index] = t
    return t


def check_status(device) -> None:
    """Raises if a bounded wait inside a GEMM kernel ran out since the last check (synchronises)."""
    t = _STATUS.get(device.index)
    if t is not None and int(t.item()) != 0:
        t.zero_()
        raise _lib.GefenB200Error("a tcgen05 GEMM gave up waiting on one of its barriers; results are incomplete")


def gemm_tn(a: torch.Tensor, b: torch.Tensor, c: Optional[torch.Tensor] = None, alpha: float = 1.0, beta: float = 0.0,
            out: Optional[torch.Tensor] = None, out_t: Optional[torch.Tensor] = None, symmetric: bool = False) -> torch.Tensor:
    """out[M,N] = alpha * a[M,K] @ b[N,K]^T + beta * c[M,N]; out_t[N,M] = out^T if given. bf16, row-major.
    symmetric=True promises a symmetric result (a is b, c symmetric): half of the tiles are computed."""
    M, K = a.shape
    N = b.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=torch.bfloat16, device=a.device)
    for t in (a, b, c, out, out_t):
        if t is not None and (t.dtype != torch.bfloat16 or t.stride(-1) != 1):
            raise ValueError("gemm_tn expects bf16 matrices with unit inner stride")
    with _lib.device_guard(a.device):
        _lib.check(_lib.load().gefen_b200_ns_gemm_tn(
            _lib.ptr(a), _lib.ptr(b), _lib.ptr(c), _lib.ptr(out), _lib.ptr(out_t), M, N, K, a.stride(0), b.stride(0),
            0 if c is None else c.stride(0), out.stride(0), 0 if out_t is None else out_t.stride(0), float(alpha),
            float(beta), int(symmetric), _lib.ptr(_status(a.device)), _lib.current_stream(a.device)))
    return out


def gemm_nn(a: torch.Tensor, b: torch.Tensor, c: Optional[torch.Tensor] = None, alpha: float = 1.0, beta: float = 0.0,
            out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """out[M,N] = alpha * a[M,K] @ b[K,N] + beta * c[M,N]. bf16, row-major."""
    M, K = a.shape
    N = b.shape[1]
    if out is None:
        out = torch.empty((M, N), dtype=torch.bfloat16, device=a.device)
    for t in (a, b, c, out):
        if t is not None and (t.dtype != torch.bfloat16 or t.stride(-1) != 1):
            raise ValueError("gemm_nn expects bf16 matrices with unit inner stride")
    with _lib.device_guard(a.device):
        _lib.check(_lib.load().gefen_b200_ns_gemm_nn(
            _lib.ptr(a), _lib.ptr(b), _lib.ptr(c), _lib.ptr(out), M, N, K, a.stride(0), b.stride(0),
            0 if c is None else c.stride(0), out.stride(0), float(alpha), float(beta), _lib.ptr(_status(a.device)),
            _lib.current_stream(a.device)))
    return out


def gemm_tt(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, symmetric: bool = False) -> torch.Tensor:
    """out[M,N] = a[K,M]^T @ b[K,N]. bf16, row-major."""
    K, M = a.shape
    N = b.shape[1]
    if out is None:
        out = torch.empty((M, N), dtype=torch.bfloat16, device=a.device)
    with _lib.device_guard(a.device):
        _lib.check(_lib.load().gefen_b200_ns_gemm_tt(
            _lib.ptr(a), _lib.ptr(b), None, _lib.ptr(out), M, N, K, a.stride(0), b.stride(0), 0, out.stride(0), 1.0, 0.0,
            int(symmetric), _lib.ptr(_status(a.device)), _lib.current_stream(a.device)))
    return out


def _wide(shape) -> Tuple[int, int]:
    """Rows and columns of a matrix as the iteration holds it: wide, each a multiple of 8."""
    a, b = (shape[0] + 7) // 8 * 8, (shape[1] + 7) // 8 * 8
    return min(a, b), max(a, b)


def group_scratch_elements(shapes: Sequence[Tuple[int, int]]) -> int:
    """bf16 elements of the buffers of a group: both iterates, Gram matrix and polynomial of every matrix."""
    return sum(2 * m * k + 2 * m * m for m, k in map(_wide, shapes))


class MatrixGroup:
    """The launch tables of a group of matrices of given shapes over one scratch buffer (at least
    `group_scratch_elements` bf16 elements). It can be kept and run again as long as the shapes repeat; its work is
    ordered by the stream it runs on. One that is made under stream capture belongs to that graph: its tables are written
    when the graph runs."""

    def __init__(self, shapes: Sequence[Tuple[int, int]], scratch: torch.Tensor):
        lib = _lib.load()
        self.scratch = scratch
        self.device = scratch.device
        self.mats = np.zeros(len(shapes), dtype=_lib.NS_MATRIX_DTYPE)
        self._places = []
        base, offset = scratch.data_ptr(), 0
        for row, (rows, cols) in zip(self.mats, shapes):
            m, k = _wide((rows, cols))
            self._places.append(offset)
            row["rows"], row["cols"] = rows, cols
            for field, n in (("x0", m * k), ("x1", m * k), ("gram", m * m), ("poly", m * m)):
                row[field] = base + 2 * offset
                offset += n
        if offset > scratch.numel():
            raise ValueError("Expected {} elements of scratch for the group, got {}".format(offset, scratch.numel()))
        # one device buffer: plan, matrix table, partial norms; the first two come from one host buffer
        n = len(shapes)
        plan_bytes = lib.gefen_b200_ns_group_plan_bytes(self.mats.ctypes.data, n)
        place = (plan_bytes + 63) // 64 * 64
        self._host = np.zeros(place + self.mats.nbytes, dtype=np.uint8)
        _lib.check(lib.gefen_b200_ns_group_plan(self.mats.ctypes.data, n, self._host.ctypes.data))
        self._host[place:] = self.mats.view(np.uint8)
        self.mats = self._host[place:].view(_lib.NS_MATRIX_DTYPE)
        self._address = self._host.ctypes.data
        self._place, self._uploaded = place, 0      # bytes of the host buffer that the device has for good
        parts = (place + self.mats.nbytes + 15) // 16 * 16
        self.tables = torch.empty(parts + 256 * n, dtype=torch.uint8, device=self.device)
        self._partials = parts
        self.steps = 0

    def run(self, sources: Sequence[torch.Tensor], ns_coefficients, ns_steps: int, eps: float) -> None:
        """Normalises the (contiguous, 16-byte aligned, equally typed) sources and iterates. `update_of` set the
        scalars of `apply` beforehand, if that follows."""
        a, b, c = ns_coefficients
        self.mats["src"] = [t.data_ptr() for t in sources]
        self.steps = int(ns_steps)
        lib, tables, mats, sent = _lib.load(), self.tables.data_ptr(), self._address + self._place, self._uploaded
        with _lib.device_guard(self.device):
            stream = _lib.current_stream(self.device)
            _lib.check(lib.gefen_b200_upload(tables + sent, self._address + sent, self._host.nbytes - sent, stream))
            if not sent and not torch.cuda.is_current_stream_capturing():
                self._uploaded = self._place
            _lib.check(lib.gefen_b200_ns_group(
                mats, len(self.mats), tables + self._place, tables, tables + self._partials, _lib.dtype_tag(sources[0].dtype),
                self.steps, float(a), float(b), float(c), float(eps), _lib.ptr(_status(self.device)), stream))

    def update_of(self, params: Sequence[torch.Tensor], wd_muls, alphas) -> None:
        self.mats["p"] = [p.data_ptr() for p in params]
        self.mats["wd_mul"], self.mats["alpha"] = wd_muls, alphas
        self.mats["decay"] = [int(w != 1.0) for w in wd_muls]

    def apply(self, dtype: torch.dtype, peers=None) -> None:
        """Weight decay and update of the parameters given to `update_of` (before `run`)."""
        n_peers = 0 if peers is None else len(peers)
        with _lib.device_guard(self.device):
            _lib.check(_lib.load().gefen_b200_ns_group_apply(
                self._address + self._place, len(self.mats), self.tables.data_ptr() + self._place, _lib.dtype_tag(dtype), self.steps,
                peers.ctypes.data if n_peers else None, n_peers, _lib.current_stream(self.device)))

    def result(self, i: int) -> torch.Tensor:
        """The orthogonalised matrix i: a view of the scratch."""
        rows, cols = int(self.mats[i]["rows"]), int(self.mats[i]["cols"])
        m, k = _wide((rows, cols))
        start = self._places[i] + (m * k if self.steps % 2 else 0)
        x = self.scratch[start:start + m * k].view(m, k)
        return x[:rows, :cols] if rows <= cols else x[:cols, :rows].t()


def check_arguments(ns_coefficients, ns_steps: int) -> None:
    if ns_steps >= 100:
        raise ValueError("Number of steps must be less than 100 for computational efficiency")
    if len(ns_coefficients) != 3:
        raise ValueError("Coefficients must be a tuple of exactly 3 values")


def _checked_source(grad: torch.Tensor, ns_coefficients, ns_steps: int) -> torch.Tensor:
    check_arguments(ns_coefficients, ns_steps)
    if len(grad.shape) != 2:
        raise ValueError("Input tensor gradient must be a 2D matrix")
    if grad.device.type != "cuda":
        raise ValueError("gefen_b200 runs Newton-Schulz on the GPU only, got device {}".format(grad.device))
    if grad.dtype not in (torch.float32, torch.float16, torch.bfloat16):
        grad = grad.bfloat16()
    grad = grad.contiguous()
    return grad if grad.data_ptr() % 16 == 0 else grad.clone()


def zeropower_via_newtonschulz(grad: torch.Tensor, ns_coefficients: Tuple[float, float, float], ns_steps: int,
                               eps: float) -> torch.Tensor:
    """reference: gefen_muon.py:16-51. Returns a new tensor."""
    out = []
    orthogonalize_all([(grad, ns_coefficients, ns_steps, eps)],
                      lambda i, ortho: out.append(ortho.clone(memory_format=torch.contiguous_format)))
    return out[0]


def group_runs(keys: Sequence, numels: Sequence[int]) -> List[Tuple[int, int]]:
    """Cuts a sequence of matrices into runs of equal keys, at most GROUP_MATRICES matrices and GROUP_ELEMENTS elements
    (one matrix at least)."""
    runs, begin, total = [], 0, 0
    for i, (key, n) in enumerate(zip(keys, numels)):
        if i > begin and (key != keys[begin] or total + n > GROUP_ELEMENTS or i - begin == GROUP_MATRICES):
            runs.append((begin, i))
            begin, total = i, 0
        total += n
    if len(numels) > begin:
        runs.append((begin, len(numels)))
    return runs


def orthogonalize_all(items, consume) -> None:
    """Newton-Schulz for many matrices, grouped (see MatrixGroup).

    items: list of (matrix, ns_coefficients, ns_steps, eps); consume(i, ortho) is called in order with the
    orthogonalised matrix i (a view of scratch memory: use it at once, on the current stream)."""
    sources = [_checked_source(matrix, coefficients, steps) for matrix, coefficients, steps, _ in items]
    keys = [(s.dtype, s.device, tuple(item[1]), int(item[2]), float(item[3]), s.numel() == 0) for s, item in zip(sources, items)]
    for begin, end in group_runs(keys, [s.numel() for s in sources]):
        run = sources[begin:end]
        if run[0].numel() == 0:
            for i in range(begin, end):
                consume(i, sources[i].bfloat16())
            continue
        shapes = [tuple(s.shape) for s in run]
        scratch = torch.empty(group_scratch_elements(shapes), dtype=torch.bfloat16, device=run[0].device)
        group = MatrixGroup(shapes, scratch)
        _, coefficients, steps, eps = items[begin]
        group.run(run, coefficients, steps, eps)
        for i in range(begin, end):
            consume(i, group.result(i - begin))
