"""Newton-Schulz for groups of matrices: every matrix comes out as it does alone, whatever else is in its group, and
the fused update equals torch's two operations on that result."""
import pytest
import torch

SHAPES = [(300, 500), (1000, 300), (127, 64), (64, 127), (513, 1026), (8, 8), (1, 40), (40, 1), (256, 256), (2048, 192), (129, 2056)]
NS = (3.4445, -4.7750, 2.0315)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("steps", [0, 1, 4, 5])
def test_group_equals_single_runs_and_the_torch_update(cuda_device, dtype, steps):
    from gefen_b200 import newton_schulz as ns

    gen = torch.Generator(device=cuda_device).manual_seed(steps)
    grads = [(torch.randn(s, generator=gen, device=cuda_device) * 0.1).to(dtype) for s in SHAPES]
    params = [(torch.randn(s, generator=gen, device=cuda_device) * 0.02).to(dtype) for s in SHAPES]
    scratch = torch.full((ns.group_scratch_elements(SHAPES),), float("nan"), dtype=torch.bfloat16, device=cuda_device)
    group = ns.MatrixGroup(SHAPES, scratch)
    wd = [1.0 if i % 3 == 0 else 0.998 for i in range(len(SHAPES))]
    alpha = [-0.02 * (1 + i) for i in range(len(SHAPES))]
    mine = [p.clone() for p in params]
    for _ in range(2):   # the second run over the same buffers starts again from the sources
        group.update_of(mine, wd, alpha)
        group.run(grads, NS, steps, 1e-7)
    group.apply(dtype)
    ns.check_status(cuda_device)
    for i, (g, p, got) in enumerate(zip(grads, params, mine)):
        ortho = group.result(i).clone()
        assert ortho.shape == g.shape
        assert torch.equal(ortho, ns.zeropower_via_newtonschulz(g, NS, steps, 1e-7)), SHAPES[i]
        x = g.bfloat16()
        x = x / x.norm().clamp(min=1e-7)
        x = x.T if g.shape[0] > g.shape[1] else x
        for _ in range(steps):
            gram = x @ x.T
            x = torch.addmm(x, torch.addmm(gram, gram, gram, beta=NS[1], alpha=NS[2]), x, beta=NS[0])
        want = (x.T if g.shape[0] > g.shape[1] else x).float()
        assert float((ortho.float() - want).norm() / want.norm()) <= 2e-2, SHAPES[i]
        if wd[i] != 1.0:
            p.mul_(wd[i])
        p.add_(ortho, alpha=alpha[i])
        assert torch.equal(got, p), SHAPES[i]


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [0, 1])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_values_that_are_not_finite(cuda_device, steps, bad):
    """As torch's x / x.norm().clamp(min=eps): a NaN makes the whole matrix NaN, an infinity leaves zeros and a NaN."""
    from gefen_b200 import newton_schulz as ns

    for shape in [(16, 64), (64, 16), (20, 33)]:
        g = torch.ones(shape, device=cuda_device)
        g[3, 5] = bad
        x = g.bfloat16()
        want = x / x.norm().clamp(min=1e-7)
        if steps:
            assert bool(want.isnan().any())
            want = torch.full_like(want, float("nan"))   # the Gram matrix of a row with a NaN, twice
        got = ns.zeropower_via_newtonschulz(g, NS, steps, 1e-7)
        assert torch.equal(torch.nan_to_num(got.float(), nan=7.0), torch.nan_to_num(want.float(), nan=7.0)), shape


@pytest.mark.gpu
def test_float64_sources(cuda_device):
    """Wide, tall, padded and square sources in float64 give what their float32 values give."""
    from gefen_b200 import newton_schulz as ns

    gen = torch.Generator(device=cuda_device).manual_seed(2)
    grads = [torch.randn(s, generator=gen, device=cuda_device) * 0.1 for s in SHAPES]
    results = []
    for dtype in (torch.float32, torch.float64):
        scratch = torch.full((ns.group_scratch_elements(SHAPES),), float("nan"), dtype=torch.bfloat16, device=cuda_device)
        group = ns.MatrixGroup(SHAPES, scratch)
        group.run([g.to(dtype) for g in grads], NS, 5, 1e-7)
        results.append([group.result(i).clone() for i in range(len(SHAPES))])
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_step_of_float64_parameters(cuda_device, monkeypatch):
    """GefenMuon on float64 parameters (fp32 state): the update is torch's, on the orthogonalised momentum."""
    import gefen_b200.gefen as gefen
    from gefen_b200 import GefenMuon, newton_schulz as ns

    monkeypatch.setattr(gefen, "F_FP32", True)
    gen = torch.Generator(device=cuda_device).manual_seed(4)
    shapes = [(64, 128), (256, 64), (48, 36)]
    params = [torch.nn.Parameter((torch.randn(s, generator=gen, device=cuda_device) * 0.02).double()) for s in shapes]
    opt = GefenMuon(params, lr=0.02, weight_decay=0.1, nesterov=False)
    for _ in range(2):
        for p in params:
            p.grad = (torch.randn(p.shape, generator=gen, device=cuda_device) * 1e-3).double()
        before = [p.detach().clone() for p in params]
        opt.step()
        for p, old in zip(params, before):
            st = opt.state[p]
            period = st["automatic_period"]
            block = opt._period_one_divisor_from_state(st, p.numel()) if period == 1 else period
            codes = st["m_codebook"].reshape(-1, block).long()
            momentum = (opt._gefen_codebook[codes] * st["m_magnitude"].float()).reshape(p.shape)
            ortho = ns.zeropower_via_newtonschulz(momentum, NS, 5, 1e-7)
            want = old.mul_(1 - 0.02 * 0.1).add_(ortho, alpha=-0.02 * max(1, p.shape[0] / p.shape[1]) ** 0.5)
            assert torch.equal(p.detach(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 200), (200, 64), (768, 768), (1032, 264), (256, 2304)])
@pytest.mark.parametrize("steps", [1, 4, 5])
def test_single_matrix_entry_of_the_c_interface(cuda_device, shape, steps):
    """gefen_b200_newton_schulz on a normalised matrix in the caller's buffers, wide and tall."""
    from gefen_b200 import _lib, newton_schulz as ns

    gen = torch.Generator(device=cuda_device).manual_seed(steps)
    x = torch.randn(shape, generator=gen, device=cuda_device).bfloat16()
    x = x / x.norm()
    m = min(shape)
    x0, x1 = x.clone(), torch.full_like(x, float("nan"))
    gram, poly = (torch.full((m, m), float("nan"), dtype=torch.bfloat16, device=cuda_device) for _ in range(2))
    _lib.check(_lib.load().gefen_b200_newton_schulz(
        _lib.ptr(x0), _lib.ptr(x1), _lib.ptr(gram), _lib.ptr(poly), shape[0], shape[1], steps, *NS,
        _lib.ptr(ns._status(cuda_device)), _lib.current_stream(cuda_device)))
    got = (x1 if steps % 2 else x0).float()
    ns.check_status(cuda_device)
    want = x.T if shape[0] > shape[1] else x
    for _ in range(steps):
        g = want @ want.T
        want = torch.addmm(want, torch.addmm(g, g, g, beta=NS[1], alpha=NS[2]), want, beta=NS[0])
    want = (want.T if shape[0] > shape[1] else want).float()
    assert float((got - want).norm() / want.norm()) <= 2e-2


def test_runs_of_a_group():
    from gefen_b200 import newton_schulz as ns

    cap = ns.GROUP_ELEMENTS
    assert ns.group_runs([], []) == []
    assert ns.group_runs("aab", [1, 2, 3]) == [(0, 2), (2, 3)]
    assert ns.group_runs("aaaa", [cap, 1, cap - 1, 1]) == [(0, 1), (1, 3), (3, 4)]
    assert ns.group_runs("aa", [2 * cap, 2 * cap]) == [(0, 1), (1, 2)]
    most = ns.GROUP_MATRICES
    assert ns.group_runs("a" * (2 * most + 1), [8] * (2 * most + 1)) == [(0, most), (most, 2 * most), (2 * most, 2 * most + 1)]


def test_largest_group_is_what_the_library_takes():
    import numpy as np

    from gefen_b200 import _lib, newton_schulz as ns

    mats = np.zeros(ns.GROUP_MATRICES + 1, dtype=_lib.NS_MATRIX_DTYPE)
    mats["rows"], mats["cols"] = 8, 16
    for field in ("x0", "x1", "gram", "poly"):
        mats[field] = 4096   # (sizes only: nothing is read)
    plan_bytes = _lib.load().gefen_b200_ns_group_plan_bytes
    assert plan_bytes(mats.ctypes.data, ns.GROUP_MATRICES) > 0
    assert plan_bytes(mats.ctypes.data, ns.GROUP_MATRICES + 1) == 0
    for rows, cols in ((1 << 25, 4), (4, 3 << 24), (1 << 30, 8)):   # long and thin ones
        mats["rows"], mats["cols"] = rows, cols
        assert plan_bytes(mats.ctypes.data, 1) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [
    [(2048, 2304), (2048, 2048), (2056, 2120)],                                   # 256 x 256 tiles on pairs, ragged edges
    [(768, 3072)] * 5 + [(3072, 768)] * 5 + [(768, 768), (776, 1000), (200, 900), (8, 16)] * 2,
])
def test_groups_that_fill_the_gpu(cuda_device, shapes):
    """Enough tiles for pairs of CTAs: every matrix against torch's chain and, bit for bit, against the same matrix alone
    (smaller tiles, single CTAs): a sharded run groups the matrices otherwise than one process and has to give the same."""
    from gefen_b200 import newton_schulz as ns

    gen = torch.Generator(device=cuda_device).manual_seed(7)
    grads = [(torch.randn(s, generator=gen, device=cuda_device) * 1e-3).bfloat16() for s in shapes]
    group = ns.MatrixGroup(shapes, torch.full((ns.group_scratch_elements(shapes),), float("nan"), dtype=torch.bfloat16, device=cuda_device))
    group.run(grads, NS, 5, 1e-7)
    ns.check_status(cuda_device)
    for i, g in enumerate(grads):
        got = group.result(i).float()
        x = g / g.norm().clamp(min=1e-7)
        x = x.T if g.shape[0] > g.shape[1] else x
        for _ in range(5):
            gram = x @ x.T
            x = torch.addmm(x, torch.addmm(gram, gram, gram, beta=NS[1], alpha=NS[2]), x, beta=NS[0])
        want = (x.T if g.shape[0] > g.shape[1] else x).float()
        assert float((got - want).norm() / want.norm()) <= 2e-2, shapes[i]
        assert torch.equal(group.result(i), ns.zeropower_via_newtonschulz(g, NS, 5, 1e-7)), shapes[i]


@pytest.mark.gpu
def test_mixed_settings_and_strides_in_one_step(cuda_device):
    """Parameter groups with iterations of their own, and parameters that are not contiguous (torch updates their run):
    every matrix moves by the orthogonalisation of its own momentum."""
    from gefen_b200 import GefenMuon, newton_schulz as ns

    gen = torch.Generator(device=cuda_device).manual_seed(6)
    shapes = [(64, 128), (96, 64), (48, 36), (128, 128), (40, 200), (72, 24)]
    settings = [dict(ns_steps=5, eps=1e-7), dict(ns_steps=3, eps=1e-7), dict(ns_steps=5, eps=1e-3)]
    params = []
    for i, s in enumerate(shapes):
        t = torch.randn((s[1], s[0]) if i in (1, 4) else s, generator=gen, device=cuda_device) * 0.02
        params.append(torch.nn.Parameter(t.t() if i in (1, 4) else t))
    assert not params[1].is_contiguous() and not params[4].is_contiguous()
    opt = GefenMuon(params, lr=0.02, weight_decay=0.1, nesterov=False)
    by_param = {}
    for group in opt.param_groups:   # (one per parameter)
        for p in group["params"]:
            i = next(k for k, q in enumerate(params) if q is p)
            group.update(settings[(i // 2) % 3])
            by_param[i] = group
    for step in range(2):
        for p in params:
            p.grad = torch.randn(p.shape, generator=gen, device=cuda_device) * 1e-3
        before = [p.detach().clone() for p in params]
        opt.step()
        for i, (p, old) in enumerate(zip(params, before)):
            st = opt.state[p]
            period = st["automatic_period"]
            block = opt._period_one_divisor_from_state(st, p.numel()) if period == 1 else period
            momentum = opt._gefen_codebook[st["m_codebook"].reshape(-1, block).long()] * st["m_magnitude"]
            group = by_param[i]
            ortho = ns.zeropower_via_newtonschulz(momentum.reshape(p.shape), NS, group["ns_steps"], group["eps"])
            want = old.mul_(1 - 0.02 * 0.1).add_(ortho, alpha=-0.02 * max(1, p.shape[0] / p.shape[1]) ** 0.5)
            assert torch.equal(p.detach(), want), (step, i)
