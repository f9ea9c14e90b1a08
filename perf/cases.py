"""What is timed when this library's speed is compared between two versions, and on which inputs.

The cases are optimizer work as a training program has it done through the public classes and functions:
the steady-state step of `Gefen` (one call after every backward pass, by far the most frequent), the step of
`GefenMuon`, the calibrating first step of a run, and the optional Lloyd-Max codebook fit. The models are the
parameter sets of the benchmark configurations plus small and ragged ones; fp32, bf16 and fp16 occur.

A model is given by name (a function of `gefen_b200.workloads`, optionally a run of its tensors) or as a text
of shapes, "300x500;1200". Its tensors are views of one flat buffer per kind (parameters, gradients, codes,
magnitudes, second moments), 256-byte aligned as separate allocations are, so that the outputs of a step are
these few buffers and nothing is copied to return them.
"""
import math

import torch

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
BETA1, BETA2, EPS = 0.9, 0.999, 1e-8          # Gefen's defaults
MOMENTUM, MUON_EPS, MUON_STEPS = 0.95, 1e-7, 5  # GefenMuon's defaults
NS = (3.4445, -4.7750, 2.0315)
STEPS_BEFORE = 100    # a run that is under way: bias corrections away from their first values
ENTRIES = 256


def listed():
    return [
        # A small fully connected network in fp32 (classifiers, probes, policies): six tensors, half a million
        # elements; the call's own latency.
        {"name": "step_mlp_f32", "kind": "step", "dtype": "f32", "wd": 0.0, "shapes": "512x784;512;256x512;256;10x256;10"},
        # GPT-2 125M in fp32: 148 tensors, most of them small, blocks of 768 to 1536 elements.
        {"name": "step_gpt2_f32", "kind": "step", "dtype": "f32", "wd": 0.0, "model": "gpt2_125m"},
        # Llama-style 1.5B in bf16 with weight decay, the headline workload: 1.5 G elements, blocks of 512 and 2048.
        {"name": "step_llama1.5b_bf16", "kind": "step", "dtype": "bf16", "wd": 0.1, "model": "llama_1_5b"},
        # One layer of the Llama-style 32B (what one of many ranks steps at a time): blocks of 1664 and 1120 elements.
        {"name": "step_llama32b_layer_bf16", "kind": "step", "dtype": "bf16", "wd": 0.1, "model": "llama_32b", "first": 1, "count": 9},
        # Rows whose length is no multiple of eight (300-wide word embeddings, a patch embedding of 147 inputs,
        # 1500-wide hidden layers, a 3 x 3 kernel stack): the kernels for any block length, in bf16.
        {"name": "step_ragged_bf16", "kind": "step", "dtype": "bf16", "wd": 0.01,
         "shapes": "30000x300;1200x300;1200x300;1200;1500x1500;1500;64x147;64;1000x1500;1000;96x27;4500x1500"},
        # The launch structure of one call per tensor (fused=False) on a transformer layer in fp16.
        {"name": "step_unfused_f16", "kind": "unfused", "dtype": "f16", "wd": 0.1, "model": "llama_1_5b", "first": 1, "count": 9},
        # GefenMuon on four layers of Qwen3-1.7B-shaped matrices, bf16: Newton-Schulz on the tensor cores.
        {"name": "muon_qwen_4layers_bf16", "kind": "muon", "dtype": "bf16", "model": "qwen3_1_7b_matrices", "first": 0, "count": 28},
        # GefenMuon on the matrices of a 768-wide transformer in fp32 (24 matrices of six layers): many small products.
        {"name": "muon_768_f32", "kind": "muon", "dtype": "f32", "shapes": ";".join(["768x2304;768x768;768x3072;3072x768"] * 6)},
        # GefenMuon on a few small matrices of ragged sizes, bf16: padding and latency.
        {"name": "muon_ragged_bf16", "kind": "muon", "dtype": "bf16", "shapes": "300x500;1000x300;127x64;513x1026"},
        # The first step of a run: period search, histogram, codebook fit and one step, GPT-2 125M in fp32.
        {"name": "first_step_gpt2_f32", "kind": "first", "dtype": "f32", "wd": 0.0, "model": "gpt2_125m"},
        # The same for the large tensors of the Llama-style 1.5B in bf16 (the embedding and two layers).
        {"name": "first_step_llama_bf16", "kind": "first", "dtype": "bf16", "wd": 0.1, "model": "llama_1_5b", "first": 0, "count": 19},
        # Lloyd-Max refinement of a codebook, ten iterations over 2^25 fp32 values in blocks of 2048.
        {"name": "lloyd_fit_f32", "kind": "lloyd", "dtype": "f32", "shapes": "16384x2048", "iterations": 10},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A layer width: half the time a multiple of 64 or 8 as models have them, otherwise any number."""
    w = _spread(rng, lo, hi)
    kind = rng.random()
    if kind < 0.35 and w >= 64:
        return w // 64 * 64
    if kind < 0.6 and w >= 8:
        return w // 8 * 8
    return w


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "unfused", "muon", "muon", "first", "lloyd"])
    dtype = rng.choice(["bf16", "bf16", "f32", "f16"])
    most = {"step": 6e8, "unfused": 1e8, "muon": 4e7, "first": 2e8, "lloyd": 3e7}[kind]   # elements
    if kind == "lloyd":
        cols = _width(rng, 64, 8000)
        rows = max(4, int(_spread(rng, 1e5, most) // cols))
        return {"kind": kind, "dtype": dtype, "shapes": "%dx%d" % (rows, cols), "iterations": rng.randint(1, 10)}
    shapes, total = [], 0
    width = _width(rng, 64, 2500 if kind == "muon" else 9000)
    for _ in range(_spread(rng, 1, 24)):
        # (matrices of a first step have rows enough for the period search to be sure of them)
        rows = _width(rng, 128 if kind == "first" else 24, 9000 if kind == "muon" else 40000)
        for shape in ((rows, width), (width, max(32 if kind == "first" else 8, rows // 4)), (width,)):
            n = math.prod(shape)
            if total + n > most or (kind == "muon" and len(shape) == 1):
                continue
            shapes.append(shape)
            total += n
    if not shapes:
        shapes = [(96, 64)]
    case = {"kind": kind, "dtype": dtype, "shapes": ";".join("x".join(map(str, s)) for s in shapes)}
    if kind != "muon":
        case["wd"] = rng.choice([0.0, 0.01, 0.1])
    return case


# ---------------------------------------------------------------------------------------------- models
def _tensors(case):
    """[(name, shape)] of a case."""
    if "model" in case:
        from gefen_b200 import workloads

        out = getattr(workloads, case["model"])()
        return out[case.get("first", 0):][:case.get("count", len(out))]
    out = []
    for i, text in enumerate(case["shapes"].split(";")):
        out.append(("t%d" % i, tuple(int(d) for d in text.split("x"))))
    return out


def _period(shape):
    """The block length that the calibration finds for gradients with a scale of their own per row: the row, or
    its smallest divisor above 1024; vectors have no blocks."""
    if len(shape) < 2 or shape[1] <= 8 or shape[0] < 4:
        return 1
    cols = shape[1]
    if cols <= 1024:
        return cols
    return min(q for q in range(1025, cols + 1) if cols % q == 0)


def _magnitudes(numel, period):
    """(number of magnitudes, elements per magnitude): blocks, or for vectors their largest divisor up to 256."""
    if period == 1:
        period = max(d for d in range(1, 257) if numel % d == 0)
    return numel // period, period


def _layout(sizes, element_size):
    """Offsets of tensors of these sizes in one buffer, each 256-byte aligned, and the buffer's length."""
    step = 256 // element_size
    offsets, end = [], 0
    for n in sizes:
        offsets.append(end)
        end += (n + step - 1) // step * step
    return offsets, end


def _per_block(values, numel):
    """A state column of the first step as an output. The block length of a small tensor depends on chance: there the
    values are given per element, so that the output's size does not."""
    values = values.reshape(-1)
    return values if numel >= 65536 else values.repeat_interleave(numel // values.numel())


class _Buffer:
    """One zeroed flat buffer and its tensors as views of the given shapes."""

    def __init__(self, shapes, dtype, device):
        sizes = [math.prod(s) for s in shapes]
        offsets, end = _layout(sizes, torch.empty(0, dtype=dtype).element_size())
        self.flat = torch.zeros(end, dtype=dtype, device=device)
        self.views = [self.flat[o:o + n].view(s) for o, n, s in zip(offsets, sizes, shapes)]


def _codebook(device):
    """A codebook like the ones that the fit finds for bell-shaped values: quantiles of a normal law, ends at +-1."""
    at = (torch.arange(ENTRIES, dtype=torch.float64) + 0.5) / ENTRIES
    cb = (torch.special.ndtri(at) * 0.36).float()
    cb[0], cb[-1] = -1.0, 1.0
    return cb.to(device)


def _generator(device, seed, index, what):
    g = torch.Generator(device=device)
    g.manual_seed((seed * 4099 + index) * 16 + what)
    return g


def _tensor_inputs(case, shape, index, seed, device):
    """The values of one tensor, made from the seed: parameter, gradient (normal with a log-normal scale per row,
    the same in the momentum and the second moment) and the optimizer state of a run under way."""
    dtype = DTYPES[case["dtype"]]
    tau = 0.5 if case["kind"] == "muon" else 1.0
    rows = shape[0] if len(shape) == 2 else 1
    scale = torch.exp(torch.randn(rows, 1, generator=_generator(device, seed, index, 0), device=device) * tau)
    scale *= 0.1 if dtype == torch.float16 else 1e-3     # fp16 gradients come with a scaled loss
    n = math.prod(shape)

    def normal(what, spread):
        x = torch.randn((rows, n // rows), generator=_generator(device, seed, index, what), device=device)
        return x.mul_(spread)

    p = normal(1, 0.02).to(dtype).view(shape)
    g = normal(2, scale).to(dtype).view(shape)
    if case["kind"] in ("first", "lloyd"):
        return {"p": p, "g": g}
    period = _period(shape)
    count, block = _magnitudes(n, period)
    m = normal(3, scale * 0.3).view(count, block)
    mag = m.abs().amax(1, keepdim=True)
    cb = _codebook(device)
    mids = (cb[1:] + cb[:-1]) * 0.5
    codes = torch.empty((count, block), dtype=torch.uint8, device=device)
    for i in range(0, count, 1 << 17):     # in runs of blocks: bucketize's indices are eight bytes each
        codes[i:i + (1 << 17)] = torch.bucketize(m[i:i + (1 << 17)] / mag[i:i + (1 << 17)], mids).to(torch.uint8)
    out = {"p": p, "g": g, "codes": codes.view(n // period, period), "mag": mag.to(dtype), "period": period, "block": block}
    if case["kind"] != "muon":
        v = (scale * scale * 1e-1).expand(rows, n // rows).reshape(-1, period)[:, :1]
        out["v"] = (v * torch.rand(v.shape, generator=_generator(device, seed, index, 4), device=device).add_(0.5)).to(dtype)
    return out


# ---------------------------------------------------------------------------------------------- the calls
def prepare(case, seed):
    device = torch.device("cuda", 0)
    dtype = DTYPES[case["dtype"]]
    named = _tensors(case)
    shapes = [s for _, s in named]
    state = {"case": case}
    params, grads = _Buffer(shapes, dtype, device), _Buffer(shapes, dtype, device)
    state["params"] = params.flat
    if case["kind"] == "lloyd":
        values = _tensor_inputs(case, shapes[0], 0, seed, device)["g"]
        return {"case": case, "values": values.reshape(-1), "period": shapes[0][1], "codebook": _codebook(device)}
    leaves = [(name, torch.nn.Parameter(v)) for (name, _), v in zip(named, params.views)]
    for (_, leaf), g in zip(leaves, grads.views):
        leaf.grad = g
    state["leaves"] = leaves
    if case["kind"] == "first":
        for i, shape in enumerate(shapes):
            x = _tensor_inputs(case, shape, i, seed, device)
            params.views[i].copy_(x["p"])
            grads.views[i].copy_(x["g"])
        return state

    from gefen_b200 import Gefen, GefenMuon

    if case["kind"] == "muon":
        opt = GefenMuon(leaves, lr=0.02, weight_decay=0.1, momentum=MOMENTUM)
    else:
        opt = Gefen(leaves, lr=3e-4, betas=(BETA1, BETA2), eps=EPS, weight_decay=case["wd"], fused=case["kind"] == "step")
    periods = [_period(s) for s in shapes]
    counts = [_magnitudes(math.prod(s), q)[0] for s, q in zip(shapes, periods)]
    codes = _Buffer([(math.prod(s) // q, q) for s, q in zip(shapes, periods)], torch.uint8, device)
    mags = _Buffer([(c, 1) for c in counts], dtype, device)
    state.update(opt=opt, codes=codes.flat, mag=mags.flat)
    if case["kind"] != "muon":
        moments = _Buffer([(math.prod(s) // q, 1) for s, q in zip(shapes, periods)], dtype, device)
        state["v"] = moments.flat
    resumed = opt.state_dict()
    resumed["gefen_global_step"], resumed["gefen_codebook"] = STEPS_BEFORE, _codebook(device)
    for i, shape in enumerate(shapes):
        x = _tensor_inputs(case, shape, i, seed, device)
        params.views[i].copy_(x["p"])
        grads.views[i].copy_(x["g"])
        codes.views[i].copy_(x["codes"])
        mags.views[i].copy_(x["mag"])
        own = {"automatic_period": x["period"], "step": STEPS_BEFORE, "m_codebook_shape": tuple(codes.views[i].shape),
               "m_codebook": codes.views[i], "m_magnitude": mags.views[i]}
        if x["period"] == 1:
            own["period_one_divisor"] = x["block"]
        if case["kind"] != "muon":
            moments.views[i].copy_(x["v"])
            own["vmean"] = moments.views[i]
        resumed["state"][i] = own
        del x
    opt.load_state_dict(resumed)     # as a program resumes from a checkpoint
    for i, (_, leaf) in enumerate(leaves):   # the state stays in the flat buffers, whatever loading copies
        opt.state[leaf].update({k: v for k, v in resumed["state"][i].items() if torch.is_tensor(v)})
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "lloyd":
        from gefen_b200.kernels.lloyd_max_fused import lloyd_max_fit

        return lloyd_max_fit([(state["values"], state["period"])], state["codebook"], iterations=state["case"]["iterations"])
    if kind == "first":
        from gefen_b200 import Gefen

        opt = Gefen(state["leaves"], lr=3e-4, betas=(BETA1, BETA2), eps=EPS, weight_decay=state["case"]["wd"])
        opt.step()
        own = [opt.state[leaf] for _, leaf in state["leaves"]]
        # the new state is one allocation per tensor: put together here because there are hundreds of them
        numels = [leaf.numel() for _, leaf in state["leaves"]]
        return {"params": state["params"], "codebook": opt._gefen_codebook,
                "periods": torch.tensor([s["automatic_period"] for s in own]),
                "codes": torch.cat([s["m_codebook"].reshape(-1) for s in own]),
                "mag": torch.cat([_per_block(s["m_magnitude"], n) for s, n in zip(own, numels)]),
                "v": torch.cat([_per_block(s["vmean"], n) for s, n in zip(own, numels)])}
    state["opt"].step()
    return {k: state[k] for k in ("params", "codes", "mag", "v") if k in state}


# ---------------------------------------------------------------------------------------------- what it takes
def work(case):
    s = 4 if case["dtype"] == "f32" else 2
    total = flops = 0
    for _, shape in _tensors(case):
        n = math.prod(shape)
        period = _period(shape)
        if case["kind"] == "lloyd":
            total += n * s
            continue
        count = _magnitudes(n, period)[0]
        # gradient in, parameter in and out, code in and out (the first step: out), the scalars of the blocks
        total += n * (3 * s + (1 if case["kind"] == "first" else 2)) + 2 * s * count
        if case["kind"] == "muon":
            m, k = min(shape), max(shape)
            # per iteration X X^T and the polynomial (symmetric: half of each) and the product with X
            flops += MUON_STEPS * (m * m * k + m * m * m + 2 * m * m * k)
        else:
            total += 2 * s * (n // period)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Between two correct implementations of the same precision. The codes, magnitudes and new codebooks follow from
    fixed fp32 operations; the order of the sum of squares moves a second moment by one rounding of the state's type
    now and then, and with it a block's update."""
    if case["kind"] == "muon":
        # five bf16 iterations whose products may add up in any order; the parameters hold the update
        # (measured against 64 bits: 2.6e-4 of fp32 parameters, 2.6e-3 of bf16 ones, 1.6e-3 of it their rounding)
        return {"rel": 1e-3 if case["dtype"] == "f32" else (1.5e-3 if case["dtype"] == "f16" else 1e-2), "max": 0.2, "differ": 1e-5}
    if case["kind"] == "lloyd":
        return {"rel": 1e-5, "max": 1e-4}   # (the same inputs twice: 7e-7, the sums are added up in any order)
    if case["dtype"] == "f32":
        return {"rel": 2e-6, "max": 1e-4, "differ": 1e-5}
    return {"rel": 1e-3 if case["dtype"] == "bf16" else 2e-4, "max": 0.02, "differ": 1e-5}


# ---------------------------------------------------------------------------------------------- in 64 bits
def _nearest(x, cb):
    return torch.bucketize(x, (cb[1:] + cb[:-1]) * 0.5)


def _step_exact(x, wd, lr):
    """The Gefen step of one tensor: (parameter, codes, magnitude, second moment)."""
    n, t = x["p"].numel(), STEPS_BEFORE + 1
    cb = _codebook(x["p"].device).double()
    g = x["g"].double().view(-1, x["block"])
    mag = x["mag"].double()
    m = BETA1 * mag * cb[x["codes"].view(-1, x["block"]).int()] + (1 - BETA1) * g
    new = m.abs().amax(1, keepdim=True)
    codes = _nearest(m / new, cb)
    del m
    q = cb[codes] * new
    if x["period"] == 1:
        v = BETA2 * x["v"].double().view(-1) + (1 - BETA2) * g.view(-1).square()
        step = (1 / (1 - BETA1 ** t)) / ((v / (1 - BETA2 ** t)).sqrt() + EPS)
        change = q.view(-1) * step
    else:
        v = BETA2 * x["v"].double() + (1 - BETA2) * g.square().mean(1, keepdim=True)
        # the step size is formed from the second moment as the state holds it
        step = (1 / (1 - BETA1 ** t)) / ((v / (1 - BETA2 ** t)).sqrt() + EPS)
        change = (q * step).view(-1)
    p = x["p"].double().view(-1) * (1 - lr * wd) - lr * change
    return p, codes.to(torch.uint8).view(-1), new.view(-1), v.view(-1)


def _muon_exact(x, shape, lr, wd):
    n = x["p"].numel()
    cb = _codebook(x["p"].device).double()
    g = x["g"].double().view(-1, x["block"])
    m = MOMENTUM * x["mag"].double() * cb[x["codes"].view(-1, x["block"]).int()] + (1 - MOMENTUM) * g
    new = m.abs().amax(1, keepdim=True)
    codes = _nearest(m / new, cb)
    y = (cb[codes] * new * MOMENTUM + (1 - MOMENTUM) * g).view(shape)
    y = y.T if shape[0] > shape[1] else y
    y = y / y.norm().clamp(min=MUON_EPS)
    a, b, c = NS
    for _ in range(MUON_STEPS):
        gram = y @ y.T
        y = a * y + (b * gram + c * gram @ gram) @ y
    y = y.T if shape[0] > shape[1] else y
    p = x["p"].double() * (1 - lr * wd) - lr * math.sqrt(max(1, shape[0] / shape[1])) * y
    return p.reshape(-1), codes.to(torch.uint8).view(-1), new.view(-1)


def _period_exact(g):
    """The period search: the highest local maximum over the divisors above 8 of the mean step between the mean
    logarithms of neighbouring blocks, brought down to the smallest divisor above 1024."""
    n = g.numel()
    if n == 1:
        return 1
    small = [d for d in range(1, math.isqrt(n) + 1) if n % d == 0]
    divisors = sorted(set([d for d in small if d != n] + [n // d for d in small]))
    cands = [d for d in divisors if n // d >= 4]
    at = next((i for i, d in enumerate(cands) if d > 8), None)
    if at is None:
        return 1
    cands = cands[max(at - 1, 0):]
    logs = (g.double().reshape(-1).square() + 1e-12).log()
    scores = []
    for d in cands:
        means = logs.view(-1, d).mean(1)
        scores.append((means[1:] - means[:-1]).abs().mean())
    scores = torch.stack(scores).tolist() if scores else []
    best = max(((scores[i], d) for i, d in enumerate(cands) if 0 < i < len(cands) - 1 and d > 8
                and scores[i] > scores[i - 1] and scores[i] > scores[i + 1]), default=(0, 1))[1]
    if best > 1024:
        best = min(q for q in divisors if 1024 < q <= best and best % q == 0)
    return best


def _lloyd_exact(values, period, cb, iterations):
    v = values.double().view(-1, period)
    x = (v / v.abs().amax(1, keepdim=True)).view(-1)
    cb = cb.double()
    for _ in range(iterations):
        at = _nearest(x, cb)
        counts = torch.bincount(at, minlength=ENTRIES)
        sums = torch.bincount(at, weights=x, minlength=ENTRIES)
        cb = torch.where(counts > 0, sums / counts.clamp(min=1), cb)
        cb[0], cb[-1] = -1.0, 1.0
        cb = cb.sort().values
    return cb


def exact(case, seed):
    device = torch.device("cuda", 0)
    shapes = [s for _, s in _tensors(case)]
    if case["kind"] == "lloyd":
        values = _tensor_inputs(case, shapes[0], 0, seed, device)["g"].reshape(-1)
        return _lloyd_exact(values, shapes[0][1], _codebook(device), case["iterations"])
    if case["kind"] == "first":
        # the codebook fit (and what follows from it) takes too long without compiled code
        mags, moments = [], []
        for i, shape in enumerate(shapes):
            g = _tensor_inputs(case, shape, i, seed, device)["g"]
            period = _period_exact(g)
            flat = g.double().reshape(-1)
            mags.append(_per_block((flat.view(-1, _magnitudes(flat.numel(), period)[1]) * (1 - BETA1)).abs().amax(1), flat.numel()))
            moments.append(_per_block(flat.view(-1, period).square().mean(1) * (1 - BETA2), flat.numel()))
        return {"params": None, "codebook": None, "periods": None, "codes": None, "mag": torch.cat(mags), "v": torch.cat(moments)}
    out = {}

    def place(key, sizes, element_size, dtype):
        offsets, end = _layout(sizes, element_size)
        out[key] = torch.zeros(end, dtype=dtype, device=device)
        return offsets

    s = torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size()
    numels = [math.prod(shape) for shape in shapes]
    periods = [_period(shape) for shape in shapes]
    at = {"params": place("params", numels, s, torch.float64), "codes": place("codes", numels, 1, torch.uint8),
          "mag": place("mag", [_magnitudes(n, q)[0] for n, q in zip(numels, periods)], s, torch.float64)}
    if case["kind"] != "muon":
        at["v"] = place("v", [n // q for n, q in zip(numels, periods)], s, torch.float64)
    for i, shape in enumerate(shapes):
        x = _tensor_inputs(case, shape, i, seed, device)
        if case["kind"] == "muon":
            got = _muon_exact(x, shape, 0.02, 0.1)
        else:
            got = _step_exact(x, case["wd"], 3e-4)
        for key, value in zip(("params", "codes", "mag", "v"), got):
            out[key][at[key][i]:at[key][i] + value.numel()] = value
        del x, got
    return out
