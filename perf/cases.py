"""Performance cases of the framework: the optimizer work a training program has it do, through the public entry points.

A case is a dict of plain values.  Its "kind" says which entry points one pass calls:

  linear       ActivationStatistics.capture() around the forward of a few nn.Linear layers, commit(), MuonT / AdamT.step()
  stack        the same around the forward of a stack of transformer-block projections
  fast         FastTonerCore.begin() + step(): the layer-sharded engine behind FastMuonT / FastAdamT, one rank
  muon         the plain Muon baseline's step()
  capture      capture_recomputed(): the sampled rows of one micro-batch of every layer
  syrk         syrk_upper(): one statistic stack's X^T X with the moving average
  polar        ns_polar(): the Newton-Schulz polar iteration
  roots        inv_roots(): inverse roots of a statistic stack, nothing known of the spectrum

Sizes are those of the benchmark, the tests and the kernel sweep of this repository, and of the ranges around them.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch
from torch import nn

import toner_b200
from toner_b200 import capture, ops
from toner_b200.fast import Muon
from toner_b200.fast.engine import FastTonerCore
from toner_b200.statistics import sample_positions
from toner_b200.synthetic import fill_rows_spectrum, make_stack

HEAD, STRIDE = 32, 16      # position sampling of every optimizer here
NS_STEPS = 10
LLAMA = (("q", 0), ("k", 0), ("v", 0), ("o", 0), ("gate", 1), ("up", 1), ("down", 2))
NANOGPT = (("q", 0), ("k", 0), ("v", 0), ("attn_proj", 0), ("fc", 1), ("mlp_proj", 2))


def listed():
    return [
        # One projection, 8192 rows of 768: the smallest real step, where launches and waits are all there is.
        dict(name="muont_one_768", kind="linear", optimizer="muont", out=768, inp=768, count=1, rows=8192),
        # Three odd-sized projections under AdamT with few, odd rows: remainders in every tile and pass.
        dict(name="adamt_odd_680x1000", kind="linear", optimizer="adamt", out=1000, inp=680, count=3, rows=1111),
        # AdamT + ActivationStatistics on the 12-layer 768 / 3072 stack, 8 x 1024 tokens: the general interface as the
        # benchmark runs it (752 sampled rows for 3072-wide statistics: rank-deficient, the hardest spectrum there is).
        dict(name="adamt_stack_12x768", kind="stack", optimizer="adamt", layers=12, hidden=768, mlp=3072, sequences=8,
             seq_len=1024),
        # FastMuonT on the same stack, 64 x 1024 tokens.
        dict(name="fast_muont_12x768", kind="fast", optimizer="muont", layout="nanogpt", layers=12, hidden=768, mlp=3072,
             rows=6016, spectrum="iid"),
        # FastAdamT on a 32-layer, 512-wide stack (the small published training run), one rank's rows of eight.
        dict(name="fast_adamt_32x512", kind="fast", optimizer="adamt", layout="llama", layers=32, hidden=512, mlp=2048,
             rows=18304, spectrum="iid"),
        # FastMuonT, widths that are no power of two, outlier directions in the statistics, an odd number of rows.
        dict(name="fast_muont_spiked_4x1280", kind="fast", optimizer="muont", layout="llama", layers=4, hidden=1280,
             mlp=3328, rows=10001, spectrum="spiked:8"),
        # FastMuonT at the headline widths and rows: the six layers that one of four ranks owns.  The largest case.
        dict(name="fast_muont_6x2048", kind="fast", optimizer="muont", layout="llama", layers=6, hidden=2048, mlp=5632,
             rows=73216, spectrum="iid"),
        # The plain Muon baseline over eight 768 / 3072 blocks.
        dict(name="muon_8x768", kind="muon", layers=8, hidden=768, mlp=3072),
        # Row capture after one micro-batch's forward: 24 layers, one sequence of 4096 tokens.  Latency and HBM.
        dict(name="capture_24x2048", kind="capture", layers=24, hidden=2048, mlp=5632, batch=1, seq_len=4096),
        # One statistic of a long accumulation (the sweep's 256 K rows).
        dict(name="syrk_262144x2048", kind="syrk", k=1, rows=262144, n=2048),
        # Newton-Schulz on two d x 4d matrices (the sweep's shape), five steps as the plain Muon recipe takes.
        dict(name="polar_2x2048x8192", kind="polar", batch=2, m=2048, n=8192, steps=5),
        # Inverse roots of four 2048-wide statistics at condition 1e4, as a first step or a repair runs them.
        dict(name="roots_4x2048", kind="roots", k=4, n=2048, p=8, q=4, cond=1e4),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _eights(rng, lo, hi):
    return max(8, 8 * round(_log(rng, lo, hi) / 8))


def _draw_once(rng):
    kind = rng.choice(("linear", "linear", "stack", "fast", "fast", "fast", "muon", "capture", "syrk", "polar", "roots"))
    if kind == "linear":
        return dict(kind=kind, optimizer=rng.choice(("muont", "adamt")), out=_eights(rng, 256, 2560),
                    inp=_eights(rng, 256, 2560), count=rng.randint(1, 4), rows=round(_log(rng, 512, 8192)))
    if kind == "stack":
        hidden = 64 * rng.randint(6, 16)
        return dict(kind=kind, optimizer=rng.choice(("muont", "adamt")), layers=rng.randint(2, 12), hidden=hidden,
                    mlp=hidden * rng.choice((3, 4)), sequences=rng.randint(2, 12), seq_len=rng.choice((512, 768, 1024)))
    if kind == "fast":
        hidden = 256 * rng.randint(2, 8)
        mlp = 256 * round(hidden * rng.uniform(2.5, 4.0) / 256)
        return dict(kind=kind, optimizer=rng.choice(("muont", "muont", "adamt")), layout=rng.choice(("llama", "nanogpt")),
                    layers=rng.randint(2, 16), hidden=hidden, mlp=min(mlp, 5632), rows=round(_log(rng, 3000, 73216)),
                    spectrum=rng.choice(("iid", "iid", "spiked:4", "spiked:8")))
    if kind == "muon":
        hidden = 64 * rng.randint(4, 24)
        return dict(kind=kind, layers=rng.randint(2, 8), hidden=hidden, mlp=hidden * 4)
    if kind == "capture":
        return dict(kind=kind, layers=rng.randint(4, 24), hidden=256 * rng.randint(2, 8), mlp=256 * rng.randint(6, 22),
                    batch=rng.randint(1, 4), seq_len=rng.choice((1024, 2048, 4096)))
    if kind == "syrk":
        return dict(kind=kind, k=rng.randint(1, 6), rows=round(_log(rng, 4000, 262144)), n=_eights(rng, 768, 4096))
    if kind == "polar":
        m = _eights(rng, 512, 2560)
        return dict(kind=kind, batch=rng.randint(1, 6), m=m, n=m * rng.choice((1, 3, 4)), steps=rng.choice((2, 3, 5)))
    p, q = rng.choice(((8, 4), (8, 4), (4, 1)))
    return dict(kind=kind, k=rng.randint(1, 8), n=_eights(rng, 512, 3072), p=p, q=q, cond=10.0 ** rng.uniform(2, 5))


def draw(rng):
    top = next(c for c in listed() if c["name"] == "fast_muont_6x2048")
    most = work(top)
    while True:
        case = _draw_once(rng)
        w = work(case)
        if w["flops"] <= most["flops"] and w["bytes"] <= most["bytes"]:
            return case


# ------------------------------------------------------------------ what a program has in hand before the call
def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + salt)


def _stacked(count, out, inp, gen, std):
    return torch.randn(count, out, inp, device="cuda", generator=gen) * std


def _optimizer(case, params):
    if case["optimizer"] == "muont":
        return toner_b200.MuonT(params, lr=0.02, weight_decay=0.1, momentum=0.95)
    return toner_b200.AdamT(params, lr=2e-3, weight_decay=0.1, betas=(0.9, 0.95), eps=1e-15)


def _prepare_linear(case, seed):
    g = _generator(seed)
    out, inp, count = case["out"], case["inp"], case["count"]
    weights = _stacked(count, out, inp, g, 0.02)
    layers = {}
    for i in range(count):
        layer = nn.Linear(inp, out, bias=False, device="meta")
        layer.weight = nn.Parameter(weights[i])
        layer.weight.grad = torch.randn(out, inp, device="cuda", generator=g) * 1e-3
        layers[f"linear.{i}"] = layer
    mean = torch.randn(1, inp, device="cuda", generator=g) * 0.5
    xs = [(torch.randn(case["rows"], inp, device="cuda", generator=g) + mean).to(torch.bfloat16) for _ in range(count)]
    params = [layer.weight for layer in layers.values()]
    stats = toner_b200.ActivationStatistics(layers, head=HEAD, stride=STRIDE, distributed=False)
    modules = list(layers.values())

    def forward():
        for layer, x in zip(modules, xs):
            layer(x)

    return SimpleNamespace(opt=_optimizer(case, params), stats=stats, forward=forward, params=params, flats=[weights])


def _prepare_stack(case, seed):
    g = _generator(seed)
    blocks = make_stack("nanogpt", case["layers"], case["hidden"], case["mlp"], torch.device("cuda"), seed=seed)
    layers = {}
    for i, b in enumerate(blocks):
        for name, mod in (("attn.q", b.attn.q), ("attn.k", b.attn.k), ("attn.v", b.attn.v), ("attn.proj", b.attn.proj),
                          ("mlp.fc", b.mlp.fc), ("mlp.proj", b.mlp.proj)):
            layers[f"blocks.{i}.{name}"] = mod
    params = [m.weight for m in layers.values()]
    # weights of one shape share a storage, as in a flattened parameter buffer
    by_shape = {}
    for p in params:
        by_shape.setdefault(tuple(p.shape), []).append(p)
    flats = [torch.stack([p.detach() for p in ps]) for ps in by_shape.values()]
    for ps, flat in zip(by_shape.values(), flats):
        for p, w in zip(ps, flat):
            p.data = w
    for p in params:
        p.grad = torch.randn(p.shape, device="cuda", generator=g) * 1e-3
    x = torch.randn(case["sequences"], case["seq_len"], case["hidden"], device="cuda", generator=g).to(torch.bfloat16)
    stats = toner_b200.ActivationStatistics(layers, head=HEAD, stride=STRIDE, distributed=False)

    def forward():
        h = x
        for b in blocks:
            h = nn.functional.layer_norm(b(h).float(), (case["hidden"],)).to(torch.bfloat16)

    return SimpleNamespace(opt=_optimizer(case, params), stats=stats, forward=forward, params=params, flats=flats)


def _shapes(case):
    h, m = case["hidden"], case["mlp"]
    return ((h, h), (m, h), (h, m))


def _prepare_fast(case, seed):
    g = _generator(seed)
    roles = LLAMA if case["layout"] == "llama" else NANOGPT
    shapes, layers = _shapes(case), case["layers"]
    named, flats = {}, []
    for role, kind in roles:
        flat = _stacked(layers, *shapes[kind], g, 0.02)
        flats.append(flat)
        for i in range(layers):
            p = nn.Parameter(flat[i])
            p.grad = torch.randn(shapes[kind], device="cuda", generator=g) * 1e-3
            named[f"body.blocks.{i}.{role}.weight"] = p
    blocks = [SimpleNamespace(input_rows_attn=torch.empty(case["rows"], 1, dtype=torch.bfloat16)) for _ in range(layers)]
    muont = case["optimizer"] == "muont"
    args = SimpleNamespace(toner_decay=0.95, toner_split=muont, toner_alpha=0.25, toner_alpha_in=0.5, toner_alpha_out=0.125,
                           wd=0.1, beta1=0.9, beta2=0.95, eps=1e-15, muon_momentum=0.95, muon_nesterov=True,
                           muon_ns_steps=NS_STEPS, muon_eps=1e-5, muon_ns_mode="tpu")
    core = FastTonerCore.from_blocks(blocks, named, case["optimizer"], hid=case["hidden"], mlp=case["mlp"],
                                     rows_total=case["rows"], args=args, world=1, rank=0, device=torch.device("cuda", 0))
    core.param_groups[0]["lr"] = 0.02 if muont else 2e-3
    # every layer's rows come from the model's own population (one mean and spectrum a statistic), other tokens a layer
    for i, block in enumerate(blocks):
        for j, name in enumerate(("attn", "o", "mlp", "down")):
            buf = getattr(block, f"input_rows_{name}")
            fill_rows_spectrum(buf.unsqueeze(0), seed=(seed * 7919 + i * 4 + j) % (1 << 31), spectrum=case["spectrum"],
                               mean_seed=(seed * 31 + j) % (1 << 31))
    return SimpleNamespace(core=core, flats=flats, blocks=blocks, muont=muont)


def _prepare_muon(case, seed):
    g = _generator(seed)
    shapes = _shapes(case)
    params, flats = [], []
    for role, kind in NANOGPT:
        flat = _stacked(case["layers"], *shapes[kind], g, 0.02)
        flats.append(flat)
        for w in flat:
            p = nn.Parameter(w)
            p.grad = torch.randn(shapes[kind], device="cuda", generator=g) * 1e-3
            params.append(p)
    return SimpleNamespace(opt=Muon(params, lr=0.02, weight_decay=0.1, distributed=False), flats=flats, params=params)


def _prepare_capture(case, seed):
    g = _generator(seed)
    layers, b, t, d, dm = case["layers"], case["batch"], case["seq_len"], case["hidden"], case["mlp"]
    mk = lambda w: [torch.randn(b, t, w, device="cuda", generator=g, dtype=torch.bfloat16) for _ in range(layers)]  # noqa: E731
    idx = torch.tensor(sample_positions(t, HEAD, STRIDE), device="cuda")
    rows = b * idx.numel()
    norm = lambda: [1 + 0.1 * torch.randn(d, device="cuda", generator=g) for _ in range(layers)]  # noqa: E731
    flat_d = torch.zeros(3 * layers, rows, d, device="cuda", dtype=torch.bfloat16)
    flat_f = torch.zeros(layers, rows, dm, device="cuda", dtype=torch.bfloat16)
    bufs = [x for i in range(layers) for x in (flat_d[3 * i], flat_d[3 * i + 1], flat_d[3 * i + 2], flat_f[i])]
    return SimpleNamespace(a=(mk(d), mk(d), mk(d), mk(dm), mk(dm), norm(), norm(), bufs),
                           at=torch.arange(rows, device="cuda"), idx=idx, flats=[flat_d, flat_f])


def _prepare_syrk(case, seed):
    x = torch.empty(case["k"], case["rows"], case["n"], device="cuda", dtype=torch.bfloat16)
    fill_rows_spectrum(x, seed=seed, spectrum="iid")
    return SimpleNamespace(x=x, ema=torch.zeros(case["k"], case["n"], case["n"], device="cuda"))


def _prepare_polar(case, seed):
    b, m, n = case["batch"], case["m"], case["n"]
    u = torch.randn(b, m, n, device="cuda", generator=_generator(seed))
    ws = torch.empty(ops.ns_polar_workspace_bytes(b, m, n), device="cuda", dtype=torch.uint8)
    return SimpleNamespace(u=u, out=torch.empty_like(u), ws=ws)


def _prepare_roots(case, seed):
    g = _generator(seed)
    k, n = case["k"], case["n"]
    q, _ = torch.linalg.qr(torch.randn(n, n, device="cuda", generator=g))   # one basis, a spectrum of its own each
    ema = torch.empty(k, n, n, device="cuda")
    for i in range(k):
        lam = torch.exp(torch.rand(n, device="cuda", generator=g) * math.log(case["cond"]))
        c = (q * lam) @ q.T
        ema[i] = 0.5 * (c + c.T)
    ws = torch.empty(ops.inv_roots_workspace_bytes(k, n), device="cuda", dtype=torch.uint8)
    hi = torch.empty_like(ema) if case["q"] > 1 else None
    return SimpleNamespace(ema=ema, ws=ws, lo=torch.empty_like(ema), hi=hi, fro2=torch.empty(k, device="cuda"),
                           status=torch.zeros(k, device="cuda", dtype=torch.int32))


def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    s.case = case
    return s


# ------------------------------------------------------------------ one pass
def _whole(tensors):
    """The stacks that per-parameter tensors are rows of, each once; a tensor that stands alone is itself."""
    out = {}
    for t in tensors:
        base = t._base if t._base is not None and t._base.ndim == t.ndim + 1 else t
        out[base.data_ptr()] = base.detach()
    return list(out.values())


def _state_of(opt, params, keys):
    return {key: _whole([opt.state[p][key] for p in params]) for key in keys}


def _run_general(s):
    with s.stats.capture():
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            s.forward()
    s.stats.commit(s.opt)
    s.opt.step()
    moments = ("momentum_buffer",) if s.case["optimizer"] == "muont" else ("exp_avg", "exp_avg_sq")
    return {"weights": s.flats, **_state_of(s.opt, s.params, ("input_ema",) + moments)}


_run_linear = _run_stack = _run_general


def _run_fast(s):
    s.core.begin()
    s.core.step()
    groups = [info["group"] for info in s.core.roles.values()]
    out = {"weights": s.flats, "ema": [g.factors.ema for g in s.core.groups.values()], "m": [g.m for g in groups]}
    if not s.muont:
        out["v"] = [g.v for g in groups]
    return out


def _run_muon(s):
    s.opt.step()
    return {"weights": s.flats, **_state_of(s.opt, s.params, ("momentum_buffer",))}


def _run_capture(s):
    capture.capture_recomputed(*s.a, s.at, s.idx, 1e-5)
    return s.flats


def _run_syrk(s):
    ops.syrk_upper(s.x, s.ema, ops.EMA_FULL, 0.95, 0.05 / s.case["rows"])
    return s.ema


def _run_polar(s):
    return ops.ns_polar(s.u, s.case["steps"], out=s.out, workspace=s.ws)


def _run_roots(s):
    return ops.inv_roots(s.ema, 1e-3, s.case["p"], s.case["q"], root_lo=s.lo, root_hi=s.hi, fro2_lo=s.fro2, status=s.status,
                         workspace=s.ws)


def run(state):
    return globals()["_run_" + state.case["kind"]](state)


# ------------------------------------------------------------------ what a pass cannot do without
def _polar_flops(m, n, steps=NS_STEPS):
    a, b = min(m, n), max(m, n)
    return steps * (a * a * b + a ** 3 + 2 * a * a * b)      # two symmetric products (half each) and the update


def _root_flops(n, muont):
    # two coupled Newton steps and a finishing polynomial of degree four, products of symmetric matrices (n^3 each)
    return (2 + 3 + 3 + (2 if muont else 0)) * n ** 3


def _update(out, inp, optimizer):
    """(bytes, flops) of one matrix's update: weight, gradient and moments once each way; right products."""
    size = out * inp
    if optimizer == "muont":
        return 4 * size * 5, _polar_flops(out, inp) + 3 * 2 * size * inp
    return 4 * size * 7, 5 * 2 * size * inp


def work(case):
    kind = case["kind"]
    if kind in ("linear", "stack", "fast"):
        muont = case["optimizer"] == "muont"
        if kind == "linear":
            mats = [(case["out"], case["inp"])] * case["count"]
            stats, rows, forward = [case["inp"]] * case["count"], case["rows"], case["rows"]
        else:
            roles = LLAMA if case.get("layout") == "llama" else NANOGPT
            mats = [_shapes(case)[k] for _, k in roles] * case["layers"]
            stats = ([case["hidden"]] * 3 + [case["mlp"]]) * case["layers"]
            rows, forward = case.get("rows"), 0
            if kind == "stack":
                rows = case["sequences"] * len(sample_positions(case["seq_len"], HEAD, STRIDE))
                forward = case["sequences"] * case["seq_len"]
        byts = sum(2 * rows * n + 8 * n * n for n in stats)
        flops = sum(rows * n * (n + 1) + _root_flops(n, muont) for n in stats)
        for out, inp in mats:
            b, f = _update(out, inp, case["optimizer"])
            byts, flops = byts + b, flops + f + 2 * forward * out * inp
        return {"bytes": byts, "flops": flops}
    if kind == "muon":
        mats = [_shapes(case)[k] for _, k in NANOGPT] * case["layers"]
        return {"bytes": sum(4 * o * i * 5 for o, i in mats), "flops": sum(_polar_flops(o, i) for o, i in mats)}
    if kind == "capture":
        rows = case["batch"] * len(sample_positions(case["seq_len"], HEAD, STRIDE))
        return {"bytes": case["layers"] * rows * (3 * 4 * case["hidden"] + 6 * case["mlp"]),
                "flops": case["layers"] * rows * (8 * case["hidden"] + 8 * case["mlp"])}
    if kind == "syrk":
        k, rows, n = case["k"], case["rows"], case["n"]
        return {"bytes": k * (2 * rows * n + 8 * n * n), "flops": k * rows * n * (n + 1)}
    if kind == "polar":
        return {"bytes": 8 * case["batch"] * case["m"] * case["n"],
                "flops": case["batch"] * _polar_flops(case["m"], case["n"], case["steps"])}
    k, n = case["k"], case["n"]
    return {"bytes": k * n * n * (12 if case["q"] > 1 else 8), "flops": k * _root_flops(n, case["q"] > 1)}


def tolerance(case):
    kind, optimizer = case["kind"], case.get("optimizer")
    if kind == "capture":      # BF16 rows: one unit in the last place on the few elements that round the other way
        return {"rel": 1e-3, "max": 1.6e-2}
    if kind == "syrk":         # 32-bit sums
        return {"rel": 2e-5, "max": 1e-3}
    if kind == "polar":        # BF16 operands; the iteration's slope 3.44 at zero multiplies every rounding
        return {"rel": 2e-2, "max": 0.5}
    if kind == "roots":        # products of FP16 hi/lo planes, divided by the smallest eigenvalue
        return {"rel": 5e-4, "max": 2e-2}
    if optimizer == "adamt":   # a moment's sign can turn where the preconditioned gradient is nearly zero
        return {"rel": 5e-3, "max": 0.5}
    return {"rel": 1e-2, "max": 0.2}   # the polar factor's BF16 noise on a change of a few percent of the weight
