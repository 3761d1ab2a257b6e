"""The fused stages of an update (toner_muont_input, toner_muont_delta, toner_adamt_delta) against the same update put together
from the library's single entry points: the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tb():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200 import core, ops
    return core, ops


def _group(core, ops, kind, out, n, count, first, step, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = first + step * (count - 1) + 1
    f = core.FactorSet(k, n, torch.device("cuda"), (0.5, 0.125), 1e-3, interleave=core.may_reorder(kind))
    x = torch.randn(k, 3 * n, n, device="cuda", generator=g)
    f.ema.copy_(x.mT @ x / (3 * n))
    f.compute()
    assert f.finish() == 0
    weights = [torch.randn(out, n, device="cuda", generator=g) * 0.02 for _ in range(count)]
    grads = lambda: [torch.randn(out, n, device="cuda", generator=g) * 1e-3 for _ in range(count)]  # noqa: E731
    return core.MatrixGroup(weights, f, first, step, kind), grads


def _scratch(group):
    like = lambda *s, t=torch.float32: torch.zeros(*s, device="cuda", dtype=t)  # noqa: E731
    c, shape = group.count, (group.count, group.out_features, group.in_features)
    return dict(work=like(*shape), work2=like(*shape), planes=like(2, *shape, t=torch.float16), inv=like(c),
                maxabs=like(c, t=torch.int32), c1=like(c), c2=like(c))


def _product(ops, s, group, which, d, coarse=False, **kw):
    """d[b] = A[b] R[first + b step], A's planes in the scratch."""
    f, count, n = group.factors, group.count, group.in_features
    r_planes, r_inv = f.planes(which)
    seg_a = (0, 0, 0 if coarse else count)
    seg_b = (group.first, group.first if coarse else f.k + group.first, group.first)
    ops.gemm(ops.operand(s["planes"], seg_z=seg_a), ops.operand(r_planes, seg_z=seg_b, z_step=group.step), m=group.out_features,
             n=n, k=n, batch=count, fmt=0, segs=1 if coarse else 3, d=d, alpha_a=s["inv"], alpha_b=r_inv[group.first:],
             alpha_b_step=group.step, interleave=f.interleave, **kw)


def _decay_term(ops, s, group, d, **kw):
    """d = c1 W R (+ ...) from the hi planes; max |d| in the scratch."""
    ops.split16_list(group.weight_ptrs, group.count, group.out_features, group.in_features, s["planes"], s["inv"], s["maxabs"])
    ops.scale_vec(s["inv"], s["c1"])
    s["maxabs"].zero_()
    _product(ops, s, group, "outer", d, coarse=True, maxabs=s["maxabs"], **kw)
    ops.split16(d, planes=s["planes"], inv_scale=s["inv"], maxabs=s["maxabs"])


@pytest.mark.parametrize("out,n,count,first,step", [(72, 136, 1, 0, 1), (264, 72, 3, 1, 2), (200, 520, 2, 0, 1)])
@pytest.mark.parametrize("wd", [0.0, 0.1])
def test_adamt(tb, out, n, count, first, step, wd):
    core, ops = tb
    group, draw = _group(core, ops, "adamt", out, n, count, first, step, out + n)
    m, v = torch.zeros_like(group.m), torch.zeros_like(group.v)
    lr, b1, b2, eps, f = 2e-3, 0.9, 0.95, 1e-15, group.factors
    scratch, delta, want = core.Scratch(), torch.empty_like(group.m), torch.empty_like(group.m)
    for t in range(1, 9):         # (1 / (1 - b1^t) in FP32 is not the reciprocal of the rounded 1 - b1^t at t = 5, 7, 8)
        grads = draw()
        core.adamt_group_delta(group, grads, delta, scratch, lr=lr, weight_decay=wd, betas=(b1, b2), eps=eps, t=t)
        s, gp = _scratch(group), ops.pointer_table(grads)
        ops.adamt_first_moment(gp, m, b1)
        ops.split16_list(gp, count, out, n, s["planes"], s["inv"], s["maxabs"])
        _product(ops, s, group, "inner", s["work"])
        ops.split16(m, planes=s["planes"], inv_scale=s["inv"], scratch=s["maxabs"])
        _product(ops, s, group, "inner", s["work2"], alpha=1.0 / (1 - b1 ** t))
        ops.adamt_ratio(s["work"], v, s["work2"], b2, 1 - b2 ** t, eps, s["maxabs"])
        before = ops.sumsq(s["work2"])
        ops.split16(s["work2"], planes=s["planes"], inv_scale=s["inv"], maxabs=s["maxabs"])
        _product(ops, s, group, "inner", s["work"])
        ops.adamt_coeffs(f.fro2_outer, first, step, count, n, lr, wd, before, ops.sumsq(s["work"]), s["c1"], s["c2"])
        if wd:
            _decay_term(ops, s, group, s["work2"])
            _product(ops, s, group, "outer", want, alpha=-1.0, c=s["work"], beta=1.0, beta_v=s["c2"])
        else:
            ops.scale_stack(s["work"], s["c2"], want)
        assert torch.equal(delta, want) and torch.equal(group.m, m) and torch.equal(group.v, v), t
    ops.assert_healthy()


@pytest.mark.parametrize("out,n,count,first,step", [(72, 136, 1, 0, 1), (264, 72, 3, 1, 2), (200, 520, 2, 0, 1)])
@pytest.mark.parametrize("wd", [0.0, 0.1])
def test_muont(tb, out, n, count, first, step, wd):
    core, ops = tb
    group, draw = _group(core, ops, "muont", out, n, count, first, step, out + n)
    m = torch.zeros_like(group.m)
    lr, mu, scale = 0.02, 0.95, max(1.0, out / n) ** 0.5
    scratch, delta, want = core.Scratch(), torch.empty_like(group.m), torch.empty_like(group.m)
    for _ in range(2):
        grads = draw()
        core.muont_group_delta(group, grads, delta, scratch, lr=lr, weight_decay=wd, momentum=mu, nesterov=True, ns_steps=3,
                               ns_eps=1e-5)
        s = _scratch(group)
        ops.muont_momentum(ops.pointer_table(grads), m, s["work"], mu, True, s["maxabs"])
        ops.split16(s["work"], planes=s["planes"], inv_scale=s["inv"], maxabs=s["maxabs"])
        _product(ops, s, group, "inner", s["work"])
        ops.ns_polar(s["work"], 3, 1e-5, out=s["work"], maxabs=s["maxabs"])
        ops.muont_coeffs(group.factors.fro2_outer, first, step, count, n, lr, wd, scale, s["c1"], s["c2"])
        if wd:
            _decay_term(ops, s, group, s["work"], c=s["work"], beta=1.0, beta_v=s["c2"])
        else:
            ops.split16(s["work"], planes=s["planes"], inv_scale=s["inv"], maxabs=s["maxabs"])
            ops.scale_vec(s["inv"], s["c2"])
        _product(ops, s, group, "outer", want, alpha=-1.0)
        assert torch.equal(delta, want) and torch.equal(group.m, m)
    ops.assert_healthy()
