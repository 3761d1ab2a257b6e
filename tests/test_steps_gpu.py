"""Roots after steps of higher degree (toner_inv_roots_steps_for) against FP64, beside those after linear steps."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DAMPING = 1e-3


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200 import ops as _ops
    return _ops


def _statistics(n, cond, k=2):
    g = torch.Generator(device="cuda").manual_seed(n)
    q, _ = torch.linalg.qr(torch.randn(n, n, device="cuda", generator=g, dtype=torch.float64))
    lam = torch.exp(torch.rand(k, n, device="cuda", generator=g, dtype=torch.float64) * torch.tensor(float(cond)).log())
    lam[:, 0], lam[:, -1] = 1.0, cond
    c = ((q * lam[:, None, :]) @ q.T).float()
    return 0.5 * (c + c.mT)


@pytest.mark.parametrize("n", [248, 264, 520])
@pytest.mark.parametrize("p,q", [(2, 1), (4, 1), (8, 4), (8, 1), (16, 8), (32, 2)])
def test_every_path_of_steps(ops, p, q, n):
    """Bounds from the one that always holds to the spectrum's own end take schedules of every degree, first and later, with
    every kind of finish.  Linear steps are what calls in plane order take, all calls below 256 columns and square roots.  Measured, the errors
    are 0.4 times theirs in the median and 1.2 times in the worst (p = 16); 1e-6 q for the operand planes' rounding,
    2^-22 of norms up to four times the root's, the q-th power of it."""
    stats = _statistics(n, 300.0)
    a = stats.double()
    a = a / a.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] + DAMPING * torch.eye(n, device="cuda", dtype=torch.float64)
    lam, vec = torch.linalg.eigh(a)
    norms = torch.zeros(2, device="cuda")
    ops.inv_roots(stats, DAMPING, p, q, norms=norms)
    end = 0.95 * float((lam[:, 0] / norms.double()).min())
    first, later = set(), set()
    for k in range(9):
        lower = end * 0.25 ** k
        if lower <= DAMPING / (n * 1.001):
            break
        steps = ops.inv_roots_steps(lower, p, n)
        degrees = [step[0] for step in steps["steps"]] if steps else []
        first.update(degrees[:1])
        later.update(degrees[1:])
        errors = []
        for interleave in (True, False):
            lo, hi, _, st = ops.inv_roots(stats, DAMPING, p, q, lower=lower, lower_is_estimate=True, interleave=interleave,
                                          track=torch.zeros(2, n, device="cuda"), lmin=torch.empty(2, device="cuda"),
                                          track_sweeps=8, track_restart=True)
            ops.assert_healthy()
            assert st.tolist() == [0, 0], (k, degrees, st.tolist())
            for root, s in ((lo, 1.0 / p), (hi, q / p)):
                if root is not None:
                    want = (vec * lam.pow(-s)[:, None, :]) @ vec.mT
                    errors.append(float((root.double() - want).norm() / want.norm()))
        half = len(errors) // 2
        for got, linear in zip(errors[:half], errors[half:]):
            assert got <= 1.2 * linear + 1e-6 * q, (k, degrees, got, linear)
    assert not first if n < 256 or p < 4 else (4 in first and later), (first, later)


@pytest.mark.parametrize("p,q", [(4, 1), (8, 4), (16, 8)])
@pytest.mark.parametrize("n,rows", [(256, 0.1), (512, 0.17), (768, 0.9), (1280, 0.5)])
def test_directions_the_statistic_is_large_in(ops, p, q, n, rows):
    """Fewer rows than columns, the bound that always holds, the norm's and the spectrum's own: errors weighted by the statistic
    (what a gradient of such activations sees), which the small eigenvalues' share of the Frobenius norm hides.  Measured 0.3 to
    0.6 of the linear steps' in the mean and 1.02 in the worst (p = 8); 1.2 for another draw's rounding."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(2, int(n * rows), n, device="cuda", generator=g) + 0.3 * torch.randn(2, 1, n, device="cuda", generator=g)
    c = x.mT @ x
    c = (0.5 * (c + c.mT)).contiguous()
    a = c.double() / c.double().diagonal(dim1=1, dim2=2).mean(1)[:, None, None]
    lam, vec = torch.linalg.eigh(a + DAMPING * torch.eye(n, device="cuda", dtype=torch.float64))
    norms = torch.zeros(2, device="cuda")
    ops.inv_roots(c, DAMPING, p, q, norms=norms)
    for lower in (0.0, 0.6 * DAMPING / float(norms.max()), 0.5 * float((lam[:, 0] / norms.double()).min())):
        weighted = []
        for interleave in (True, False):
            lo, hi, _, st = ops.inv_roots(c, DAMPING, p, q, lower=lower, interleave=interleave)
            ops.assert_healthy()
            assert st.tolist() == [0, 0]
            for root, s in ((lo, 1.0 / p), (hi, q / p)):
                if root is not None:
                    want = (vec * lam.pow(-s)[:, None, :]) @ vec.mT
                    d = root.double() - want
                    of = lambda m: (m @ a @ m).diagonal(dim1=1, dim2=2).sum(1)
                    weighted.append(float((of(d) / of(want)).max().sqrt()))
        half = len(weighted) // 2
        assert all(got <= 1.2 * linear for got, linear in zip(weighted[:half], weighted[half:])), (lower, weighted)


def _hidden_top(n, low, reach, share):
    """Two statistics whose largest eigenvalue is 1.4 reach times the next, a block of one vector that is the next one's eigenvector but
    for `share` of the top's -- four sweeps gain a factor of ten at most, so the norm comes out near 1.4 times the next -- and A."""
    g = torch.Generator(device="cuda").manual_seed(n)
    q, _ = torch.linalg.qr(torch.randn(n, n, device="cuda", generator=g, dtype=torch.float64))
    lam = low * torch.exp(torch.rand(2, n, device="cuda", generator=g, dtype=torch.float64) * torch.tensor(1.5 / low).log())
    lam[:, 0], lam[:, -2], lam[:, -1] = low, 1.6, 1.6 * 1.4 * reach
    c = ((q * lam[:, None, :]) @ q.T).float()
    stats = (0.5 * (c + c.mT)).contiguous()
    a = stats.double()
    a = a / a.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] + DAMPING * torch.eye(n, device="cuda", dtype=torch.float64)
    lam, vec = torch.linalg.eigh(a)
    block = torch.zeros(2, 8, n, device="cuda")
    block[:, 0] = (vec[:, :, -2] + share * vec[:, :, -1]).float()
    return stats, lam, vec, block


@pytest.mark.parametrize("share", [0.003, 0.03])
@pytest.mark.parametrize("low", [1e-4, 1e-3, 1e-2, 0.05, 0.15])
@pytest.mark.parametrize("p,q", [(8, 4), (4, 1), (16, 8)])
def test_a_norm_above_which_the_spectrum_reaches_is_forgiven_or_flagged(ops, p, q, low, share):
    """The norm as an estimate is too low for a direction the block holds next to nothing of.  Up to a reach of 1.06 T is levelled and
    the roots are right (2e-5 of FP64 from a lower bound of 5e-5); beyond, the statistic is flagged or its root is right all the same."""
    n = 384
    flagged = 0
    for reach in (1.02, 1.05, 1.1, 1.15, 1.2, 1.3, 1.5, 2.0):
        stats, lam, vec, block = _hidden_top(n, low, reach, share)
        lower = 0.5 * float((lam[:, 0] / (1.4 * lam[:, -2])).min())
        steps = ops.inv_roots_steps(lower, p, n)
        if steps is None:      # (linear steps forgive more, and flag where they do not)
            continue
        assert ops.inv_roots_graded(lower, p, n) is None or 2 * q != p
        if steps["steps"][0][0] == 1 and reach > 1.3:     # (where a linear T is negative: as after linear steps alone)
            continue
        norms = torch.zeros(2, device="cuda")
        lo, _, _, st = ops.inv_roots(stats, DAMPING, p, q, lower=lower, lower_is_estimate=True, norms=norms,
                                     track=vec[:, :, 0].float().contiguous(), lmin=torch.empty(2, device="cuda"), track_sweeps=4,
                                     deflate=block, deflate_rank=1, ritz_norm=True)
        ops.assert_healthy()
        reached = (lam[:, -1] / norms.double()).tolist()
        assert all(x <= 1.06 for x in reached) if reach < 1.06 else share > 0.01 or all(x > 1.08 for x in reached), reached
        want = (vec * lam.pow(-1.0 / p)[:, None, :]) @ vec.mT
        error = ((lo.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)).tolist()
        for s, e, x in zip(st.tolist(), error, reached):
            assert s in (1, 4) or e < 1e-4, (low, reach, x, s, e)
            assert x > 1.06 or s == 0, (low, reach, x, s, e)
            flagged += s != 0
    assert flagged > 0 or steps is None


def test_an_overflow_is_the_calls_alone():
    """A norm far too low overflows steps of higher degree although A is finite: status 1, the call is repaired, and the tracked
    vectors stay what they were, so that estimates are used again after the usual eight calls.  A that is not finite is status 2."""
    from toner_b200 import core, ops
    n = 384
    g = torch.Generator(device="cuda").manual_seed(0)
    q, _ = torch.linalg.qr(torch.randn(n, n, device="cuda", generator=g, dtype=torch.float64))

    def statistic(top):
        lam = torch.linspace(1e-3, 1.5, n, device="cuda", dtype=torch.float64)
        lam[-1], lam[-2] = 1.6, 1.6 * top
        c = ((q * lam) @ q.T).float()
        return (0.5 * (c + c.T)).expand(2, n, n).contiguous()

    f = core.FactorSet(2, n, torch.device("cuda"), (0.5, 0.125), DAMPING, slots=12)
    used = []
    for call in range(18):
        f.ema.copy_(statistic(0.9 if call < 6 else 2.1))
        if call == 6:          # the block knows every large direction but the one that is now the largest
            for j in range(f.deflate.shape[1]):
                f.deflate[:, j] = q[:, n - 1 if j == 0 else n - 2 - j].float()
        f.compute()
        torch.cuda.synchronize()
        used.append(f._used_estimate)
        assert f.status.tolist() == ([1, 1] if call == 6 else [0, 0]), (call, f.status.tolist())
        assert torch.isfinite(f.root_lo).all().item() == (call != 6)
        f.finish()
        assert torch.isfinite(f.track).all() and torch.isfinite(f.root_lo).all()
    assert used[6] and f.repairs == 2 and f.fallbacks == 0 and all(used[-3:]), used
    bad = statistic(2.1)
    bad[1, 5, 5] = float("inf")
    _, _, _, st = ops.inv_roots(bad, DAMPING, 8, 4, lower=1e-4, lower_is_estimate=True, track=torch.ones(2, n, device="cuda"),
                                lmin=torch.empty(2, device="cuda"), track_sweeps=4, deflate=f.deflate[:, :8].contiguous(), deflate_rank=4, ritz_norm=True)
    ops.assert_healthy()
    assert st.tolist()[1] == 2, st.tolist()


@pytest.mark.parametrize("p,q", [(4, 1), (8, 4)])
@pytest.mark.parametrize("n", [264, 1032, 1288, 2056])
def test_a_first_step_left_out_by_some_statistics(ops, p, q, n):
    """(From 1288 columns on with planes stored by half.)  The bound that always holds: statistics of a small norm start with the second step, those of a large one (two directions of one
    size, which are not deflated) with the first.  Each comes out as beside others of its kind, and as close to FP64 as linear steps
    bring it."""
    small = _statistics(n, 300.0)
    spikes = _statistics(n, 30.0, 1)
    g = torch.Generator(device="cuda").manual_seed(3)
    d, _ = torch.linalg.qr(torch.randn(n, 2, device="cuda", generator=g))
    spikes = spikes + (d @ d.T) * spikes.diagonal(dim1=1, dim2=2).sum(1)[:, None, None]
    stats = torch.cat([small[:1], spikes, small[1:]]).contiguous()
    late = ops.inv_roots_steps(DAMPING / (n * 1.001), p, n, 2)["late"]
    norms = torch.zeros(3, device="cuda")
    lo, hi, _, st = ops.inv_roots(stats, DAMPING, p, q, norms=norms)
    ops.assert_healthy()
    assert st.tolist() == [0, 0, 0]
    starts_late = [DAMPING / x > late for x in norms.tolist()]
    assert late > 0 and starts_late == [True, False, True], (late, norms.tolist())
    a = stats.double()
    a = a / a.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] + DAMPING * torch.eye(n, device="cuda", dtype=torch.float64)
    lam, vec = torch.linalg.eigh(a)
    linear = ops.inv_roots(stats, DAMPING, p, q, interleave=False)
    for root, plain, s in ((lo, linear[0], 1.0 / p), (hi, linear[1], q / p)):
        if root is None:
            continue
        want = (vec * lam.pow(-s)[:, None, :]) @ vec.mT
        got, ref = [(x.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1) for x in (root, plain)]
        assert (got <= 1.2 * ref + 1e-6 * q).all(), (got.tolist(), ref.tolist())
    for b in range(3):
        own = ops.inv_roots(stats[b:b + 1].expand(3, n, n).contiguous(), DAMPING, p, q)     # (of one tile choice: three as well)
        assert torch.equal(own[0][b], lo[b]) and (hi is None or torch.equal(own[1][b], hi[b]))
