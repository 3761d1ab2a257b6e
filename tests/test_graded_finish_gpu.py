"""The graded finish (toner_inv_roots_graded_for): roots of statistics whose lower bound is a verified estimate, with no Newton
step before it and with one or two, against FP64; and what its verification must flag."""

import numpy as np
import pytest
import torch

from oracle import toner_oracle as orc

DAMPING = 1e-3


@pytest.mark.parametrize("n", [64, 768, 5632])
@pytest.mark.parametrize("p", [2, 4, 8, 16])
def test_the_stated_polynomial_takes_every_eigenvalue_to_its_root(p, n):
    """Scalars through the stated Newton steps and the graded polynomial, over all bounds it is used for (no device)."""
    from toner_b200 import ops
    used = set()
    for lower in np.exp(np.linspace(np.log(5e-4), np.log(0.8), 60)):
        lower = float(np.float32(lower))
        g = ops.inv_roots_graded(lower, p, n)
        if g is None:
            continue
        used.add(g["steps"])
        lam = np.exp(np.linspace(np.log(lower), 0.0, 4001))
        x, mu = np.ones_like(lam), lam.copy()
        # (the Newton coefficients depend on the bound and the step alone: those of a longer schedule begin with them)
        for a, b in ops.inv_roots_schedule(lower, p, max(2, g["steps"] + 1))["steps"][:g["steps"]]:
            t = a - b * mu
            x, mu = x * t, mu * t ** p
        zb, za = g["z"]
        z = zb + za * mu
        u, w = 2 * z * z - 1, np.zeros_like(z)
        assert np.abs(z).max() <= 1.0 + 1e-9
        for alpha, beta in g["coefficients"][::-1]:
            w = alpha + beta * z + u * w
        assert np.abs(x * w * lam ** (1.0 / p) - 1).max() < 4e-6, (p, lower, g["steps"])
        assert 0 <= g["split"] <= g["products"] - 2
    assert n < 768 or (0 in used and (p < 8 or n < 2048 or max(used) >= 1)), used


def _stack(spectra, seed):
    """FP32 statistics with the given spectra (unit mean), their exact roots' spectra being known."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    for lam in spectra:
        q, _ = torch.linalg.qr(torch.randn(lam.numel(), lam.numel(), generator=gen, dtype=torch.float64))
        c = (q * lam) @ q.T
        out.append((0.5 * (c + c.T)).float())
    return torch.stack(out)


@pytest.mark.gpu
@pytest.mark.parametrize("n,cond", [(680, 2.0), (776, 2.4), (1000, 6.0), (1288, 12.0), (2056, 30.0), (2048, 100.0)])
@pytest.mark.parametrize("outliers", [0, 2])
def test_roots_against_fp64(n, cond, outliers):
    """Three statistics of one width, factored as the optimizers do until both ends of the spectrum are estimates.  Bounds: an
    error of 3e-6 of the interpolant, 2e-6 of the single passes, the operand planes' 22 bits and short accumulation chains; what
    the Newton steps before it (from condition 30) add is 1e-6 times the spread of the M they leave."""
    from toner_b200 import core, ops
    k = 3
    spectra = []
    for i in range(k):
        gen = torch.Generator().manual_seed(100 * n + i)
        lam = torch.exp(torch.rand(n, generator=gen, dtype=torch.float64) * np.log(cond))
        lam[0], lam[1] = 1.0, cond
        if outliers:
            lam[2:2 + outliers] = cond * 40.0
        spectra.append(lam / lam.mean())
    f = core.FactorSet(k, n, torch.device("cuda"), (0.5, 0.125), DAMPING)
    f.ema.copy_(_stack(spectra, n))
    seen = set()
    for call in range(6):
        f.compute()
        assert f.finish() == 0
        if f._used_estimate:
            g = ops.inv_roots_graded(f._lower_used, f.p, n)
            seen.add(None if g is None else g["steps"])
            for b in range(k):
                c = f.ema[b].cpu()
                e_lo = orc.rel_fro(f.root_lo[b].cpu(), orc.inverse_root_truth(c, 0.125, DAMPING))
                e_hi = orc.rel_fro(f.root_hi[b].cpu(), orc.inverse_root_truth(c, 0.5, DAMPING))
                assert e_lo < (8e-6 if cond < 30 else 2e-5) and e_hi < (3e-5 if cond < 30 else 1e-4), (call, b, e_lo, e_hi)
                assert torch.equal(f.root_lo[b], f.root_lo[b].T)
    ops.assert_healthy()
    assert f.repairs == 0 and f.fallbacks == 0
    assert seen - {None}, "the graded finish was not used"


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["smaller", "larger", "non-finite"])
def test_what_the_interval_does_not_hold_is_flagged(what):
    """Both ends are estimates from earlier calls.  A statistic whose smallest eigenvalue has fallen far below the bound, whose
    bulk has grown past the norm, or that has become non-finite must come back flagged and be repaired, whatever the
    interpolant makes of it."""
    from toner_b200 import core
    n, k = 1000, 2
    lam = torch.exp(torch.linspace(0, 1, n, dtype=torch.float64) * np.log(6.0))
    f = core.FactorSet(k, n, torch.device("cuda"), (0.5, 0.125), DAMPING)
    f.ema.copy_(_stack([lam / lam.mean()] * k, 5))
    for _ in range(5):
        f.compute()
        assert f.finish() == 0
    assert f.lower_is_estimate and f.repairs == 0
    if what == "smaller":
        lam = torch.cat([torch.full((n // 8,), 0.01, dtype=torch.float64), lam[n // 8:]])
    elif what == "larger":
        lam = torch.cat([lam[: -n // 4], 5.0 * lam[-n // 4:]])
    f.ema[0].copy_(_stack([lam / lam.mean()], 6)[0])
    if what == "non-finite":
        f.ema[0, 3, 3] = float("inf")
        f.compute()
        f.status_event.synchronize()
        assert f.status.tolist()[0] == 2 and f.status.tolist()[1] == 0
        return
    f.compute()
    assert f.finish() == 0 and f.repairs >= 1
    for b in range(k):
        c = f.ema[b].cpu()
        assert orc.rel_fro(f.root_lo[b].cpu(), orc.inverse_root_truth(c, 0.125, DAMPING)) < 2e-4
        assert orc.rel_fro(f.root_hi[b].cpu(), orc.inverse_root_truth(c, 0.5, DAMPING)) < 6e-4
