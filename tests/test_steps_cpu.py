"""Steps of higher degree (toner_inv_roots_steps_for): scalars through the stated schedule, over all bounds (no device)."""

import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "toner_b200", "csrc")


def _take(s, lam, steps, p):
    """Scalars lam through these steps of schedule s and its finish."""
    x, mu = np.ones_like(lam), lam.copy()
    for degree, zb, za, kappa, top, lin, con in steps:
        z = zb + za * mu
        t = con + lin * mu + top * {1: 0.0, 2: z ** 2, 4: (z ** 2 + kappa) ** 2}[degree]
        assert t.min() > 0 and (t.max() / t.min()) ** p < 1.05 * (1e3 if degree == 1 else min(400.0, 6.25 * p * p))
        x, mu = x * t, mu * t ** p
        assert mu.max() < 1.0 + 1e-6, (p, lam[0], mu.max())
    assert 1.0 - mu.min() <= s["distance"] + 1e-9, (p, lam[0])
    q = np.polyval(np.array(s["coefficients"])[::-1], 1.0 - mu)
    assert np.abs(x * q * lam ** (1.0 / p) - 1.0).max() < 5e-6, (p, lam[0])


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n", [264, 768, 3072])
@pytest.mark.parametrize("p", [4, 8, 16, 32])
def test_the_stated_steps_take_every_eigenvalue_to_its_root(p, n, kind):
    """x = 1, mu = lambda; t = T(mu), x *= t, mu *= t^p per step; then x q(1 - mu) must be lambda^(-1/p) for every lambda the
    bound allows.  mu stays at 1 or below, ends within the stated distance of 1, T^p
    keeps the dynamic range its products may have (5 % for what the grid misses), and products are saved."""
    from toner_b200 import ops
    used = 0
    for lower in np.geomspace(1.5e-7, 0.3, 60):
        s = ops.inv_roots_steps(float(lower), p, n, kind)
        if s is None:
            continue
        used += 1
        assert s["late"] == 0.0
        lam = np.unique(np.concatenate([np.geomspace(float(np.float32(lower)), 1.0, 4001), np.linspace(float(np.float32(lower)), 1.0, 4001)]))
        _take(s, lam, s["steps"], p)
        # fewer products than the linear steps for the same bound, single passes by what they take
        linear = (ops.inv_roots_iterations_for(float(lower), p) - 1) * (p.bit_length() + 1)
        single = ops.inv_roots_finish_products(n, 1e-3, p, float(lower))
        weight = 0.35 + 320.0 / n
        assert s["products"][0] + weight * s["products"][1] < linear + weight * single
    assert used >= 30, used


@pytest.mark.parametrize("n", [256, 512, 776, 2048, 5632, 16384])
@pytest.mark.parametrize("p", [4, 8, 16, 32])
def test_the_bound_that_always_holds_with_and_without_its_first_step(p, n):
    """All steps for a spectrum down to damping / n, the steps from the second on for one down to the stated bound, which a norm of
    16 puts every spectrum above where one step of degree four gets that far."""
    from toner_b200 import ops
    worst = 1e-3 / (n * 1.001)
    s = ops.inv_roots_steps(worst, p, n, 2)
    lam = lambda low: np.unique(np.concatenate([np.geomspace(low, 1.0, 4001), np.linspace(low, 1.0, 4001)]))
    _take(s, lam(float(np.float32(worst))), s["steps"], p)
    if s["late"]:
        assert s["steps"][1][0] > 1 and s["late"] <= 1e-3 / 16
        _take(s, lam(s["late"]), s["steps"][1:], p)
    assert s["late"] > 0 or p not in (4, 8) or n == 16384     # (not where the second step would be a linear one)


def _turned(steps, coefficients, distance, p, mu0):
    """Of norms that are too low by these factors (the top of M_0's spectrum), those after which the checks of an estimated bound (the
    convergence test's 0.7, the distance with its allowance, 0.03 below zero) see nothing and the root is wrong."""
    x, mu = np.ones_like(mu0), mu0.copy()
    with np.errstate(over="ignore", invalid="ignore"):
        for degree, zb, za, kappa, top, lin, con in steps:
            z = zb + za * mu
            t = con + lin * mu + top * {1: 0.0, 2: z ** 2, 4: (z ** 2 + kappa) ** 2}[degree]
            x, mu = x * t, mu * t ** p
        r = 1.0 - mu
        seen = ~np.isfinite(r) | (np.abs(r) > 0.7) | (r > 1.15 * distance + 1e-3) | (r < -0.03)
        right = np.abs(x * np.polyval(np.array(coefficients)[::-1], r) * mu0 ** (1.0 / p) - 1.0) < 1e-4
    return mu0[~seen & ~right]


@pytest.mark.parametrize("n", [264, 768, 3072])
@pytest.mark.parametrize("p", [4, 8, 16, 32])
def test_a_norm_that_is_too_low_is_seen_or_does_no_harm(p, n):
    """Under an estimated bound the norm is an estimate too, and M_0 may reach above 1.  A schedule with steps of higher degree lets
    through no wrong root that the linear steps for the same bound would not, nothing at all up to a reach of 1.3 for p = 4 and 2
    from p = 8 on: after a step of even degree no linear T follows, whose sign could turn."""
    from toner_b200 import ops
    reach = np.linspace(1.0, 4.0, 30001)
    used = 0
    for lower in np.geomspace(1.5e-7, 0.3, 200):
        s = ops.inv_roots_steps(float(lower), p, n, 0)
        if s is None:
            continue
        used += 1
        degrees = [step[0] for step in s["steps"]]
        assert degrees == sorted(degrees, key=lambda d: d > 1), degrees
        wrong = _turned(s["steps"], s["coefficients"], s["distance"], p, reach)
        assert not (wrong < (1.3 if p == 4 else 2.0)).any(), (lower, degrees, wrong.min())
        if wrong.size:
            linear = ops.inv_roots_schedule(float(lower), p)
            of_linear = _turned([(1, 0.0, 0.0, 0.0, 0.0, -b, a) for a, b in linear["steps"]], linear["coefficients"],
                                linear["distance"], p, reach)
            assert of_linear.size and of_linear.min() <= wrong.min() + 1e-3, (lower, degrees, wrong.min())
    assert used >= 100, used


@pytest.mark.parametrize("n,p,lower", [(264, 8, 0.3), (264, 8, 0.18), (264, 16, 0.108), (384, 8, 0.3), (384, 8, 0.18), (384, 16, 0.0648), (512, 4, 0.18),
                                       (512, 16, 0.18), (512, 16, 0.0648), (768, 4, 0.108), (768, 16, 0.0648)])
def test_no_steps_where_fewer_products_took_longer(n, p, lower):
    """Chains of one and two k-blocks and squarings in short chains make each product dearer.  Here one or two products fewer took 1.04
    to 1.19 times as long as linear steps, whatever the number of statistics (1 to 80)."""
    from toner_b200 import ops
    assert ops.inv_roots_steps(lower, p, n, 1) is None


def test_square_roots_and_narrow_statistics_keep_linear_steps():
    from toner_b200 import ops
    for lower in np.geomspace(1.5e-7, 0.3, 60):
        assert all(ops.inv_roots_steps(float(lower), p, n, kind) is None for p, n in ((1, 768), (2, 768), (8, 248)) for kind in range(3))


BOUNDS = r"""
#include "root_steps.cuh"
#include <cstdio>
int main() {
  using namespace toner;
  int steps = 0;
  for (int p : {4, 8, 16, 32})
    for (int j = 1; j < 256; ++j)
      for (int degree : {2, 4}) {
        NewtonStep s;
        if (!best_step(p, std::exp2(-j / 8.0), degree, std::min(400.0, 6.25 * p * p), s)) continue;
        double z_most = 0.0, y_most = 0.0;
        for (int i = 0; i <= 2000; ++i) {
          const double z = s.zb + s.za * kStepHigh * i / 2000;
          z_most = std::max(z_most, std::fabs(z));
          y_most = std::max(y_most, std::fabs(z * z + s.kappa));
        }
        const bool holds = z_most <= s.most_z && y_most <= s.most_y && s.most_z < 1.001 * z_most && s.most_y < 1.001 * y_most;
        if (!holds) return std::printf("p %d bound %d degree %d: %g %g, %g %g", p, j, degree, z_most, s.most_z, y_most, s.most_y), 1;
        ++steps;
      }
  return std::printf("%d", steps), 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_operand_planes_are_scaled_for_all_that_z_and_its_square_reach(tmp_path):
    """Every step that can be planned states the largest |z| and |z^2 + kappa| on [0, 1.06]: what their FP16 planes are scaled for, a
    factor four below overflow.  (Constants of 1.2 and 1.1 + |kappa| were up to 3.9 and 3.5 times too small.)"""
    (tmp_path / "bounds.cpp").write_text(BOUNDS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(tmp_path / "bounds.cpp"), "-o", str(tmp_path / "bounds")], check=True)
    out = subprocess.run([str(tmp_path / "bounds")], capture_output=True, text=True)
    assert out.returncode == 0 and int(out.stdout) > 1500, out.stdout
