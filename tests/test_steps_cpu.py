"""Steps of higher degree (toner_inv_roots_steps_for): scalars through the stated schedule, over all bounds (no device)."""

import numpy as np
import pytest


@pytest.mark.parametrize("n", [264, 768, 3072])
@pytest.mark.parametrize("p", [2, 4, 8, 16, 32])
def test_the_stated_steps_take_every_eigenvalue_to_its_root(p, n):
    """x = 1, mu = lambda; t = T(mu), x *= t, mu *= t^p per step; then x q(1 - mu) must be lambda^(-1/p) for every lambda the
    bound allows.  mu stays at 1 or below, ends within the stated distance of 1, T^p
    keeps the dynamic range its operand planes resolve (1e3, the grid's miss beside it), and products are saved."""
    from toner_b200 import ops
    used = 0
    for lower in np.geomspace(1.5e-7, 0.3, 60):
        s = ops.inv_roots_steps(float(lower), p, n)
        if s is None:
            continue
        used += 1
        lam = np.unique(np.concatenate([np.geomspace(float(np.float32(lower)), 1.0, 4001), np.linspace(float(np.float32(lower)), 1.0, 4001)]))
        x, mu = np.ones_like(lam), lam.copy()
        for degree, zb, za, kappa, top, lin, con in s["steps"]:
            z = zb + za * mu
            t = con + lin * mu + top * {1: 0.0, 2: z ** 2, 4: (z ** 2 + kappa) ** 2}[degree]
            assert t.min() > 0 and (t.max() / t.min()) ** p < 1.05e3
            x, mu = x * t, mu * t ** p
            assert mu.max() < 1.0 + 1e-6, (p, lower, mu.max())
        assert 1.0 - mu.min() <= s["distance"] + 1e-9, (p, lower)
        q = np.polyval(np.array(s["coefficients"])[::-1], 1.0 - mu)
        assert np.abs(x * q * lam ** (1.0 / p) - 1.0).max() < 5e-6, (p, lower)
        # fewer products than the linear steps for the same bound, single passes by what they take
        linear = (ops.inv_roots_iterations_for(float(lower), p) - 1) * (p.bit_length() + 1)
        single = ops.inv_roots_finish_products(n, 1e-3, p, float(lower))
        weight = 0.35 + 320.0 / n
        assert s["products"][0] + weight * s["products"][1] < linear + weight * single
    assert used >= 30, used
