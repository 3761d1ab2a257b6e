"""Operand planes of the factor engine stored by half (stacks of 4 Mi elements and more): the same roots as from whole planes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DAMPING = 1e-3


@pytest.fixture(autouse=True, scope="module")
def _give_back():
    yield
    torch.cuda.empty_cache()     # (gigabytes, of which later tests that count memory would be handed pieces)


@pytest.mark.parametrize("n,k", [(264, 64), (520, 16), (768, 8), (1000, 5), (1288, 3), (2040, 2)])
@pytest.mark.parametrize("p,q", [(8, 4), (4, 1), (2, 1)])
def test_the_same_roots_as_from_whole_planes(n, k, p, q):
    """A workspace for a few statistics makes the call go through them in chunks below the size from which planes are stored by half.
    In plane order an element's sum does not depend on the tile, so the roots are the same bits; interleaved they are as close to
    FP64 (1 % for other tiles; not after linear steps, p = 2, whose long chains follow the tile whoever stores what: 1.34 times with
    whole planes too).  Widths off and on the blocks of 256 and the tiles; the bound that always holds, then an estimate with deflated
    directions and, for 2 q = p, the graded finish."""
    from toner_b200 import ops
    assert k * n * n >= 4 << 20
    few = ((4 << 20) - 1) // (n * n)
    assert few >= 1
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(k, 3 * n, n, device="cuda", generator=g)
    x[:, :, 0] *= 30.0
    ema = x.mT @ x / (3 * n)
    ema = (0.5 * (ema + ema.mT)).contiguous()
    del x
    a = ema.double()
    a = a / a.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] + DAMPING * torch.eye(n, device="cuda", dtype=torch.float64)
    lam, vec = torch.linalg.eigh(a)
    want = [(vec * lam.pow(-s)[:, None, :]) @ vec.mT for s in (1.0 / p, q / p)]
    del a, vec
    small = torch.empty(ops.inv_roots_workspace_bytes(few, n), device="cuda", dtype=torch.uint8)
    large = torch.empty(ops.inv_roots_workspace_bytes(k, n), device="cuda", dtype=torch.uint8)
    for interleave in (False, True) if p >= 4 else (False,):
        states = [dict(track=torch.zeros(k, n, device="cuda"), lmin=torch.zeros(k, device="cuda"), norms=torch.zeros(k, device="cuda"),
                       deflate=torch.zeros(k, 8, n, device="cuda")) for _ in range(2)]
        lower = 0.0
        for call in range(3):
            out = []
            for ws, kw in zip((small, large), states):
                lo, hi, fro, st = ops.inv_roots(ema, DAMPING, p, q, workspace=ws, lower=lower, lower_is_estimate=lower > 0,
                                                track_sweeps=8, track_restart=call == 0, deflate_rank=3, deflate_restart=call == 0,
                                                interleave=interleave, ritz_norm=call == 2, **kw)
                ops.assert_healthy()
                # (768 columns, p = 4, in plane order: linear steps that end at 0.527 of I are converged)
                assert st.tolist() == [0] * k, (call, st.tolist())
                out.append((lo, hi))
            for whole, half, w in zip(*out, want):
                if whole is None:
                    continue
                assert torch.equal(half, half.mT)
                if not interleave:
                    assert torch.equal(whole, half), call
                errors = [float(((r.double() - w).flatten(1).norm(dim=1) / w.flatten(1).norm(dim=1)).mean()) for r in (whole, half)]
                assert errors[1] <= 1.01 * errors[0] + 2e-8, (call, errors)
            lower = 0.5 * float((states[0]["lmin"] / states[0]["norms"]).min())


@pytest.mark.parametrize("n", [2048, 2056, 3072])
@pytest.mark.parametrize("p,q", [(8, 4), (4, 1)])
def test_widths_of_which_one_statistic_is_a_large_stack(n, p, q):
    """From 2048 columns on there is no call on whole planes to compare with, but a block read from the wrong place is of the root's own
    size.  The limit: truncation is 1.2e-7 a k-block of 64 in one chain, in each of the linear steps' products with X and as much again
    for the powers of T; q times that for the root's q-th power."""
    from toner_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(2, 2 * n, n, device="cuda", generator=g)
    x[:, :, 0] *= 30.0
    ema = x.mT @ x / (2 * n)
    ema = (0.5 * (ema + ema.mT)).contiguous()
    del x
    a = ema.double()
    a = a / a.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] + DAMPING * torch.eye(n, device="cuda", dtype=torch.float64)
    lam, vec = torch.linalg.eigh(a)
    lower = 0.5 * float((lam[:, 0] / lam[:, -2]).min())
    limit = 2 * ops.inv_roots_iterations(n, DAMPING, p) * (n / 64) * 1.2e-7
    for interleave in (False, True):
        for bound in (0.0, lower):
            lo, hi, _, st = ops.inv_roots(ema, DAMPING, p, q, lower=bound, lower_is_estimate=bound > 0, interleave=interleave,
                                          track=torch.zeros(2, n, device="cuda"), lmin=torch.zeros(2, device="cuda"), track_sweeps=8,
                                          track_restart=True, deflate=torch.zeros(2, 8, n, device="cuda"), deflate_rank=3, deflate_restart=True)
            ops.assert_healthy()
            assert st.tolist() == [0, 0]
            for root, s, most in ((lo, 1.0 / p, limit), (hi, q / p, q * limit)):
                if root is not None:
                    want = (vec * lam.pow(-s)[:, None, :]) @ vec.mT
                    assert torch.equal(root, root.mT)
                    assert float(((root.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)).max()) < most


@pytest.mark.parametrize("n,k,p,q", [(128, 260, 8, 4), (264, 64, 2, 1), (264, 64, 8, 4), (432, 24, 4, 1)])
def test_narrow_stacks_keep_their_tiles(n, k, p, q):
    """Below 440 columns (512 for linear steps) the tile that half storage needs costs more than the mirror images, and interleaved products
    round by their tile: a few statistics fewer, below the size from which planes are stored by half, take the same one and come out alike."""
    from toner_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(k, 2 * n, n, device="cuda", generator=g)
    ema = x.mT @ x
    ema = (0.5 * (ema + ema.mT)).contiguous()
    fewer = ((4 << 20) - 1) // (n * n)
    few, every = [ops.inv_roots(ema, DAMPING, p, q, workspace=torch.empty(ops.inv_roots_workspace_bytes(c, n), device="cuda", dtype=torch.uint8))[0]
                  for c in (fewer, k)]
    ops.assert_healthy()
    assert fewer < k and torch.equal(few[:fewer], every[:fewer])
