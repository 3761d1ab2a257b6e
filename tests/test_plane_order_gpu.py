"""AdamT's products keep the plane-by-plane order of additions at every lower bound of the spectrum, in both of its
optimizers: where an element of the preconditioned gradient nearly vanishes, another order gives another weight."""

import hashlib
import types

import numpy as np
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


@pytest.mark.parametrize("lower", [1e-3, 6e-3, 0.03, 0.1])
@pytest.mark.parametrize("p,q", [(8, 4), (4, 1)])
def test_the_roots_of_a_statistic_do_not_depend_on_its_batch(ops, lower, p, q):
    """Alone a statistic of width 512 is factored on single-CTA tiles, in a stack of 48 on pair tiles, which interleave plane
    products where they may.  Plane by plane an element's additions come in one order on any tile: the bits are the same."""
    n, k = 512, 48
    g = torch.Generator(device="cuda").manual_seed(int(1e4 * lower) + p)
    basis, _ = torch.linalg.qr(torch.randn(n, n, device="cuda", generator=g))
    ema = torch.empty(k, n, n, device="cuda")
    for i in range(k):
        lam = 1.0 + 0.5 * torch.rand(n, device="cuda", generator=g)
        c = (basis * lam) @ basis.T
        ema[i] = 0.5 * (c + c.T)
    lo, hi, fro2, st = ops.inv_roots(ema, DAMPING, p, q, lower=lower, lower_is_estimate=True, track_sweeps=12, track_restart=True,
                                     track=torch.zeros(k, n, device="cuda"), lmin=torch.empty(k, device="cuda"), interleave=False)
    for i in (0, k - 1):
        one = ops.inv_roots(ema[i:i + 1].contiguous(), DAMPING, p, q, lower=lower, lower_is_estimate=True, track_sweeps=12,
                            track_restart=True, track=torch.zeros(1, n, device="cuda"), lmin=torch.empty(1, device="cuda"),
                            interleave=False)
        assert torch.equal(one[0][0], lo[i]) and torch.equal(one[2][0], fro2[i])
        assert q == 1 or torch.equal(one[1][0], hi[i])
    ops.assert_healthy()
    assert st.tolist() == [0] * k


def _engine(kind, hid, mlp, layers, rows):
    from toner_b200.fast.engine import FastTonerCore
    shapes = dict(q=(hid, hid), k=(hid, hid), v=(hid, hid), attn_proj=(hid, hid), fc=(mlp, hid), mlp_proj=(hid, mlp))
    named = {f"body.blocks.{i}.{role}.weight": torch.nn.Parameter(torch.randn(*s, device="cuda") * 0.02)
             for i in range(layers) for role, s in shapes.items()}
    blocks = [types.SimpleNamespace(input_rows_attn=torch.empty(rows, 1, dtype=torch.bfloat16)) for _ in range(layers)]
    args = types.SimpleNamespace(toner_decay=0.95, toner_split=kind == "muont", toner_alpha=0.25, toner_alpha_in=0.5,
                                 toner_alpha_out=0.125, wd=0.1, beta1=0.9, beta2=0.95, eps=1e-15, muon_momentum=0.95,
                                 muon_nesterov=True, muon_ns_steps=2, muon_eps=1e-5, muon_ns_mode="tpu")
    return FastTonerCore.from_blocks(blocks, named, kind, hid=hid, mlp=mlp, rows_total=rows, args=args, world=1, rank=0,
                                     device=torch.device("cuda", 0))


@pytest.mark.parametrize("kind", ["adamt", "muont"])
def test_the_layer_sharded_engine_keeps_the_order_for_adamt(ops, kind):
    for g in _engine(kind, 64, 128, 1, 96).groups.values():
        assert g.factors.interleave == (kind == "muont")


def _noise(shape, seed):
    """Integers of a bell-shaped distribution, the same everywhere."""
    i = np.arange(int(np.prod(shape)), dtype=np.uint64) + np.uint64(seed << 32)
    out = np.zeros(i.shape, dtype=np.int64)
    for _ in range(4):
        i = (i ^ (i >> np.uint64(31))) * np.uint64(0x9E3779B97F4A7C15)
        out += (i >> np.uint64(58)).astype(np.int64) - 32
    return out.reshape(shape)


# SHA-256 of (root_lo, fro2_lo) after each of five calls, from the engine before its small factorisations (Jacobi, Cholesky) and
# products could take another order: the strengths are equal, so there is one root.
_BITS = {
    (3, 264, 1200, 2, 0): ["4de1a504d3f86bfd", "d450f43f976dc89d", "dc09d693aa93dfdb", "ea193d79780b8382", "3e797a4ade6a9ffc"],
    (2, 264, 1200, 1, 2): ["a30e5a31030530f6", "6994e893ca393110", "ecefb17d25191efe", "a15433bf34014236", "5c93a26fb3926303"],
    (12, 512, 3000, 1, 0): ["a36bfd1ff76892f5", "d55f184a3cf8aa66", "338d4674d2d9c609", "aaa1260a90f7bdac", "cbf178ed872b76f5"],
}


@pytest.mark.parametrize("k,n,rows,mean,spikes", list(_BITS))
def test_factors_keep_their_bits(ops, k, n, rows, mean, spikes):
    """Statistics of integer rows (their Grams are exact) with a dominant mean and outlier directions: the calls go from the
    cold block iteration and the bound that always holds to the warm one, estimated bounds and the norm estimate."""
    from toner_b200 import core
    c = np.empty((k, n, n), dtype=np.float32)
    for b in range(k):
        x = _noise((rows, n), 7 * b + n) + mean * _noise((1, n), 1000 + b)
        for s in range(spikes):
            x = x + _noise((rows, 1), 50 + s + b) * _noise((1, n), 90 + s) // 16
        x = x.astype(np.float64)
        c[b] = (x.T @ x / rows).astype(np.float32)
    c = torch.from_numpy(c).cuda()
    f = core.FactorSet(k, n, torch.device("cuda"), (0.25, 0.25), DAMPING, interleave=False)
    got = []
    for _ in range(5):
        f.ema.copy_(c)
        f.compute()
        assert f.finish() == 0
        h = hashlib.sha256()
        for t in (f.root_lo, f.fro2_lo):
            h.update(t.cpu().numpy().tobytes())
        got.append(h.hexdigest()[:16])
    ops.assert_healthy()
    assert f.repairs == 0 and f.lower_is_estimate
    assert got == _BITS[k, n, rows, mean, spikes]


def _undivided(ops, x):
    """Grams of a (k, rows, n) stack, every tile's rows on one CTA (pair): the entry point without scratch."""
    from toner_b200 import _lib
    k, rows, n = x.shape
    out = torch.zeros(k, n, n, device="cuda")
    _lib.check(_lib.load().toner_syrk_upper(None, x.data_ptr(), x.stride(0), k, rows, n, x.stride(1), out.data_ptr(),
                                            ops.EMA_FULL, 0.0, 1.0, ops._stream()), "toner_syrk_upper")
    return out


@pytest.mark.parametrize("k,n,rows", [(1, 72, 200), (2, 328, 2170), (4, 1064, 3208), (1, 264, 4096), (1, 264, 4097), (1, 768, 8192),
                                      (1, 520, 12289), (9, 512, 48036)])
def test_rows_are_divided_only_where_the_sum_keeps_its_bits(ops, k, n, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(k, rows, n, device="cuda", generator=g).to(torch.bfloat16)
    want = _undivided(ops, x)
    out = torch.full_like(want, float("nan"))
    ops.syrk_upper(x, out, ops.EMA_FULL, 0.0, 1.0, keep_order=True)
    assert torch.equal(out, want)
    packed = torch.empty(k, n * (n + 1) // 2, device="cuda")
    ops.syrk_upper(list(x.unbind(0)), packed, ops.PACKED, keep_order=True)
    r, c = torch.triu_indices(n, n, device="cuda")
    assert torch.equal(packed, want[:, r, c])


def test_activation_statistics_keep_the_bits_of_undivided_sums(ops):
    import toner_b200
    layers = {str(i): torch.nn.Linear(328, 16, bias=False).cuda().to(torch.bfloat16) for i in range(2)}
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(2, 2170, 328, device="cuda", generator=g).to(torch.bfloat16)
    stats, got = toner_b200.ActivationStatistics(layers, distributed=False), {}
    with stats.capture(), torch.no_grad():
        for layer, rows in zip(layers.values(), x):
            layer(rows)
    stats.commit(types.SimpleNamespace(update_statistics=got.update))
    stats.close()
    for layer, sums in zip(layers.values(), _undivided(ops, x)):
        assert torch.equal(got[layer.weight], sums * (1.0 / 2170))


def test_the_layer_sharded_engine_divides_no_chain_for_adamt(ops):
    core = _engine("adamt", 512, 1024, 1, 3000)
    want = []
    for g in core.groups.values():
        g.rows_buf.normal_(generator=torch.Generator(device="cuda").manual_seed(g.n))
        want.append(_undivided(ops, g.rows_buf))
    core._stats()
    torch.cuda.synchronize()
    gamma = (1 - core.decay) / core.rows_total
    for g, sums in zip(core.groups.values(), want):
        assert torch.equal(g.factors.ema, sums * gamma)
