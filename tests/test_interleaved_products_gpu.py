"""Split products with interleaved plane products, the roots' operand planes from the engine's last pass, and groups of work
side by side on streams."""

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


def _planes(x):
    hi = x.half()
    return torch.stack([hi, (x - hi.float()).half()])


@pytest.mark.parametrize("k", [8, 64, 72, 136, 200, 648])          # one k-block and less, odd and even counts, remainders
@pytest.mark.parametrize("promote", [0, 2, 8])
@pytest.mark.parametrize("m,n,tri,tile_n", [(264, 264, True, 512), (520, 136, False, 512), (264, 264, True, -128),
                                            (136, 392, False, -128)])
def test_interleaved_plane_products(ops, m, n, k, promote, tri, tile_n):
    batch = 2
    g = torch.Generator().manual_seed(m + n + k)
    a = _planes(torch.randn(batch, m, k, generator=g).cuda())
    b = a if tri else _planes(torch.randn(batch, n, k, generator=g).cuda())
    d = torch.full((batch, m, n), float("nan"), device="cuda")
    ops.gemm(ops.operand(a, seg_z=(0, 0, batch)), ops.operand(b, seg_z=(0, batch, 0)), m=m, n=n, k=k, batch=batch, fmt=0,
             segs=3, d=d, tri=tri, mirror=tri, promote=promote, tile_n=tile_n, interleave=True)
    ops.assert_healthy()
    ah, al, bh, bl = a[0].double(), a[1].double(), b[0].double(), b[1].double()
    want = ah @ bh.mT + ah @ bl.mT + al @ bh.mT
    # each of the four MMA steps of a k-block and plane product adds into the accumulator by truncation: one unit in the last
    # place (2^-23) of the running sum, which sum |a| |b| bounds; a chain's own length counts, and one rounding per chain
    blocks = -(-k // 64)
    chain = blocks if promote == 0 else min(blocks, promote)
    bound = (12 * chain + -(-blocks // chain) + 2) * 2.0 ** -23 * (ah.abs() @ bh.abs().mT).max().item()
    assert (d.double() - want).abs().max().item() <= bound
    if tri:
        assert torch.equal(d, d.mT.contiguous())


@pytest.mark.parametrize("n,p,q,k,chunk", [(72, 4, 1, 3, 3), (200, 8, 4, 3, 2), (264, 4, 2, 2, 2), (136, 8, 1, 5, 2)])
@pytest.mark.parametrize("block", [False, True])
def test_planes_of_the_roots_are_those_of_split16(ops, n, p, q, k, chunk, block):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(k, 3 * n, n, device="cuda", generator=g)
    x[:, :, 0] *= 30.0                                                # a direction that is deflated and put back
    ema = x.mT @ x / (3 * n)
    new = lambda: torch.empty(2, k, n, n, device="cuda", dtype=torch.float16)  # noqa: E731
    lo_p, hi_p = new(), new() if q > 1 else None
    lo_i, hi_i = torch.empty(k, device="cuda"), torch.empty(k, device="cuda") if q > 1 else None
    kw = {}
    if block:
        kw = dict(deflate=torch.zeros(k, 8, n, device="cuda"), deflate_rank=3, deflate_restart=True,
                  deflated=torch.zeros(k, device="cuda", dtype=torch.int32))
    lo, hi, fro2, st = ops.inv_roots(ema, DAMPING, p, q, chunk=chunk, lo_planes=lo_p, lo_inv=lo_i, hi_planes=hi_p,
                                     hi_inv=hi_i, **kw)
    ops.assert_healthy()
    assert st.tolist() == [0] * k
    for root, planes, inv, s in ((lo, lo_p, lo_i, 1.0 / p), (hi, hi_p, hi_i, q / p)):
        if root is None:
            continue
        bound = torch.full((k,), 1.01 * DAMPING ** -s, device="cuda", dtype=torch.float32).view(torch.int32)
        want, want_inv = torch.empty_like(planes), torch.empty_like(inv)
        ops.split16(root, planes=want, inv_scale=want_inv, maxabs=bound)
        assert torch.equal(planes, want) and torch.equal(inv, want_inv)
    assert torch.equal(fro2, ops.sumsq(lo, out=torch.empty_like(fro2),
                                       scratch=torch.empty(ops.sumsq_scratch_bytes(k), device="cuda", dtype=torch.uint8)))


def test_a_block_of_outliers_needs_no_repair(ops):
    """Eight outlier directions fill the block iteration's eight vectors: the call in which the last one converges must not
    take its norm from a vector that is not there."""
    from toner_b200 import core
    from toner_b200.synthetic import fill_rows_spectrum
    k, n, rows = 2, 512, 4096
    x = torch.empty(k, rows, n, device="cuda", dtype=torch.bfloat16)
    fill_rows_spectrum(x, seed=5, spectrum="spiked:8")
    f = core.FactorSet(k, n, torch.device("cuda"), (0.5, 0.125), DAMPING)
    most = 0
    for _ in range(12):
        ops.syrk_upper(x, f.ema, ops.EMA_FULL, 0.0, 1.0 / rows)
        f.compute()
        assert f.finish() == 0
        most = max(most, int((f.deflated_host & 255).max()))
    assert (f.repairs, f.bound_failures, f.fallbacks) == (0, 0, 0) and most == 8


def test_shapes_side_by_side_give_the_bits_of_each_alone(ops):
    """Four shapes on three lanes: one lane runs two of them, and none may see another's scratch."""
    import toner_b200
    from toner_b200.fast import Muon
    shapes = [(64, 136), (136, 64), (128, 128), (264, 72)]
    g = torch.Generator(device="cuda").manual_seed(1)
    weights = [torch.randn(2, *s, device="cuda", generator=g) * 0.02 for s in shapes]
    grads = [torch.randn(2, *s, device="cuda", generator=g) * 1e-3 for s in shapes]
    rows = [torch.randn(2, 600, s[1], device="cuda", generator=g) for s in shapes]

    def run(which, make):
        params = [torch.nn.Parameter(weights[i][j].clone()) for i in which for j in range(2)]
        for p, (i, j) in zip(params, [(i, j) for i in which for j in range(2)]):
            p.grad = grads[i][j].clone()
        opt = make(params)
        for _ in range(3):
            if hasattr(opt, "update_statistics"):
                opt.update_statistics({p: rows[i][j].mT @ rows[i][j] / 600
                                       for p, (i, j) in zip(params, [(i, j) for i in which for j in range(2)])})
            opt.step()
        torch.cuda.synchronize()
        return [p.detach() for p in params]

    for make in (lambda ps: toner_b200.MuonT(ps, lr=0.02, weight_decay=0.1), lambda ps: toner_b200.AdamT(ps, lr=1e-3),
                 lambda ps: Muon(ps, lr=0.02, weight_decay=0.1, distributed=False)):
        together = run(range(4), make)
        for i in range(4):
            for a, b in zip(together[2 * i:2 * i + 2], run([i], make)):
                assert torch.equal(a, b)
    ops.assert_healthy()
