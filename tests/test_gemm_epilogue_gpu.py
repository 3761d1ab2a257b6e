"""The GEMM's epilogue at the sizes where its block paths change: remainders of the 32 x 32 blocks and of the tiles, diagonal
blocks of a symmetric result written whole from their upper half, C read for the upper triangle only.  Against FP64 products
of the same 16-bit operands; tolerance as for the products themselves (a few ulp of FP32 times sqrt(k) of accumulation)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200 import ops as _ops
    return _ops


def _rnd(shape, seed, dtype=torch.float32):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


def _close(got, want, k):
    err = (got.double() - want).abs().max().item()
    assert err <= 4e-7 * (k ** 0.5) * want.abs().max().item() + 1e-30, err


@pytest.mark.parametrize("n", [8, 24, 40, 128, 136, 264, 520, 776])
@pytest.mark.parametrize("tile_n", [0, 64, 128, -128, 512])
def test_symmetric_with_c(ops, n, tile_n):
    batch, k = 2, 72
    a = _rnd((batch, n, k), n, torch.bfloat16)
    c = _rnd((batch, n, n), n + 1)
    want = a.double() @ a.double().mT
    want = 0.5 * want + 2.0 * (torch.triu(c.double()) + torch.triu(c.double(), 1).mT)
    c = torch.triu(c) + torch.tril(torch.full_like(c, float("nan")), -1)   # nothing below the diagonal may be used
    d = torch.full((batch, n, n), float("nan"), device="cuda")
    d16 = torch.full((batch, n, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    mx = torch.zeros(batch, device="cuda", dtype=torch.int32)
    ss = torch.zeros(batch, device="cuda")
    op = ops.operand(a)
    ops.gemm(op, op, m=n, n=n, k=k, batch=batch, fmt=1, d=d, d16=d16, c=c, alpha=0.5, beta=2.0, tri=True, mirror=True,
             tile_n=tile_n, maxabs=mx, sumsq=ss)
    ops.assert_healthy()
    _close(d, want, k)
    assert torch.equal(d, d.mT.contiguous()) and torch.equal(d16, d.to(torch.bfloat16))
    assert torch.equal(mx.view(torch.float32), d.abs().amax(dim=(1, 2)))
    assert torch.allclose(ss, d.double().square().sum(dim=(1, 2)).float(), rtol=1e-5)   # n^2 FP32 additions in tree order


@pytest.mark.parametrize("m,n", [(8, 8), (40, 264), (136, 8), (200, 520), (392, 264)])
@pytest.mark.parametrize("tile_n", [0, 64, 128, -128, 256, 512, 1024])
def test_full_result_with_c_in_place(ops, m, n, tile_n):
    batch, k = 2, 136
    a, b = _rnd((batch, m, k), m, torch.bfloat16), _rnd((batch, n, k), n, torch.bfloat16)
    d = _rnd((batch, m, n), m + n)
    want = a.double() @ b.double().mT + 0.25 * d.double()
    guard = torch.full((batch, 8, n), 7.0, device="cuda")
    held = torch.cat([d, guard], dim=1)          # rows below the result must stay untouched
    view = held[:, :m]
    ops.gemm(ops.operand(a), ops.operand(b), m=m, n=n, k=k, batch=batch, fmt=1, d=view, c=view, beta=0.25, tile_n=tile_n)
    ops.assert_healthy()
    _close(view, want, k)
    assert torch.equal(held[:, m:], guard)


@pytest.mark.parametrize("n", [8, 40, 136, 392])
def test_packed_triangle_accumulates(ops, n):
    k = 200
    x = _rnd((3, k, n), n, torch.bfloat16)
    out = torch.full((3, n * (n + 1) // 2), float("nan"), device="cuda")
    ops.syrk_upper(x, out, ops.PACKED)
    ops.syrk_upper(x, out, ops.PACKED_ACC)
    ops.assert_healthy()
    iu = torch.triu_indices(n, n)
    want = 2.0 * (x.double().mT @ x.double())[:, iu[0], iu[1]]
    _close(out, want, k)


@pytest.mark.parametrize("k,rows,n", [(1, 4097, 8), (1, 20001, 136), (2, 9000, 264), (1, 2500, 768), (3, 33000, 520)])
@pytest.mark.parametrize("mode", ["packed", "ema"])
def test_rows_divided_among_ctas(ops, k, rows, n, mode):
    """Few tiles, many rows: each tile's rows are divided among several CTAs (one chain, and chains of 4096 rows)."""
    from toner_b200 import _lib
    assert _lib.load().toner_syrk_workspace_bytes(k, rows, n) > 0
    x = _rnd((k, rows, n), rows + n, torch.bfloat16)
    want = x.double().mT @ x.double()
    got = []
    for _ in range(2):
        if mode == "ema":
            out = torch.ones(k, n, n, device="cuda")
            ops.syrk_upper(x, out, ops.EMA_FULL, 0.5, 1.0 / rows)
            ref = 0.5 + want / rows
        else:
            out = torch.full((k, n * (n + 1) // 2), float("nan"), device="cuda")
            ops.syrk_upper(x, out, ops.PACKED)
            iu = torch.triu_indices(n, n)
            ref = want[:, iu[0], iu[1]]
        got.append(out)
    ops.assert_healthy()
    assert torch.equal(got[0], got[1])           # whichever part comes last, the parts are added in one order
    # the tensor core truncates: up to 1.2e-7 of the sum per 64 rows, over chains of at most 64 such blocks
    err = (got[0].double() - ref).abs().max().item() / ref.abs().max().item()
    assert err < 1.5e-5, err
