"""Sums of squares at the sizes where one warp instead of a block takes a partial sum (1024 16-byte accesses), and below a
warp's width."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(8, 8), (24, 40), (296, 4), (512, 512), (1184, 1024), (1184, 1028), (8, 6)])
def test_sum_of_squares(rows, cols):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(3, rows, cols, device="cuda", generator=g)
    got = ops.sumsq(x)
    # positive terms: the relative error is at most the longest chain of additions (a thread's own, 5 levels of a warp, 8
    # warps, 296 partial sums) times 2^-24
    chain = rows * cols / (296 * 1024) + 8 + 5 + 8 + 296
    want = x.double().square().sum(dim=(1, 2))
    assert ((got.double() - want).abs() <= chain * 2.0 ** -24 * want).all()
    for b in range(3):
        assert torch.equal(ops.sumsq(x[b:b + 1].clone()), got[b:b + 1])
