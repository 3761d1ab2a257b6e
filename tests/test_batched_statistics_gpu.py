"""Kernels over lists of matrices, and the statistics that are summed for all layers of a width together: edges of the list
length and of the vector loads, captures whose microbatches differ in size, dtype and in the layers they run."""

import pytest
import torch

from oracle import toner_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("count,numel", [(1, 4), (3, 64), (129, 1000), (2, 768 * 768)])
def test_lists(ops, count, numel):
    g = torch.Generator(device="cuda").manual_seed(count)
    src = [torch.randn(numel, device="cuda", generator=g) for _ in range(count)]
    dst = [torch.randn(numel, device="cuda", generator=g) for _ in range(count)]
    want = [0.75 * d.double() + 0.5 * s.double() for d, s in zip(dst, src)]
    ops.list_axpby(src, dst, 0.75, 0.5)
    for d, w in zip(dst, want):
        assert torch.allclose(d.double(), w, rtol=1e-6, atol=1e-6)
    fresh = [torch.full((numel,), float("nan"), device="cuda") for _ in range(count)]
    ops.list_axpby(src, fresh, 0.0, 2.0)                                # beta == 0: what dst held does not matter
    assert all(torch.equal(f, 2.0 * s) for f, s in zip(fresh, src))
    flag = torch.zeros(1, dtype=torch.int32).pin_memory()
    ops.list_finite(src, flag)
    torch.cuda.synchronize()
    assert int(flag[0]) == 0
    for where, value in ((0, float("inf")), (numel - 1, float("nan"))):
        bad = [s.clone() for s in src]
        bad[-1][where] = value
        flag[0] = 0
        ops.list_finite(bad, flag)
        torch.cuda.synchronize()
        assert int(flag[0]) == 1


def test_microbatches_that_differ():
    """Layers of two widths; a second microbatch of another size, a third without autocast (FP32 rows), one of 2-D rows, and
    a layer that runs in only some of them: every mean is the Gram of all of its rows over their number."""
    import toner_b200
    g = torch.Generator().manual_seed(3)
    layers = {"a": torch.nn.Linear(64, 16, bias=False).cuda(), "b": torch.nn.Linear(64, 16, bias=False).cuda(),
              "c": torch.nn.Linear(40, 16, bias=False).cuda()}
    stats = toner_b200.ActivationStatistics(layers, head=4, stride=3, distributed=False)
    for step in range(2):                                             # the second step reuses the first one's buffers
        seen = {name: [] for name in layers}
        plan = [("abc", 3, True), ("ab", 5, True), ("bc", 3, False), ("a", 0, True), ("abc", 3, True)]
        for names, batch, autocast in plan:
            with stats.capture(), torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
                for name in names:
                    n = layers[name].in_features
                    x = torch.randn(*((batch, 23, n) if batch else (37, n)), generator=g)
                    rows = orc.sampled_rows(x, 4, 3) if batch else x
                    seen[name].append(rows.to(torch.bfloat16).float() if autocast else rows)
                    y = x.cuda()
                    layers[name](y)
                    y.zero_()                                         # an activation may be overwritten after its layer ran
        got = {}

        class Recorder:
            def update_statistics(self, means):
                got.update(means)

        stats.commit(Recorder())
        for name, layer in layers.items():
            rows = torch.cat(seen[name])
            # FP32 rows are summed from FP16 hi/lo planes (22 bits), BF16 rows exactly: a few 1e-7 either way
            assert orc.rel_fro(got[layer.weight].cpu(), orc.gram(rows) / rows.shape[0]) < 2e-6, (step, name)
    stats.close()
