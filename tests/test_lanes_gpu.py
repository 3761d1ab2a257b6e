"""Pieces of a step side by side on streams: no piece sees another's scratch, whatever grows while the others run."""

import pytest
import torch

pytestmark = pytest.mark.gpu

# Three lanes: lane 1 runs the second piece and then the fifth, which needs more scratch.
SHAPES = [(64, 136), (64, 64), (136, 64), (128, 128), (520, 264), (264, 72)]


@pytest.fixture(scope="module")
def data():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    g = torch.Generator(device="cuda").manual_seed(4)
    return [(torch.randn(*s, device="cuda", generator=g) * 0.02, torch.randn(*s, device="cuda", generator=g) * 1e-3,
             torch.randn(900, s[1], device="cuda", generator=g)) for s in SHAPES]


def _run(make, groups, data):
    """Weights after two steps; `groups`: the parameter groups, as indices of shapes."""
    params = {i: torch.nn.Parameter(data[i][0].clone()) for group in groups for i in group}
    for i, p in params.items():
        p.grad = data[i][1].clone()
    opt = make([{"params": [params[i] for i in group]} for group in groups])
    for _ in range(2):
        if hasattr(opt, "update_statistics"):
            opt.update_statistics({p: data[i][2].mT @ data[i][2] / 900 for i, p in params.items()})
        opt.step()
    torch.cuda.synchronize()
    return {i: p.detach() for i, p in params.items()}


@pytest.mark.parametrize("groups", [[[0, 1, 2, 3, 4, 5]], [[0, 1, 2], [3, 4, 5]]])
@pytest.mark.parametrize("kind", ["Muon", "MuonT", "AdamT"])
def test_six_shapes_on_three_lanes(data, kind, groups):
    import toner_b200
    from toner_b200 import ops
    from toner_b200.fast import Muon
    make = {"Muon": lambda ps: Muon(ps, lr=0.02, weight_decay=0.1, distributed=False),
            "MuonT": lambda ps: toner_b200.MuonT(ps, lr=0.02, weight_decay=0.1),
            "AdamT": lambda ps: toner_b200.AdamT(ps, lr=1e-3)}[kind]
    together = _run(make, groups, data)
    for i in range(len(SHAPES)):
        assert torch.equal(together[i], _run(make, [[i]], data)[i]), SHAPES[i]
    ops.assert_healthy()
