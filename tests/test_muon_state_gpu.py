"""What the plain Muon keeps between steps: its state, and neither gradients nor workspaces; lanes by what every group adds."""

import weakref

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def muon():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200.fast import Muon
    return Muon


def _params(*shapes):
    g = torch.Generator(device="cuda").manual_seed(1)
    params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=g) * 0.02) for s in shapes]
    for p in params:
        p.grad = torch.randn(*p.shape, device="cuda", generator=g)
    return params


def test_gradients_are_not_kept(muon):
    params = _params((64, 64), (64, 64), (136, 64))
    seen = [weakref.ref(p.grad) for p in params]
    opt = muon(params, lr=0.02, distributed=False)
    opt.step()
    opt.precond = lambda p, grad: grad.half()         # converted copies: of nobody's after the step
    opt.step()
    before = torch.cuda.memory_allocated()
    opt.zero_grad(set_to_none=True)
    assert all(ref() is None for ref in seen)
    assert before - torch.cuda.memory_allocated() == sum(p.numel() * 4 for p in params)


@pytest.mark.parametrize("shapes", [[(512, 512)] * 4, [(256, 512), (512, 256), (512, 512), (512, 1024)]])
def test_workspaces_are_given_back(muon, shapes):
    params = _params(*shapes)
    before = torch.cuda.memory_allocated()
    opt = muon(params, lr=0.02, distributed=False)
    opt.step()
    size = sum(p.numel() * 4 for p in params)
    assert torch.cuda.memory_allocated() - before <= 2 * size + (64 << 10)     # momentum and direction, tables of addresses
    del opt


def test_every_group_has_the_lanes_its_workspaces_allow(muon, monkeypatch):
    """Two small shapes in the first group, two large ones in the second, and a large one whose gradient comes later in the
    first: the limit holds for each, and a group of one shape keeps another group from no lane."""
    from toner_b200 import core
    monkeypatch.setattr(core.Lanes, "MOST_ADDED", 3 << 20)
    small, large = [(64, 64), (64, 136)], [(512, 512), (512, 1024)]
    first, second = _params(*small, (512, 512), (512, 520)), _params(*large)
    late = first[2:]
    kept = [p.grad for p in late]
    for p in late:
        p.grad = None
    opt = muon([{"params": first}, {"params": second}], lr=0.02, distributed=False)
    count = lambda gi: len(opt._lanes[gi][1].scratch)  # noqa: E731
    opt.step()
    assert (count(0), count(1)) == (2, 1)
    for p, g in zip(late, kept):
        p.grad = g
    opt.step()
    assert (count(0), count(1)) == (1, 1)
    opt = muon([{"params": _params((64, 64))}, {"params": _params(*small)}], lr=0.02, distributed=False)
    opt.step()
    assert (count(0), count(1)) == (1, 2)
