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
