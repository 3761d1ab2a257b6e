"""State of the general optimizers in unusual but legal circumstances: empty parameter groups, a step that is refused."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tb():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import toner_b200
    return toner_b200


def _params(*shapes):
    g = torch.Generator(device="cuda").manual_seed(3)
    params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=g) * 0.02) for s in shapes]
    for p in params:
        p.grad = torch.randn(*p.shape, device="cuda", generator=g) * 1e-3
    return params


def _statistics(params):
    g = torch.Generator(device="cuda").manual_seed(4)
    rows = [torch.randn(300, p.shape[1], device="cuda", generator=g) for p in params]
    return {p: x.T @ x / 300 for p, x in zip(params, rows)}


@pytest.mark.parametrize("kind", ["MuonT", "AdamT"])
def test_a_first_group_without_parameters(tb, kind):
    results = []
    for groups in (lambda p: [{"params": []}, {"params": p}], lambda p: [{"params": p}]):
        params = _params((64, 72), (72, 64))
        opt = getattr(tb, kind)(groups(params), lr=1e-3)
        opt.update_statistics(_statistics(params))
        opt.step()
        results.append([p.detach().clone() for p in params])
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_a_refused_adamt_step_counts_for_nobody(tb):
    """Two parameters of one shape that have taken different numbers of steps are refused; those of the shape before them must
    not count a step that changed no weight."""
    first, second = _params((64, 72)), _params((72, 64), (72, 64))
    params = first + second
    opt = tb.AdamT(params, lr=1e-3)
    opt.update_statistics(_statistics(params))
    opt.step()
    weights = [p.detach().clone() for p in params]
    opt.state[second[0]]["step"] = 5
    opt.update_statistics(_statistics(params))
    with pytest.raises(RuntimeError, match="same number of steps"):
        opt.step()
    assert [opt.state[p]["step"] for p in params] == [1, 5, 1]
    assert all(torch.equal(p, w) for p, w in zip(params, weights))
