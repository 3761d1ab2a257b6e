"""What ActivationStatistics keeps between its calls: sums after a refused commit, row buffers, streams and process groups."""

import threading
import time
import types

import pytest
import torch

from oracle import toner_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tb():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import toner_b200
    return toner_b200


def _layers(widths):
    return {f"l{i}": torch.nn.Linear(n, 16, bias=False).cuda().to(torch.bfloat16) for i, n in enumerate(widths)}


def _forward(stats, layers, rows):
    with stats.capture(), torch.no_grad():
        for layer, x in zip(layers.values(), rows):
            layer(x)


def _rows(layers, count, gen, batch=0):
    """(count, n) rows of every layer, or (batch, count, n) sequences."""
    shape = (batch, count) if batch else (count,)
    return [torch.randn(*shape, layer.in_features, device="cuda", generator=gen).to(torch.bfloat16) for layer in layers.values()]


@pytest.mark.parametrize("batch", [0, 2])     # rows summed in the hook, and sampled rows summed when the capture ends
def test_a_refused_commit_can_be_made_again(tb, batch):
    layers = _layers([64, 64, 40])
    stats = tb.ActivationStatistics(layers, head=1000, stride=1, distributed=False)
    opt = tb.MuonT([l.weight.data.float().requires_grad_() for l in layers.values()], lr=1e-3)
    owned = dict(zip((l.weight for l in layers.values()), opt.param_groups[0]["params"]))
    got = {}

    def update(means):
        got.clear()
        got.update(means)
        opt.update_statistics({owned[w]: m for w, m in means.items()})

    target, gen = types.SimpleNamespace(update_statistics=update), torch.Generator(device="cuda").manual_seed(2)
    first = _rows(layers, 96, gen, batch)
    _forward(stats, layers, first)
    stats.commit(target)
    second, third = _rows(layers, 80, gen, batch), _rows(layers, 48, gen, batch)
    _forward(stats, layers, second)
    with pytest.raises(RuntimeError, match="already updated"):
        stats.commit(target)                      # the first statistics have not been used yet
    for p in opt.param_groups[0]["params"]:
        p.grad = torch.zeros_like(p)
    opt.step()
    _forward(stats, layers, third)                # more rows on top of those that are pending
    stats.commit(target)
    stats.close()
    for layer, a, b in zip(layers.values(), second, third):
        n = layer.in_features
        x = torch.cat([a.reshape(-1, n), b.reshape(-1, n)]).float().cpu()
        assert orc.rel_fro(got[layer.weight].cpu(), orc.gram(x) / x.shape[0]) < 2e-6


def test_row_buffers_are_bounded_where_row_counts_vary(tb, monkeypatch):
    """A new sequence length with every microbatch: what is kept of a width stays below the limit, within a capture and over
    many, and no row is lost when a buffer makes room."""
    limit = 3 * 2 * 40 * 64 * 2            # three buffers of 40 rows for two 64-wide layers
    monkeypatch.setattr(tb.ActivationStatistics, "_ROWS_KEPT", limit)
    layers = _layers([64, 64, 40])
    stats, got = tb.ActivationStatistics(layers, head=1000, stride=1, distributed=False), {}
    gen = torch.Generator(device="cuda").manual_seed(6)
    seen = [[] for _ in layers]
    for lengths in ((20,), (21, 33), (40, 12, 40), (70,), (25,), (26, 27, 28, 20)):
        with stats.capture(), torch.no_grad():
            for length in lengths:         # several lengths within one capture
                for j, (layer, x) in enumerate(zip(layers.values(), _rows(layers, length, gen, batch=1))):
                    layer(x)
                    seen[j].append(x.reshape(-1, layer.in_features).float().cpu())
                for n in (64, 40):
                    assert sum(b.numel() * 2 for key, b in stats._rows.items() if key[0] == n) <= limit
    stats.commit(types.SimpleNamespace(update_statistics=got.update))
    for layer, rows in zip(layers.values(), seen):
        x = torch.cat(rows)
        assert orc.rel_fro(got[layer.weight].cpu(), orc.gram(x) / x.shape[0]) < 2e-6
    assert stats._rows
    stats.close()
    assert not stats._rows


@pytest.mark.parametrize("batch", [0, 3])
def test_layers_on_another_stream(tb, batch):
    """The second layer runs on a side stream, behind a delay, and its input is overwritten there right after; what ends the
    capture and the commit runs on the main stream, which does not wait for the side stream."""
    layers = _layers([64, 64, 64])
    stats, got = tb.ActivationStatistics(layers, head=1000, stride=1, distributed=False), {}
    gen = torch.Generator(device="cuda").manual_seed(8)
    rows, side = _rows(layers, 48, gen, batch), torch.cuda.Stream()
    buf = torch.zeros_like(rows[1])
    side.wait_stream(torch.cuda.current_stream())
    with stats.capture(), torch.no_grad():
        for i, (layer, x) in enumerate(zip(layers.values(), rows)):
            with torch.cuda.stream(side if i == 1 else torch.cuda.current_stream()):
                if i == 1:
                    torch.cuda._sleep(20_000_000)
                    buf.copy_(x)
                    layer(buf)
                    buf.zero_()
                else:
                    layer(x)
    stats.commit(types.SimpleNamespace(update_statistics=got.update))
    stats.close()
    for layer, x in zip(layers.values(), rows):
        x = x.reshape(-1, 64).float().cpu()
        assert orc.rel_fro(got[layer.weight].cpu(), orc.gram(x) / x.shape[0]) < 2e-6
    torch.cuda.synchronize()


def test_layers_in_several_threads(tb):
    """Two layers of one width in two threads: neither takes the other's place among the sums."""

    class Slow(dict):
        def get(self, *args):
            value = super().get(*args)
            time.sleep(0.05)               # another thread may run between the look and the store
            return value

    layers = _layers([64, 64])
    stats, got = tb.ActivationStatistics(layers, distributed=False), {}
    rows = _rows(layers, 48, torch.Generator(device="cuda").manual_seed(9))
    stats._slots = Slow()
    with stats.capture(), torch.no_grad():
        threads = [threading.Thread(target=lambda l=layer, x=x: l(x)) for layer, x in zip(layers.values(), rows)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    stats.commit(types.SimpleNamespace(update_statistics=got.update))
    stats.close()
    for layer, x in zip(layers.values(), rows):
        x = x.float().cpu()
        assert orc.rel_fro(got[layer.weight].cpu(), orc.gram(x) / x.shape[0]) < 2e-6


@pytest.mark.parametrize("when", ["before commit", "between captures", "gone"])
def test_a_process_group_that_comes_or_goes(tb, monkeypatch, when):
    """Sums may be begun before a process group is initialised, or go on after one has been destroyed."""
    from toner_b200 import statistics
    there = [when == "gone"]
    monkeypatch.setattr(statistics.dist, "is_initialized", lambda: there[0])
    monkeypatch.setattr(statistics.dist, "all_reduce", lambda *a, **kw: None)     # (a group of one process)
    layers = _layers([64, 64, 40])
    stats, got = tb.ActivationStatistics(layers, head=1000, stride=1), {}
    gen = torch.Generator(device="cuda").manual_seed(10)
    seen = [[] for _ in layers]
    for step, batch in enumerate((2, 0, 2, 0)):
        rows = _rows(layers, 30 + step, gen, batch)
        _forward(stats, layers, rows)
        for j, x in enumerate(rows):
            seen[j].append(x.reshape(-1, x.shape[-1]).float().cpu())
        if step == 1 and when != "before commit":
            there[0] = not there[0]
    there[0] = when != "gone"
    stats.commit(types.SimpleNamespace(update_statistics=got.update))
    for layer, rows in zip(layers.values(), seen):
        x = torch.cat(rows)
        assert orc.rel_fro(got[layer.weight].cpu(), orc.gram(x) / x.shape[0]) < 2e-6
    stats.close()


def test_a_layer_whose_rows_were_never_summed_is_absent(tb, monkeypatch):
    """Its hook failed after it had been given a place among the sums, and the caller went on."""
    from toner_b200 import ops
    layers = _layers([64, 64])
    stats = tb.ActivationStatistics(layers, distributed=False)
    rows = _rows(layers, 48, torch.Generator(device="cuda").manual_seed(11))
    real = ops.syrk_upper
    with stats.capture(), torch.no_grad():
        layers["l0"](rows[0])
        monkeypatch.setattr(ops, "syrk_upper", lambda *a, **kw: (_ for _ in ()).throw(RuntimeError("refused")))
        with pytest.raises(RuntimeError, match="refused"):
            layers["l1"](rows[1])
        monkeypatch.setattr(ops, "syrk_upper", real)
    with pytest.raises(RuntimeError, match="nothing was captured for layer.*l1"):
        stats.commit(types.SimpleNamespace(update_statistics=lambda means: pytest.fail("committed")))
    stats.close()
