"""Which steps a trainer's step graph captures (captures and replays themselves are tested on the GPU)."""
import pytest
import torch

from fbamtrain_b200.utils import step_graph as sg


class _Model(torch.nn.Module):
    frame_chunk = 0


class _Graph:
    """Stands in for a captured step: a replay counts."""

    def __init__(self, log):
        self.cells, self.targets = torch.zeros(0), torch.zeros(0)
        self.graph, self.log = self, log
        self.flops, self.launches, self.loss = (0.0, 0.0), 0, torch.zeros(())

    def replay(self):
        self.log.append("replay")


@pytest.fixture
def graph(monkeypatch):
    log = []
    monkeypatch.setattr(sg.torch.cuda, "current_stream", lambda *a: type("S", (), {"synchronize": lambda s: log.append("wait")})())
    g = sg.StepGraph(_Model(), torch.device("cuda", 0))
    g.log = log
    monkeypatch.setattr(g, "_ordinary", lambda: True)
    monkeypatch.setattr(sg.torch.cuda, "mem_get_info", lambda *a: (64 << 30, 180 << 30))
    g.setting = ("a",)
    monkeypatch.setattr(g, "_setting", lambda: log.append("asked") or g.setting)

    def watched(watch, cells, targets, run):
        watch.steps, watch.host_ms, watch.gpu_ms = watch.steps + 1, 1.0, 1.0
        log.append("usual")
        return torch.zeros(())

    def capture(cells, targets, run):
        log.append("capture")
        captured = _Graph(log)
        captured.cells = captured.targets = torch.empty_like(cells)
        return captured

    monkeypatch.setattr(g, "_watched", watched)
    monkeypatch.setattr(g, "_capture", capture)
    return g


def _steps(g, shapes, n):
    for i in range(n):
        cells = torch.zeros(1, shapes[i % len(shapes)], 1)
        assert g.forward_backward(cells, cells, 1.0, None) is not None
    return {what: g.log.count(what) for what in ("usual", "capture", "replay", "wait")}


@pytest.mark.parametrize("shapes", [[1], [1, 2]])
def test_shapes_that_fit_are_captured_once(graph, shapes):
    seen = _steps(graph, shapes, 60)
    assert seen["usual"] == 2 * len(shapes) and seen["capture"] == len(shapes) and seen["wait"] == 0
    assert seen["replay"] == 60 - 2 * len(shapes)


@pytest.mark.parametrize("n_shapes", [3, 5, 8, 12])
def test_shapes_that_take_turns_are_not_captured_at_every_turn(graph, n_shapes):
    """300 turns: a capture at every turn would be some 290 of each shape; with waits of 2, 4, 8 ... there are at most eight."""
    seen = _steps(graph, list(range(1, n_shapes + 1)), 300 * n_shapes)
    assert seen["capture"] <= 8 * n_shapes and seen["wait"] <= seen["capture"]
    assert len(graph._graphs) <= sg.MAX_GRAPHS and len(graph._watches) <= sg.MAX_WATCHES


def test_a_capture_that_fails_is_not_tried_again(graph, monkeypatch):
    def fails(*a):
        graph.log.append("capture")
        raise RuntimeError("no")
    monkeypatch.setattr(graph, "_capture", fails)
    seen = _steps(graph, [1], 40)
    assert seen["capture"] == 1 and seen["usual"] == 40


def test_graphs_hold_a_part_of_the_free_memory_at_most(graph, monkeypatch):
    """An eighth of what is free: with 8 GB free no graph whose step leaves 0.5 GB for its backward, with 10 GB one; then
    none while it is given back more often than it is replayed."""
    free = [8 << 30]
    monkeypatch.setattr(sg.torch.cuda, "mem_get_info", lambda *a: (free[0], 180 << 30))
    _steps(graph, [1], 2)
    next(iter(graph._watches.values())).kept = 512 << 20
    assert _steps(graph, [1], 10)["capture"] == 0
    free[0] = 10 << 30
    assert _steps(graph, [1], 60)["capture"] == 1
    graph.pool_bytes = 1 << 30
    assert graph.release() == 1 << 30 and not graph._graphs and graph.pool_bytes == 0
    assert _steps(graph, [1], 4)["capture"] == 1          # it has to earn another


@pytest.mark.parametrize("pool,need,fits,released", [
    (0, 80, True, False), (0, 100, True, False), (0, 190, False, False),
    (60, 30, True, False),        # the allocator's own cache, less the graphs', is enough
    (60, 80, True, False),        # with what the driver has free
    (60, 150, True, True),        # with the graphs' memory too
    (60, 190, False, True),
])
def test_memory_of_graphs_is_no_room_for_a_step(pool, need, fits, released, monkeypatch):
    """100 bytes in the allocator's cache, of which the graphs hold ``pool``, and 100 free."""
    from types import SimpleNamespace
    from fbamtrain_b200.train import Trainer
    cuda, gave = torch.cuda, []
    monkeypatch.setattr(cuda, "memory_reserved", lambda *a: 150)
    monkeypatch.setattr(cuda, "memory_allocated", lambda *a: 50)
    monkeypatch.setattr(cuda, "mem_get_info", lambda *a: (100, 1000))
    graphs = SimpleNamespace(pool_bytes=pool, release=lambda: gave.append(pool) or pool)
    assert Trainer._memory_for(SimpleNamespace(_step_graph=graphs, device=None), need) is fits
    assert bool(gave) is released
    assert Trainer._memory_for(SimpleNamespace(_step_graph=None, device=None), need) is (need <= 180)


def test_the_first_step_of_a_shape_asks_for_no_setting(graph):
    """Walking the model takes the host 0.3 ms and more, in which nothing is launched."""
    _steps(graph, [1, 2, 3, 4, 5], 5)
    assert "asked" not in graph.log
    _steps(graph, [1], 1)
    assert graph.log.count("asked") == 1


def test_another_setting_is_watched_anew_and_the_old_graph_comes_back(graph):
    assert _steps(graph, [1], 4)["capture"] == 1
    graph.setting = ("b",)
    graph.log.clear()
    assert _steps(graph, [1], 2) == {"usual": 2, "capture": 0, "replay": 0, "wait": 0}
    assert _steps(graph, [1], 1)["capture"] == 1
    graph.setting = ("a",)
    graph.log.clear()
    assert _steps(graph, [1], 3) == {"usual": 0, "capture": 0, "replay": 3, "wait": 0}
    graph.setting = None                      # hooks on the model: the caller runs the step
    cells = torch.zeros(1, 1, 1)
    assert graph.forward_backward(cells, cells, 1.0, None) is None


def test_settings_in_turn_are_not_captured(graph):
    for i in range(60):
        graph.setting = (i % 3,)
        _steps(graph, [1], 1)
    assert graph.log.count("capture") == 0
