"""Captured steps of several shapes: one pool of memory, graphs given back, captures that fail, streams and half precision."""
import pytest
import torch

from test_gpu_step_graph import _batches, _force, _trainer

pytestmark = pytest.mark.gpu


def _losses(trainer, batches):
    """Losses and gradients of forward and backward alone, so that the steps do not depend on one another."""
    out = []
    for cells, targets in batches:
        trainer.zero_grad()
        loss = float(trainer._forward_backward(cells, targets))
        out.append((loss, [g.grad.clone() for g in trainer.all_groups()]))
    return out


def _same(a, b):
    for (la, ga), (lb, gb) in zip(a, b):
        assert la == pytest.approx(lb, rel=1e-3)
        for x, y in zip(ga, gb):         # sums by atomics in another order: a few roundings of 2^-9 (bf16) or of fp32
            assert float((x.float() - y.float()).norm()) <= 2e-2 * float(y.float().norm()) + 1e-6


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
def test_shapes_in_turn(dtype, monkeypatch):
    """Five shapes in turn, forty rounds: graphs come and go, every result is that of the step launch by launch, and the
    memory of the graphs does not grow with the captures."""
    _force(monkeypatch)
    trainer = _trainer(dtype=dtype)
    lengths = [8, 24, 16, 31, 20]
    batches = [_batches(trainer, 1, frames=n)[0] for n in lengths]
    monkeypatch.setenv("FBAMTRAIN_STEP_GRAPH", "0")
    expected = _losses(trainer, batches)
    monkeypatch.setenv("FBAMTRAIN_STEP_GRAPH", "1")
    captures = []
    capture = trainer._step_graph._capture
    monkeypatch.setattr(trainer._step_graph, "_capture", lambda *a: captures.append(1) or capture(*a))
    sizes = set()
    for i in range(40):
        _same(_losses(trainer, batches), expected)
        if i >= 8:
            sizes.add(trainer._step_graph.pool_bytes)
    assert 5 <= len(captures) <= 5 * 5 and len(trainer._step_graph._graphs) == 2
    assert len(sizes) == 1 and sizes.pop() > 0
    trainer.close()


def test_given_back_and_captured_again(monkeypatch):
    _force(monkeypatch)
    trainer = _trainer()
    batches = _batches(trainer, 2)
    expected = _losses(trainer, batches * 2)[2:]
    _losses(trainer, batches)
    graphs = trainer._step_graph
    assert len(graphs._graphs) == 1
    held = graphs.pool_bytes
    before = torch.cuda.memory_reserved()
    assert graphs.release() == held > 0 and not graphs._graphs and graphs.pool_bytes == 0
    torch.cuda.empty_cache()
    assert torch.cuda.memory_reserved() <= before - held
    _same(_losses(trainer, batches * 3)[-2:], expected)
    assert len(graphs._graphs) == 1
    _same(_losses(trainer, batches), expected)
    trainer.close()
    assert not graphs._graphs and graphs.pool_bytes == 0     # a closed trainer holds none, also while somebody holds it


def test_a_capture_that_fails_leaves_the_step(monkeypatch):
    """The failure is a call that a capture does not allow (the current stream is waited for); the step then runs as usual,
    and the next one is not captured either."""
    _force(monkeypatch)
    trainer = _trainer()
    batches = _batches(trainer, 2)
    expected = _losses(trainer, batches)
    model, calls = trainer.model, []
    forward = type(model).frame_embeddings

    def refuses(self, cells):
        if torch.cuda.is_current_stream_capturing():
            calls.append(1)
            raise RuntimeError("not in a capture")
        return forward(self, cells)

    monkeypatch.setattr(type(model), "frame_embeddings", refuses)
    for _ in range(3):
        _same(_losses(trainer, batches), expected)
    assert calls == [1] and not trainer._step_graph._graphs
    trainer.close()


def test_replayed_on_another_stream(monkeypatch):
    _force(monkeypatch)
    trainer = _trainer()
    batches = _batches(trainer, 2)
    expected = _losses(trainer, batches * 2)[2:]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        _same(_losses(trainer, batches), expected)
    assert len(trainer._step_graph._graphs) == 1
    torch.cuda.synchronize()
    _same(_losses(trainer, batches), expected)
    trainer.close()
