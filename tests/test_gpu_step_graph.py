"""Launch-bound training steps as a graph: same losses and weights as launch by launch, and no graph where something is
active that a replay would pass by."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _trainer(kind="toy", dtype="bf16"):
    from fbamtrain_b200 import RunConfiguration, Trainer, presets
    d = presets.fbam_toy()
    if kind == "muon":
        d["optimizer"].update({"type": "muon", "learning_rate": 2e-3, "momentum": 0.9, "nesterov": True})
    d["model_config"]["dtype"] = dtype
    d["micro_batch_size"] = d["total_batch_size"] = 2
    d["train_sequence_length"] = 24
    return Trainer(RunConfiguration.from_json(d), device=torch.device("cuda", 0))


def _batches(trainer, n, frames=24, host=False):
    from fbamtrain_b200.data import SyntheticBatchSource
    cfg = trainer.cfg
    out = []
    for i in range(n):
        src = SyntheticBatchSource(cfg.frame_rows, cfg.frame_cols, cfg.model_config.max_code_point, trainer.vocab, seed=i)
        cells, targets = src.next_batch(2, frames)
        out.append((cells, targets) if host else (cells.cuda(), targets.cuda()))
    return out


def _graphs(trainer):
    return len(trainer._step_graph._graphs)


def _force(monkeypatch):
    """Captures from the third step on whatever the host's speed."""
    from fbamtrain_b200.utils import step_graph
    monkeypatch.setattr(step_graph, "HOST_SHARE", 0.0)


def _run(trainer, batches):
    losses = []
    for cells, targets in batches:
        losses.append(trainer.train_step(cells, targets))
        torch.cuda.synchronize()
    return losses, [g.data.clone() for g in trainer.all_groups()]


@pytest.mark.parametrize("kind", ["toy", "muon"])
@pytest.mark.parametrize("host", [False, True])
def test_same_steps_with_and_without(kind, host, monkeypatch):
    from fbamtrain_b200.ops import native
    from fbamtrain_b200.utils import flops
    _force(monkeypatch)
    runs = []
    for switch in ("0", "0", "1"):
        monkeypatch.setenv("FBAMTRAIN_STEP_GRAPH", switch)
        trainer = _trainer(kind)
        batches = _batches(trainer, 6, host=host)
        flops0, launches0 = flops.snapshot(), native.launches()
        losses, weights = _run(trainer, batches)
        assert _graphs(trainer) == int(switch)
        counted = (flops.snapshot()[0] - flops0[0], flops.snapshot()[1] - flops0[1], native.launches() - launches0)
        runs.append((torch.stack([l.reshape(()) for l in losses]).cpu(), weights, counted))
        trainer.close()
    (la, wa, ca), (lb, wb, _), (lc, wc, cc) = runs
    assert ca == pytest.approx(cc)
    # two runs launch by launch differ by the order of atomic adds (a gradient that is zero up to rounding moves its weight
    # by the learning rate either way); the graph may differ by no more than a few times that
    spread = float((la - lb).abs().max())
    assert float((la - lc).abs().max()) <= 4 * spread + 1e-3
    for a, b, c in zip(wa, wb, wc):
        apart = float((a.float() - b.float()).norm() / a.float().norm())
        assert float((a.float() - c.float()).norm() / a.float().norm()) <= 4 * apart + 2e-3
    assert len({float(x) for x in lc}) == 6                 # every loss is a tensor of its own


def test_new_inputs_shapes_and_storage(monkeypatch):
    """Other inputs of the shape are used; another shape, and parameters that lie elsewhere, have graphs of their own."""
    _force(monkeypatch)
    trainer = _trainer()
    a, b = _batches(trainer, 2)
    for _ in range(3):
        trainer.train_step(*a)
        torch.cuda.synchronize()
    assert _graphs(trainer) == 1
    before = [g.data.clone() for g in trainer.all_groups()]
    trainer.zero_grad()
    loss_a = float(trainer._forward_backward(*a))
    grads_a = [g.grad.clone() for g in trainer.all_groups()]
    trainer.zero_grad()
    loss_b = float(trainer._forward_backward(*b))
    assert loss_a != loss_b
    trainer.zero_grad()
    assert float(trainer._forward_backward(*a)) == pytest.approx(loss_a, rel=1e-3)
    trainer._forward_backward(*a)                           # gradients add up, as launch by launch
    for g, one in zip(trainer.all_groups(), grads_a):
        assert float((g.grad.float() - 2 * one.float()).norm()) <= 2e-2 * float(one.float().norm()) + 1e-6
    assert all(torch.equal(g.data, x) for g, x in zip(trainer.all_groups(), before))     # forward and backward alone
    short = [(c[:, :16].contiguous(), t[:, :16].contiguous()) for c, t in (a, b)]
    for i in range(4):
        trainer.train_step(*short[i % 2])
        torch.cuda.synchronize()
    assert _graphs(trainer) == 2
    p = next(trainer.model.action_model.parameters())
    moved = p.data.clone()
    p.data = moved
    trainer.zero_grad()
    moved.mul_(1.5)
    changed = float(trainer._forward_backward(*a))
    monkeypatch.setenv("FBAMTRAIN_STEP_GRAPH", "0")
    trainer.zero_grad()
    assert changed == pytest.approx(float(trainer._forward_backward(*a)), rel=1e-3)
    trainer.close()


@pytest.mark.parametrize("what", ["module hook", "parameter hook", "saved tensors", "debug", "patched forward", "plan"])
def test_what_a_replay_would_pass_by(what, monkeypatch):
    _force(monkeypatch)
    from fbamtrain_b200.utils import debug, plan
    trainer = _trainer()
    batch = _batches(trainer, 1)[0]
    for _ in range(3):
        trainer.train_step(*batch)
        torch.cuda.synchronize()
    seen = []
    graph = next(iter(trainer._step_graph._graphs.values()))
    monkeypatch.setattr(graph, "graph", type("Never", (), {"replay": lambda self: pytest.fail("replayed")})())
    step = lambda: trainer.train_step(*batch)  # noqa: E731
    if what == "module hook":
        handle = trainer.model.action_model.lstm.register_forward_hook(lambda *a: seen.append(1))
        step()
        handle.remove()
    elif what == "parameter hook":
        next(trainer.model.parameters()).register_hook(lambda g: seen.append(1))
        step()
    elif what == "saved tensors":
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(1), t)[1], lambda t: t):
            step()
    elif what == "debug":
        monkeypatch.setattr(debug, "SYNC_EVERY_OP", True)
        step()
        seen.append(1)
    elif what == "patched forward":
        lstm = trainer.model.action_model.lstm
        old = lstm.forward
        lstm.forward = lambda *a: (seen.append(1), old(*a))[1]
        step()
    else:
        with plan.record() as recorded:
            step()
        seen += recorded.entries
    assert seen
    trainer.close()
