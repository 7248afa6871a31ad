"""A replayed step follows what its launches depend on: with a setting changed, the step runs as usual (or as a graph of its
own) and never as the graph that was captured under the other setting."""
import pytest
import torch

from test_gpu_step_graph import _batches, _force, _trainer

pytestmark = pytest.mark.gpu


def _no_replay(trainer, monkeypatch):
    for graph in trainer._step_graph._graphs.values():
        monkeypatch.setattr(graph, "graph", type("Never", (), {"replay": lambda self: pytest.fail("replayed")})())


@pytest.mark.parametrize("what", ["float32 products", "float32 products, setter", "convolutions", "class forward", "epsilon",
                                  "configuration", "SMs left free"])
def test_changed_setting_is_not_passed_by(what, monkeypatch):
    from fbamtrain_b200.models import RmsNorm
    from fbamtrain_b200.ops import native
    _force(monkeypatch)
    trainer = _trainer()
    batch = _batches(trainer, 1)[0]
    for _ in range(4):
        trainer.train_step(*batch)
        torch.cuda.synchronize()
    assert len(trainer._step_graph._graphs) == 1
    precision = torch.get_float32_matmul_precision()
    _no_replay(trainer, monkeypatch)
    norm = next(m for m in trainer.model.modules() if isinstance(m, RmsNorm))
    try:
        if what == "float32 products":
            torch.backends.cuda.matmul.allow_tf32 = True
        elif what == "float32 products, setter":
            torch.set_float32_matmul_precision("medium")
        elif what == "convolutions":
            monkeypatch.setattr(torch.backends.cudnn, "deterministic", True)
        elif what == "class forward":
            old = RmsNorm.forward
            monkeypatch.setattr(RmsNorm, "forward", lambda self, *a, **k: old(self, *a, **k))
        elif what == "epsilon":
            norm.eps = 1e-3
        elif what == "configuration":
            trainer.model.cfg.use_fp16_accumulation = not trainer.model.cfg.use_fp16_accumulation
        else:
            native.lib().fbam_set_reserved_sms(16)
        assert torch.isfinite(trainer.train_step(*batch))
        torch.cuda.synchronize()
    finally:
        torch.backends.cuda.matmul.allow_tf32 = False
        torch.set_float32_matmul_precision(precision)
        native.lib().fbam_set_reserved_sms(0)
    trainer.close()
