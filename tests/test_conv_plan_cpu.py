"""How a convolution whose activation is averaged is planned (the kernels themselves are tested on the GPU)."""
import pytest

from fbamtrain_b200.ops import native as nv, native_ops as no


def test_plan_follows_the_switch_of_the_pair_kernel(monkeypatch):
    """Sizes that were planned before the pair kernel was switched off, and after, follow the switch."""
    if not nv.available():
        pytest.skip("kernel library not built")
    monkeypatch.setattr(no, "TWO_CTA", "auto")
    assert no._pool_plan(1024, 12, 40, 512) == (32, 15)
    monkeypatch.setattr(no, "TWO_CTA", False)
    assert no._pool_plan(1024, 12, 40, 512) is None
    assert no._pool_plan(1024, 12, 40, 768) is None
    monkeypatch.setattr(no, "TWO_CTA", True)
    assert no._pool_plan(1024, 12, 40, 768) == (32, 15)
