"""What an attention block's norms may be: plain ones, ones with hooks, and other modules in their place."""
import pytest
import torch
from torch import nn
from torch.nn.modules.module import register_module_forward_hook

from fbamtrain_b200.models import AttentionBlock, LayerNorm, RmsNorm
from fbamtrain_b200.models.init_utils import SeedSequence


def _block():
    return AttentionBlock(16, 2, 32, True, True, 1e-5, torch.float32, SeedSequence(3))


def _x():
    return torch.randn(2, 5, 16, generator=torch.Generator().manual_seed(0))


@pytest.mark.parametrize("name", ["ln1", "ln2"])
def test_hooks_get_and_may_replace_a_tensor(name):
    block, x, seen = _block(), _x(), []
    plain = block(x)
    handle = getattr(block, name).register_forward_hook(lambda m, args, out: seen.append((len(args), out)))
    assert torch.equal(block(x), plain)
    handle.remove()
    (n_args, out), = seen
    assert n_args == 1 and isinstance(out, torch.Tensor) and out.shape[-1] == 16
    with_pre = getattr(block, name).register_forward_pre_hook(lambda m, args: (args[0] * 0,))
    assert not torch.equal(block(x), plain)
    with_pre.remove()
    grads = []
    full = getattr(block, name).register_full_backward_hook(lambda m, gi, go: grads.append((len(gi), len(go))))
    block(x.requires_grad_()).sum().backward()
    full.remove()
    assert grads == [(1, 1)]
    assert torch.equal(block(x), plain)


def test_global_hook_gets_tensors():
    block, seen = _block(), []
    handle = register_module_forward_hook(lambda m, args, out: seen.append((type(m), type(out))))
    try:
        block(_x())
    finally:
        handle.remove()
    assert [out for m, out in seen if m is RmsNorm] == [torch.Tensor] * 2


def test_other_modules_in_place_of_a_norm():
    x = _x()

    class Own(RmsNorm):
        def forward(self, x):
            return super().forward(x) * 2

    for norm in (LayerNorm(16, 1e-5, torch.float32), nn.LayerNorm(16), nn.Identity(), Own(16, 1e-5, torch.float32)):
        block = _block()
        block.ln2 = norm
        mid = block.attn(block.ln1(x), residual=x).reshape(-1, 16)
        assert torch.equal(block(x), block.mlp(norm(mid), residual=mid).view(2, 5, 16))


def test_patched_forward_is_called():
    block, x = _block(), _x()
    plain = block(x)
    block.ln1.forward = lambda x: x * 0
    assert not torch.equal(block(x), plain)
    del block.ln1.forward
    original, RmsNorm.forward = RmsNorm.forward, lambda self, x: x * 0
    try:
        assert not torch.equal(block(x), plain)
    finally:
        RmsNorm.forward = original
    assert torch.equal(block(x), plain)
