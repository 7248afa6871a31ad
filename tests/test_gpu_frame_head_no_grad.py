"""The fused frame head without gradients (validation, scoring, live frames): pre-activations are not written and nothing
is kept, which may not change the frame vectors, nor what a pass with gradients computes afterwards."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS, COLS, VOCAB = 9, 15, 50


def _problem(dtype, layers, frames):
    g = torch.Generator(device=DEV).manual_seed(layers * 100 + frames)
    cells = torch.stack([torch.randint(0, VOCAB, (frames, ROWS * COLS), device=DEV, generator=g),
                         torch.randint(0, 1 << 24, (frames, ROWS * COLS), device=DEV, generator=g),
                         torch.randint(0, 1 << 24, (frames, ROWS * COLS), device=DEV, generator=g)], -1).int()
    widths = [64, 64, 128, 192][:layers + 1]
    tables = [0.5 * torch.randn(n, 64, device=DEV, generator=g) for n in (VOCAB, ROWS * COLS, 6)]
    weights = [(torch.randn(o, 3, 3, c, device=DEV, generator=g) / (3 * c ** 0.5)).to(dtype)
               for c, o in zip(widths[:-1], widths[1:])]
    d_out = torch.randn(frames, widths[-1], device=DEV, generator=g).to(dtype)
    return cells, tables, weights, d_out


def _run(cells, tables, weights, dtype):
    from fbamtrain_b200 import ops
    n = len(weights)
    return ops.cell_conv_gelu_stack_pool(cells, *tables, ROWS, COLS, dtype, weights, 2, [1] * n, [1] * n)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("frames", [1, 37, 130])          # 130: more than one segment of frames of the table kernel
def test_vectors_and_gradients_do_not_depend_on_it(frames, layers, dtype):
    cells, tables, weights, d_out = _problem(dtype, layers, frames)
    leaves = [t.requires_grad_(True) for t in tables + weights]
    v = _run(cells, tables, weights, dtype)
    grads = torch.autograd.grad(v, leaves, d_out)
    with torch.no_grad():
        assert torch.equal(_run(cells, tables, weights, dtype), v)
    frozen = [t.detach() for t in leaves]
    w = _run(cells, frozen[:3], frozen[3:], dtype)
    assert torch.equal(w, v) and not w.requires_grad
    again = torch.autograd.grad(_run(cells, tables, weights, dtype), leaves, d_out)
    # fp32 sums by atomics in any order, rounded to the 16-bit type on their way through the table products
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, e in zip(again, grads):
        assert float((a.float() - e.float()).norm()) <= eps * float(e.float().norm())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("trainable", range(6))
def test_one_trainable_parameter(trainable, dtype):
    """Gradients are kept as soon as any table or filter asks for them."""
    cells, tables, weights, d_out = _problem(dtype, 3, 37)
    leaves = [t.requires_grad_(True) for t in tables + weights]
    v = _run(cells, tables, weights, dtype)
    want = torch.autograd.grad(v, leaves, d_out)[trainable]
    some = [t.detach().requires_grad_(i == trainable) for i, t in enumerate(leaves)]
    w = _run(cells, some[:3], some[3:], dtype)
    assert torch.equal(w, v)
    (got,) = torch.autograd.grad(w, some[trainable], d_out)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert float((got.float() - want.float()).norm()) <= eps * float(want.float().norm())
