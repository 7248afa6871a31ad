"""The fused Muon step (momentum, normalisation, Newton–Schulz, update) against the same optimizer on tensor operations,
over both orientations, every gradient type and layouts that it has to leave to the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _optimizers(shape, dtype, momentum, nesterov):
    from fbamtrain_b200.optim.muon import MuonOptimizer
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    base = (0.05 * torch.randn(shape, device=DEV, generator=g)).to(dtype)
    opts = []
    for _ in range(2):
        p = torch.nn.Parameter(base.clone())
        opts.append((p, MuonOptimizer([("w", p)], "o", 2e-2, momentum, nesterov, 0.1)))
    return opts, g


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape,momentum,nesterov", [((8, 8), 0.95, True), ((64, 200), 0.95, True), ((256, 40), 0.9, False),
                                                     ((96, 3, 3, 32), 0.0, False), ((512, 512), 0.95, True),
                                                     ((1032, 264), 0.95, True)])
def test_fused_step_matches_tensor_operations(shape, momentum, nesterov, dtype):
    from fbamtrain_b200.ops import native_ops as no
    ((p, fused), (q, plain)), g = _optimizers(shape, dtype, momentum, nesterov)
    plain._native_step = lambda *a: False
    start = fused._master("w", p).clone()
    for _ in range(3):
        grad = torch.randn(shape, device=DEV, generator=g).to(dtype)
        p.grad, q.grad = grad.clone(), grad.clone()
        rows = shape[0]
        assert no.muon_step_supported(p.grad, rows, p.numel() // rows, fused.state["w"]["momentum"], fused._master("w", p), p.data)
        fused.step()
        plain.step()
    assert torch.allclose(fused.state["w"]["momentum"], plain.state["w"]["momentum"], rtol=1e-5, atol=1e-6)
    a, e = fused._master("w", p), plain._master("w", q)
    # bf16 iterations: the normalised matrix may differ by one bf16 rounding (2^-9) per element between the two
    assert float((a - e).norm() / (e - start).norm()) < 2e-2
    assert torch.equal(p.data, a.to(dtype))


def test_steps_are_reproducible_to_the_bit():
    """Ranks that run the same step on the same gradients have to stay identical."""
    ((p, a), (q, b)), g = _optimizers((640, 1152), torch.bfloat16, 0.95, True)
    for _ in range(2):
        p.grad = torch.randn(640, 1152, device=DEV, generator=g).bfloat16()
        q.grad = p.grad.clone()
        a.step()
        b.step()
    assert torch.equal(a._master("w", p), b._master("w", q)) and torch.equal(p.data, q.data)


@pytest.mark.parametrize("shape", [(12, 64), (64, 20)])
def test_other_layouts_take_the_general_path(shape):
    ((p, a), (q, b)), g = _optimizers(shape, torch.float32, 0.95, True)
    b._native_step = lambda *args: False
    p.grad = torch.randn(shape, device=DEV, generator=g)
    q.grad = p.grad.clone()
    a.step()
    b.step()
    assert torch.equal(p.data, q.data)


def test_parameter_widened_beside_its_master():
    """A model that was widened after its optimizer was built (``model.float()``): fp32 parameter, separate fp32 master."""
    ((p, a), (q, b)), g = _optimizers((64, 128), torch.bfloat16, 0.95, True)
    b._native_step = lambda *args: False
    for t in (p, q):
        t.data = t.data.float()
    p.grad = torch.randn(64, 128, device=DEV, generator=g)
    q.grad = p.grad.clone()
    a.step()
    b.step()
    assert torch.equal(p.data, q.data) and torch.equal(p.data, a._master("w", p))


@pytest.mark.parametrize("nesterov", [True, False])
@pytest.mark.parametrize("momentum", [0.9, 0.95, 0.999, 0.9999])
def test_momentum_has_no_bias(momentum, nesterov):
    """One step from a zero buffer leaves ``(1 - momentum) * grad`` with one rounding of the complement and one of the
    product, 2^-24 each; a complement formed from the rounded momentum is off by up to 2^-25 / (1 - momentum)."""
    from fbamtrain_b200.optim.muon import MuonOptimizer
    g = torch.Generator(device=DEV).manual_seed(3)
    p = torch.nn.Parameter(0.05 * torch.randn(64, 128, device=DEV, generator=g))
    opt = MuonOptimizer([("w", p)], "o", 1e-2, momentum, nesterov, 0.0)
    p.grad = torch.randn(64, 128, device=DEV, generator=g)
    opt.step()
    exact = (1.0 - momentum) * p.grad.double()
    err = (opt.state["w"]["momentum"].double() - exact).abs() / exact.abs()
    assert float(err.max()) < 2 * 2.0 ** -24 * 1.01
