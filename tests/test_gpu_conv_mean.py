"""A convolution whose activation is only averaged over the positions (``native_ops.conv2d_gelu_mean``): segments of 4 to 32
rows of a brick, images and channels that fill their tiles partly, with and without the pre-activation kept."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("h,w,channels,segment", [
    (12, 40, 512, 32), (4, 8, 256, 32), (9, 31, 256, 32), (4, 4, 288, 16), (6, 20, 512, 8), (7, 20, 256, 4), (13, 8, 320, 8),
    (11, 33, 256, 8), (12, 40, 264, None), (12, 40, 128, None),
])
def test_mean_of_the_activation(h, w, channels, segment, dtype):
    from fbamtrain_b200.ops import native as nv, native_ops as no
    n = 39001 // (h * w) + 1
    g = torch.Generator(device=DEV).manual_seed(h * 100 + w)
    x = torch.randn(n, h, w, 64, device=DEV, generator=g).to(dtype)
    weight = (torch.randn(channels, 3, 3, 64, device=DEV, generator=g) / 24).to(dtype)
    plan = no._pool_plan(n, h, w, channels)
    assert plan is None if segment is None else plan[0] == segment
    z, z_plain = (torch.empty(n, h, w, channels, device=DEV, dtype=dtype) for _ in range(2))
    vec = no.conv2d_gelu_mean(x, weight, 1, 1, 1, z)
    y = no.conv2d_fprop(x, weight, 1, 1, 1, act="gelu", preact_out=z_plain)
    nv.check_status(x.device)
    assert torch.equal(z, z_plain)
    assert torch.equal(no.conv2d_gelu_mean(x, weight, 1, 1, 1, None), vec)
    # one rounding of the mean; y is rounded per position, z within GELU's slope (1.13 at most) of it
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for of in (y.double(), torch.nn.functional.gelu(z.double())):
        want = of.mean((1, 2))
        assert float((vec.double() - want).norm() / want.norm()) < eps
        assert bool(((vec.double() - want).abs() <= 1.2 * eps * (want.abs() + of.abs().mean((1, 2))) + 1e-6).all())


def test_few_tiles_and_single_cta_sizes_keep_the_two_kernels():
    from fbamtrain_b200.ops import native_ops as no
    assert no._pool_plan(4, 12, 40, 512) is None and no._pool_plan(1024, 12, 40, 512) == (32, 15)
    assert no._pool_plan(1024, 11, 33, 512) is None        # a brick of 128 images has one position of each
