"""The row-wise and column-wise kernels at the edges of their launch rules: single rows, partial rounds of the warps of a
block, more rows than one pass of the grid, and column counts on both sides of every vector width."""
import pytest
import torch

from fbamtrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, e):
    return float((a.detach().double() - e).norm() / e.norm().clamp_min(1e-30))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 64), (65, 256), (9, 264), (700, 512), (33, 1000), (20000, 128), (9001, 1024),
                                      (17, 2048), (5, 4096), (2, 64), (7, 72), (31, 56), (65, 128), (40001, 64),
                                      (20003, 120), (1, 2048), (2, 1536), (9, 136)])
def test_rmsnorm_backward(rows, dim, dtype):
    from fbamtrain_b200.ops import native_ops as no
    g = torch.Generator(device=DEV).manual_seed(rows + dim)
    x = torch.randn(rows, dim, device=DEV, generator=g).to(dtype).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(dim, device=DEV, generator=g)).to(dtype).requires_grad_(True)
    dy = torch.randn(rows, dim, device=DEV, generator=g).to(dtype)
    dx, dw = torch.autograd.grad(no.rms_norm(x, w, 1e-5), (x, w), dy)
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    ex, ew = torch.autograd.grad(y, (xd, wd), dy.double())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11       # one rounding of the result, relative to its norm
    assert _rel(dx, ex) < eps and _rel(dw, ew) < eps


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dim", [24, 328, 488, 656, 1312, 2624])
def test_rmsnorm_backward_mean_is_a_division(dim, dtype):
    """Rows of ones: the mean is dim / dim = 1 and the gradient exactly zero.  dim times a rounded 1 / dim is not 1 for
    most of these sizes, and leaves 6e-8."""
    import ctypes as C
    from fbamtrain_b200.ops import native as nv
    x = torch.ones(3, dim, device=DEV, dtype=dtype)
    w, rstd = torch.ones(dim, device=DEV, dtype=dtype), torch.ones(3, device=DEV)
    dx, dw = torch.full_like(x, 7.0), torch.zeros(dim, device=DEV)
    nv.check(nv.lib(x).fbam_rmsnorm_bwd(nv.ptr(x), nv.ptr(x), nv.ptr(w), nv.ptr(rstd), nv.ptr(dx), nv.ptr(dw),
                                        C.c_longlong(3), dim, nv.stream_ptr()), "fbam_rmsnorm_bwd")
    assert int(torch.count_nonzero(dx)) == 0 and bool((dw == 3).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 64), (64, 264), (65, 256), (511, 1024), (600, 248), (5000, 520)])
def test_gelu_backward_with_column_sums(rows, cols, dtype):
    from fbamtrain_b200.ops import native_ops as no
    g = torch.Generator(device=DEV).manual_seed(rows * 3 + cols)
    z, dy = (torch.randn(rows, cols, device=DEV, generator=g).to(dtype) for _ in range(2))
    dz, sums = no._gelu_bwd_colsum(z, dy)
    exp = dy.double() * ref.gelu_grad(z.double())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert _rel(dz, exp) < eps
    assert torch.equal(dz, no._gelu_bwd(z, dy))
    # fp32 sums of the rounded values: at most rows roundings of a partial sum
    bound = rows * 2.0 ** -24 * dz.double().abs().sum(0) + 1e-6
    assert bool(((sums.double() - dz.double().sum(0)).abs() <= bound).all())
    assert bool(((no._colsum(dz).double() - dz.double().sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 72), (513, 64), (2047, 136), (2048, 128), (2049, 128), (2049, 2368), (300, 2376),
                                       (200, 4744), (70, 9480), (8192, 200), (8193, 200), (20000, 8), (1024, 1024), (1025, 1024),
                                       (1025, 1032), (2048, 1032), (4096, 1024), (4097, 1024), (4097, 1032), (8192, 1032)])
def test_column_sums_of_both_kinds_of_launch(rows, cols, dtype):
    """One launch of clusters of 8, 4, 2 or 1 CTAs up to a number of rows, slabs and an adding launch above; written as fp32
    and as elements."""
    from fbamtrain_b200.ops import native_ops as no
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    z, dy = (torch.randn(rows, cols, device=DEV, generator=g).to(dtype) for _ in range(2))
    dz, sums = no._gelu_bwd_colsum(z, dy)
    assert torch.equal(dz, no._gelu_bwd(z, dy))
    # fp32 sums of the rounded values: at most rows roundings of a partial sum
    for got, of in ((sums, dz), (no._colsum(dy), dy)):
        bound = rows * 2.0 ** -24 * of.double().abs().sum(0) + 1e-6
        assert bool(((got.double() - of.double().sum(0)).abs() <= bound).all())
    assert torch.equal(no._colsum(dy, dtype), no._colsum(dy).to(dtype))
    assert torch.equal(no._gelu_bwd_colsum(z, dy, dtype)[1], sums.to(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,dim", [(1, 8), (5, 64), (70, 72), (333, 128), (17, 256), (300, 264), (40, 512), (9, 1024), (700, 1032),
                                      (5, 2048), (150, 2056), (3, 4096), (5000, 256)])
def test_rmsnorm_backward_with_a_residual_gradient(rows, dim, dtype):
    from fbamtrain_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows + dim)
    x, dy, dres = (torch.randn(rows, dim, device=DEV, generator=g).to(dtype) for _ in range(3))
    x.requires_grad_(True)
    w = (1 + 0.1 * torch.randn(dim, device=DEV, generator=g)).to(dtype).requires_grad_(True)
    y, same = ops.rms_norm_residual(x, w, 1e-5)
    assert torch.equal(same, x) and torch.equal(y, ops.rms_norm(x, w, 1e-5))
    dx, dw = torch.autograd.grad((y, same), (x, w), (dy, dres))
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    exp = torch.autograd.grad((ref.rms_norm(xd, wd, 1e-5), xd * 1.0), (xd, wd), (dy.double(), dres.double()))
    # one rounding to the 16-bit type; fp32 sums behind it
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert _rel(dx, exp[0]) < eps and _rel(dw, exp[1]) < 1.5 * eps
    # the gradients alone give the same as the two together, up to the rounding of the sum
    plain, dw_plain = torch.autograd.grad(ops.rms_norm(x, w, 1e-5), (x, w), dy)
    assert torch.equal(dw, dw_plain)
    assert float((dx.float() - (plain.float() + dres.float())).norm() / exp[0].norm()) < 2 * eps
    # an upstream gradient whose rows start two bytes off a 16-byte boundary
    odd = torch.empty(rows * dim + 1, device=DEV, dtype=dtype)[1:].view(rows, dim).copy_(dres)
    y, same = ops.rms_norm_residual(x, w, 1e-5)
    assert torch.equal(torch.autograd.grad((y, same), x, (dy, odd))[0], dx)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,pix,c", [(1, 1, 8), (3, 7, 64), (5, 480, 512), (2, 33, 528), (1, 1000, 2048), (2, 5, 2056),
                                     (66000, 2, 8), (70001, 1, 8), (5, 127, 64), (5, 128, 64), (5, 129, 64), (3001, 3, 72),
                                     (9, 31, 64), (9, 32, 64), (700, 33, 64), (5000, 27, 72), (5000, 28, 72),
                                     (7, 3, 2048), (7, 4, 2048), (2500, 3, 2056), (40000, 24, 64)])
def test_mean_pool_backward_with_gelu(n, pix, c, dtype):
    import ctypes as C
    from fbamtrain_b200.ops import native as nv
    g = torch.Generator(device=DEV).manual_seed(n + pix + c)
    z = torch.randn(n, pix, c, device=DEV, generator=g).to(dtype)
    dy = torch.randn(n, c, device=DEV, generator=g).to(dtype)
    for with_z in (True, False):
        dx = torch.empty_like(z)
        nv.check(nv.lib(z).fbam_global_avgpool(nv.ptr(dy), nv.ptr(dx), C.c_longlong(n), pix, c, 1,
                                               nv.ptr(z if with_z else None), nv.stream_ptr()), "fbam_global_avgpool")
        exp = (dy.double() / pix).unsqueeze(1).expand(n, pix, c)
        if with_z:
            exp = exp * ref.gelu_grad(z.double())
        assert _rel(dx, exp) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,h,w,c", [(1, 2, 2, 8), (3, 6, 10, 24), (2, 48, 20, 256), (5, 4, 2, 1032)])
def test_gelu_with_2x2_mean_pool(n, h, w, c, dtype):
    from fbamtrain_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n + h + w + c)
    z = torch.randn(n, h, w, c, device=DEV, generator=g).to(dtype).requires_grad_(True)
    dy = torch.randn(n, h // 2, w // 2, c, device=DEV, generator=g).to(dtype)
    y = ops.gelu_avg_pool2x2_nhwc(z)
    (dz,) = torch.autograd.grad(y, z, dy.transpose(1, 2).contiguous().transpose(1, 2))      # a strided gradient
    zd = z.detach().double().requires_grad_(True)
    e = torch.nn.functional.gelu(zd).view(n, h // 2, 2, w // 2, 2, c).mean(dim=(2, 4))
    (edz,) = torch.autograd.grad(e, zd, dy.double())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert _rel(y, e) < eps and _rel(dz, edz) < eps
    with pytest.raises(ValueError):
        ops.gelu_avg_pool2x2_nhwc(z[:, :h - 1])
