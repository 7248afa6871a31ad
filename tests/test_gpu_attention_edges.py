"""The attention kernels at the edges of their tiles (one query block to several, ragged last blocks, a single token),
on fused and on separate inputs, with an output gradient that is a strided view, against the fp32 definition."""
import pytest
import torch

from fbamtrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("t,d", [(1, 64), (47, 128), (127, 64), (128, 128), (130, 64), (257, 128), (385, 64), (640, 128),
                                 (1100, 64)])
def test_forward_and_gradients(t, d, causal, fused, dtype):
    from fbamtrain_b200.ops import mha, native as nv
    b, h = 2, 3
    g = torch.Generator(device=DEV).manual_seed(t * 7 + d)
    qkv = torch.randn(b, t, 3, h, d, device=DEV, generator=g).to(dtype)
    d_out = torch.randn(b, h, t, d, device=DEV, generator=g).to(dtype).transpose(1, 2)      # heads outside, rows inside
    f = qkv.float().requires_grad_(True)
    of = ref.attention(f[:, :, 0], f[:, :, 1], f[:, :, 2], causal)
    (ef,) = torch.autograd.grad(of, f, d_out.float())
    if fused:
        qkv.requires_grad_(True)
        o = mha.flash_attention_qkv(qkv, causal)
        (got,) = torch.autograd.grad(o, qkv, d_out)
    else:
        q, k, v = (qkv[:, :, i].contiguous().requires_grad_(True) for i in range(3))
        o = mha.flash_attention(q, k, v, causal)
        got = torch.stack(torch.autograd.grad(o, (q, k, v), d_out), 2)
    nv.check_status(qkv.device)
    # P and dS are rounded to the 16-bit type before they are multiplied (bf16: 2^-9 relative each)
    eps = 1e-2 if dtype == torch.bfloat16 else 2e-3
    assert float((o.float() - of).norm() / of.norm()) < eps
    for i, name in enumerate(("dq", "dk", "dv")):
        err = (got[:, :, i].float() - ef[:, :, i]).norm()
        # a single token has dq = dk = 0 up to rounding: measured against all three gradients
        assert float(err / ef.norm()) < eps and float(err) <= 3 * eps * float(ef[:, :, i].norm()) + 1e-3 * float(ef.norm()), name


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("t", [1, 24, 127, 128, 130, 300])
def test_gradient_scratch_is_as_large_as_the_gradient(t, d):
    """The fp32 sums of dQ take B·T·H·D values: what lies behind them stays as it was (rounded up to whole tiles they
    were 128 times as much at one token)."""
    import ctypes as C
    from fbamtrain_b200.ops import native as nv
    b, h = 2, 3
    g = torch.Generator(device=DEV).manual_seed(t + d)
    q, k, v, d_out = (torch.randn(b, t, h, d, device=DEV, generator=g).bfloat16() for _ in range(4))
    out, dq, dk, dv = (torch.empty_like(q) for _ in range(4))
    lse, delta = (torch.empty(b, h, t, device=DEV) for _ in range(2))
    room = b * h * d * ((t + 127) // 128 * 128 + 128)
    dq32 = torch.full((room,), 7.0, device=DEV)
    strides = [C.c_longlong(n) for n in q.stride()[:3]]
    status, scale = nv.status_word(q.device), d ** -0.5
    nv.check(nv.lib(q).fbam_attn_fwd2(nv.ptr(q), nv.ptr(k), nv.ptr(v), *strides, nv.ptr(out), nv.ptr(lse), b, t, h, d, 0,
                                      C.c_float(scale), nv.ptr(status), nv.stream_ptr()), "fbam_attn_fwd2")
    nv.check(nv.lib(q).fbam_attn_bwd(nv.ptr(q), nv.ptr(k), nv.ptr(v), *strides, nv.ptr(out), nv.ptr(d_out), *strides,
                                     nv.ptr(lse), nv.ptr(delta), nv.ptr(dq32), nv.ptr(dq), nv.ptr(dk), nv.ptr(dv), *strides,
                                     b, t, h, d, 0, C.c_float(scale), nv.ptr(status), nv.stream_ptr()), "fbam_attn_bwd")
    nv.check_status(q.device)
    assert bool((dq32[b * t * h * d:] == 7.0).all())
    f = [x.float().requires_grad_(True) for x in (q, k, v)]
    exp = torch.autograd.grad(ref.attention(*f, False), f, d_out.float())
    whole = float(torch.stack([e.norm() for e in exp]).norm())
    for a, e in zip((dq, dk, dv), exp):       # P and dS in bf16: 2^-9 relative each; dq = dk = 0 at one token
        assert float((a.float() - e).norm()) <= 3e-2 * float(e.norm()) + 1e-3 * whole
