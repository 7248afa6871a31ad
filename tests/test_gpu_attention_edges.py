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
