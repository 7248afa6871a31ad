"""LSTM over a whole sequence on the GPU.

Forward: one tensor-core GEMM computes the input projection of all time steps
(``X·W_ihᵀ + b_ih + b_hh``, fp32 out), then one persistent cooperative kernel runs the recurrence
with ``W_hh`` resident on chip (``csrc/lstm.cu``).  Backward: one persistent kernel does BPTT and
emits ``dGates`` for every step; the weight and input gradients are then three large GEMMs over all
``T·B`` rows (``dX = dGates·W_ih``, ``dW_ih = dGatesᵀ·X``, ``dW_hh = dGatesᵀ·H_prev``) and a column sum.
The reference performs the same mathematics one step at a time with a GEMM per step and recomputes
the gates in the backward pass (reference: ``tensorlib/src/streaming_lstm_fwd.cpp:430-465``,
``streaming_lstm_bwd.cpp:1218-1307``); here the activated gates are kept (in the buffer that held the
pre-activations), so nothing is recomputed.

Shapes beyond the persistent kernels' limits (hidden > 2048 or not a multiple of 16) and batches of many hundreds of
rows run step by step: a GEMM per step against ``W_hh`` followed by the same gate arithmetic.
"""
from __future__ import annotations


import torch

from ..utils import flops

from . import native as nv
from . import reference as ref
from .native_ops import gemm, gemm_nn, gemm_tn


def persistent_shape(hidden: int) -> bool:
    """Hidden sizes the persistent kernels take, at any batch."""
    return hidden > 0 and hidden % 16 == 0 and hidden <= nv.lib().fbam_lstm_persistent_max_hidden()


# us of one launch of the persistent kernels (32 rows): hidden up to, launch, each step; forward, forward + backward
_LAUNCH_US = ((64, 3.3, 0.95, 5.9, 2.1), (256, 3.0, 1.4, 6.0, 3.3), (512, 4.0, 1.6, 8.0, 3.6), (1024, 7.0, 3.0, 15.0, 6.9),
              (2048, 10.0, 12.4, 60.0, 23.0))


def persistent_ok(batch: int, hidden: int, steps: int = 1024, grad: bool = True) -> bool:
    """Where the persistent kernels are the faster path.  They cover 32 rows per launch and the launches follow one
    another, so their time grows with the batch; a GEMM per step costs about 140 us a step forward and 450 us with the
    backward (host and launches) until its product is large, and more the longer the sequence, since the gradient of the
    pre-activations is summed step by step: from 32 steps on it was not ahead at any batch.  Measured, us, persistent |
    GEMM per step:
      forward  H  256, batch 1536: 1 step 329 | 360, 64 steps 4702 | 8010      batch 2048: 1 step 351 | 254
      forward  H 1024, batch  512: 1 step 251 | 257, 64 steps 3263 | 8025      batch 2048: 1 step 757 | 285, 16 steps 3652 | 2793
      forward  H 2048, batch  256: 1 step 260 | 262, 64 steps 6511 | 8061      batch 1024: 1 step 818 | 300, 16 steps 6340 | 3007
      training H 1024, batch  768: 1 step 868 | 1152, 64 steps 10860 | 49738   batch 2048: 1 step 1742 | 996, 16 steps 8176 | 11191
    (Batch 32, 256 steps, H 1024, forward and backward: 1.9 ms against 107.9 ms.)"""
    if not persistent_shape(hidden):
        return False
    _, fwd_0, fwd, both_0, both = next(row for row in _LAUNCH_US if hidden <= row[0])
    launches = (batch + 31) // 32
    if not grad:
        return launches * (fwd_0 + fwd * steps) <= 140.0 * steps + 90.0
    return steps >= 32 or launches * (both_0 + both * steps) <= 450.0 * steps + 500.0


def recurrent_weight(w_hh: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """``w_hh (4H, H)`` as the persistent kernels read it: dense rows, loaded 4 bytes at a time (a GEMM per step took any
    row pitch and copied what started at an odd element)."""
    if w_hh.shape[0] != 4 * w_hh.shape[1]:
        raise ValueError(f"recurrent weight of shape {tuple(w_hh.shape)} is not (4H, H)")
    w = w_hh.to(dtype).contiguous()
    return w if w.data_ptr() % 4 == 0 else w.clone()


def _fit(t: torch.Tensor, shape) -> torch.Tensor:
    """``t`` dense in ``shape`` (broadcast, or refused); most calls are host-bound, so nothing is called without need."""
    return (t if t.shape == shape else t.expand(shape)).contiguous()


class _LstmSequence(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w_ih, w_hh, b_ih, b_hh, h0, c0):
        t_len, b, i_dim = x.shape
        h = w_hh.shape[1]
        dev = x.device
        x2 = x.reshape(t_len * b, i_dim).contiguous()
        wi, wh = w_ih.to(x.dtype), recurrent_weight(w_hh, x.dtype)
        bias = _fit(b_ih.float() + b_hh.float(), (4 * h,))
        gates = gemm(x2, wi, bias=bias, out_dtype=torch.float32).view(t_len, b, 4 * h)
        y = torch.empty(t_len, b, h, dtype=x.dtype, device=dev)
        c_all = torch.empty(t_len, b, h, dtype=torch.float32, device=dev)
        per_sample = int(h0.dim() == 2)
        shape = (b, h) if per_sample else (h,)
        h0f, c0f = _fit(h0.float(), shape), _fit(c0.float(), shape)
        nv.check(nv.lib(wh).fbam_lstm_fwd_ex(nv.ptr(gates), nv.ptr(wh), nv.ptr(h0f), nv.ptr(c0f), nv.ptr(y),
                                           nv.ptr(c_all), None, None,
                                           nv.ptr(nv.status_word(dev)), t_len, b, h, per_sample, nv.stream_ptr()),
                 "fbam_lstm_fwd")
        flops.add(2.0 * t_len * b * h * 4 * h)          # the recurrent product; the input projection is a counted GEMM
        ctx.save_for_backward(x2, wi, wh, gates, y, c_all, h0f, c0f)
        ctx.dims = (t_len, b, i_dim, h)
        ctx.per_sample = per_sample
        return y, y[-1].clone(), c_all[-1].clone()

    @staticmethod
    def backward(ctx, dy, dh_last, dc_last):
        x2, wi, wh, gates, y, c_all, h0f, c0f = ctx.saved_tensors
        t_len, b, i_dim, h = ctx.dims
        dev = dy.device
        dy = dy.contiguous()
        wh_t = wh.t().contiguous()
        dgates = torch.empty(t_len, b, 4 * h, dtype=wh.dtype, device=dev)
        dh0 = torch.empty(b, h, dtype=torch.float32, device=dev)
        dc0 = torch.empty(b, h, dtype=torch.float32, device=dev)
        dhl = None if dh_last is None else dh_last.float().contiguous()
        dcl = None if dc_last is None else dc_last.float().contiguous()
        nv.check(nv.lib(wh).fbam_lstm_bwd_ex(nv.ptr(gates), nv.ptr(c_all), nv.ptr(c0f), nv.ptr(dy), nv.ptr(wh_t),
                                           nv.ptr(dgates), nv.ptr(dh0), nv.ptr(dc0), nv.ptr(dhl), nv.ptr(dcl),
                                           None, nv.ptr(nv.status_word(dev)), t_len, b, h, ctx.per_sample,
                                           nv.stream_ptr()), "fbam_lstm_bwd")
        flops.add(2.0 * t_len * b * h * 4 * h)
        dg2 = dgates.view(t_len * b, 4 * h)
        dx = gemm_nn(dg2, wi).view(t_len, b, i_dim) if ctx.needs_input_grad[0] else None
        dw_ih = gemm_tn(dg2, x2, out_dtype=torch.float32)
        h_first = h0f.to(y.dtype).view(1, b, h) if ctx.per_sample else h0f.to(y.dtype).expand(1, b, h)
        h_prev = torch.cat([h_first, y[:-1]], 0).reshape(t_len * b, h)
        dw_hh = gemm_tn(dg2, h_prev, out_dtype=torch.float32)
        from .native_ops import _colsum
        db = _colsum(dg2)
        if ctx.per_sample:
            return dx, dw_ih, dw_hh, db, db.clone(), dh0, dc0
        return dx, dw_ih, dw_hh, db, db.clone(), dh0.sum(0), dc0.sum(0)


def _stepwise(x, w_ih, w_hh, b_ih, b_hh, h0, c0):
    """For shapes the persistent kernels do not cover, or not as fast: tensor-core GEMM per step, autograd."""
    from .native_ops import linear
    t_len, b, _ = x.shape
    hdim = w_hh.shape[1]
    wi, wh = w_ih.to(x.dtype), w_hh.to(x.dtype)
    bias = b_ih.float() + b_hh.float()
    xg = linear(x.reshape(t_len * b, -1), wi).float().view(t_len, b, 4 * hdim)
    h = h0.to(x.dtype).unsqueeze(0).expand(b, hdim).contiguous()
    c = c0.float().unsqueeze(0).expand(b, hdim)
    ys = []
    for t in range(t_len):
        hf, c = ref.lstm_cell(xg[t] + linear(h, wh).float() + bias, c)
        h = hf.to(x.dtype)
        ys.append(h)
    return torch.stack(ys, 0), h, c


def lstm_sequence(x, w_ih, w_hh, b_ih, b_hh, h0, c0, compute_dtype):
    if compute_dtype not in nv.ELEM_DTYPES:
        raise TypeError("native LSTM computes in bf16 or fp16")
    x = x.to(compute_dtype)
    t_len, b, _ = x.shape
    hidden = w_hh.shape[1]
    persistent = persistent_shape(hidden)
    if persistent and b > 32 and h0.dim() == 1:      # a state per sample is something only the persistent kernels take
        grad = torch.is_grad_enabled() and any(t.requires_grad for t in (x, w_ih, w_hh, b_ih, b_hh, h0, c0))
        persistent = persistent_ok(b, hidden, t_len, grad)
    if not persistent or x.shape[2] % 8 != 0:
        return _stepwise(x, w_ih, w_hh, b_ih, b_hh, h0, c0)
    return _LstmSequence.apply(x, w_ih, w_hh, b_ih, b_hh, h0, c0)
