"""The allocation-free LSTM forward entry point, and buffers that held other values before.

Some users of the library cannot allocate device memory where they run the recurrence (a host with a fixed memory plan, a
frozen allocator, a fully committed budget), so ``fbam_lstm_fwd_noalloc`` takes the buffers of its results and nothing
else: the hidden vectors are exchanged through ``y`` itself, where a word that is not 0xFFFFFFFF counts as written.  Such
callers hand in the same buffers again and again, so what counts is that finite values of an earlier call are never taken
for new ones.  The tests fill the buffers with such values first and compare with the PyTorch definition; the backward
exchanges ``dGates`` in the same way.
"""
import ctypes as C
import math

import pytest
import torch

from fbamtrain_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _inputs(t_len, b, h, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = 1.0 / math.sqrt(h)
    gates = torch.randn(t_len, b, 4 * h, device="cuda", generator=g)
    whh = ((torch.rand(4 * h, h, device="cuda", generator=g) * 2 - 1) * k).to(BF)
    h0 = 0.1 * torch.randn(h, device="cuda", generator=g)
    c0 = 0.1 * torch.randn(h, device="cuda", generator=g)
    return gates, whh, h0, c0


def _definition(gates, whh, h0, c0):
    """fp32 recurrence over given pre-activations, h rounded to bf16 between steps as the kernels exchange it."""
    b, h = gates.shape[1], whh.shape[1]
    ht, ct, ys, cs = h0.to(BF).float().expand(b, h), c0.expand(b, h), [], []
    for pre in gates:
        hf, ct = ref.lstm_cell(pre + ht @ whh.float().t(), ct)
        ht = hf.to(BF).float()
        ys.append(ht)
        cs.append(ct)
    return torch.stack(ys), torch.stack(cs)


def _run_regular(nv, gates, whh, h0, c0, t_len, b, h, y, c_all):
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    code = nv.lib().fbam_lstm_fwd(nv.ptr(gates), nv.ptr(whh), nv.ptr(h0), nv.ptr(c0), nv.ptr(y), nv.ptr(c_all),
                                  None, None, nv.ptr(status), t_len, b, h, nv.stream_ptr())
    assert code == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0


def _run_noalloc(nv, gates, whh, h0, c0, t_len, b, h, y, c_all):
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib = nv.lib()
    lib.fbam_lstm_fwd_noalloc.restype = C.c_int
    code = lib.fbam_lstm_fwd_noalloc(nv.ptr(gates), nv.ptr(whh), nv.ptr(h0), nv.ptr(c0), nv.ptr(y), nv.ptr(c_all),
                                     nv.ptr(status), t_len, b, h, nv.stream_ptr())
    assert code == 0, code
    torch.cuda.synchronize()
    assert int(status.item()) == 0


def _previous_values(kind, *shape):
    """What a buffer may hold before a call: the finite values of another problem, or zeros."""
    g = torch.Generator(device="cuda").manual_seed(99)
    return torch.zeros(shape, dtype=BF, device="cuda") if kind == "zeros" else \
        torch.tanh(torch.randn(shape, device="cuda", generator=g)).to(BF)


def _close(got, want):
    # one bf16 rounding per value (2^-9 of its norm) plus the different order of the fp32 sums
    assert float((got.float() - want).norm() / want.norm()) < 2.0 ** -7


@pytest.mark.parametrize("kind", ["values", "zeros"])
@pytest.mark.parametrize("t_len,b,h", [(24, 8, 512), (17, 3, 1024), (9, 5, 80)])
def test_noalloc_entry_point_ignores_what_the_output_held(t_len, b, h, kind):
    from fbamtrain_b200.ops import native as nv
    gates, whh, h0, c0 = _inputs(t_len, b, h, h)
    want_y, want_c = _definition(gates, whh, h0, c0)
    results = []
    for run in (_run_noalloc, _run_regular):
        pre, y = gates.clone(), _previous_values(kind, t_len, b, h)
        c_all = torch.empty(t_len, b, h, dtype=torch.float32, device="cuda")
        run(nv, pre, whh, h0, c0, t_len, b, h, y, c_all)
        _close(y, want_y)
        _close(c_all, want_c)
        results.append((y, c_all, pre))
    for a, e in zip(*results):                      # both entry points launch the same kernel
        assert torch.equal(a, e)


def test_noalloc_entry_point_matches_regular_entry_point_twice():
    """Two problems back to back through either entry point, into fresh buffers: the same bits."""
    from fbamtrain_b200.ops import native as nv
    for seed, (t_len, b, h) in enumerate([(24, 8, 512), (17, 3, 1024)]):
        gates, whh, h0, c0 = _inputs(t_len, b, h, seed)
        results = []
        for run in (_run_regular, _run_noalloc):
            pre, y = gates.clone(), torch.empty(t_len, b, h, dtype=BF, device="cuda")
            c_all = torch.empty(t_len, b, h, dtype=torch.float32, device="cuda")
            run(nv, pre, whh, h0, c0, t_len, b, h, y, c_all)
            results.append((y, c_all, pre))
        for name, a, e in zip(("y", "c_all", "gates"), *results):
            assert torch.equal(a, e), name


def test_noalloc_entry_point_on_one_set_of_buffers():
    """Three problems through the same buffers: the second and third find the outputs of the one before."""
    from fbamtrain_b200.ops import native as nv
    t_len, b, h = 12, 4, 256
    y = torch.empty(t_len, b, h, dtype=BF, device="cuda")
    c_all = torch.empty(t_len, b, h, dtype=torch.float32, device="cuda")
    for seed in range(3):
        gates, whh, h0, c0 = _inputs(t_len, b, h, seed)
        want_y, want_c = _definition(gates, whh, h0, c0)
        _run_noalloc(nv, gates, whh, h0, c0, t_len, b, h, y, c_all)
        _close(y, want_y)
        _close(c_all, want_c)


@pytest.mark.parametrize("kind", ["values", "zeros"])
@pytest.mark.parametrize("t_len,b,h", [(17, 3, 1024), (9, 5, 80), (6, 11, 528)])
def test_backward_ignores_what_the_gate_gradients_held(t_len, b, h, kind):
    """The same hazard in the backward: ``dGates`` is exchanged word by word."""
    from fbamtrain_b200.ops import native as nv
    gates, whh, h0, c0 = _inputs(t_len, b, h, h + 1)
    y = torch.empty(t_len, b, h, dtype=BF, device="cuda")
    c_all = torch.empty(t_len, b, h, dtype=torch.float32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(4)
    dy = torch.randn(t_len, b, h, device="cuda", generator=g).to(BF)
    leaves = [gates.clone().requires_grad_(True), h0.expand(b, h).clone().requires_grad_(True),
              c0.expand(b, h).clone().requires_grad_(True)]
    ht, ct, ys = leaves[1], leaves[2], []
    for pre in leaves[0]:
        ht, ct = ref.lstm_cell(pre + ht @ whh.float().t(), ct)
        ys.append(ht)
    want = torch.autograd.grad(torch.stack(ys), leaves, dy.float())
    _run_regular(nv, gates, whh, h0, c0, t_len, b, h, y, c_all)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    dgates = _previous_values(kind, t_len, b, 4 * h)
    dh0, dc0 = torch.empty(2, b, h, device="cuda").unbind(0)
    whh_t = whh.t().contiguous()
    code = nv.lib().fbam_lstm_bwd(nv.ptr(gates), nv.ptr(c_all), nv.ptr(c0), nv.ptr(dy), nv.ptr(whh_t), nv.ptr(dgates),
                                  nv.ptr(dh0), nv.ptr(dc0), None, None, None, nv.ptr(status), t_len, b, h, nv.stream_ptr())
    assert code == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for a, e in zip((dgates, dh0, dc0), want):      # h and dGates are rounded to bf16 once per step
        assert float((a.float() - e).norm() / e.norm()) < 2e-2


def test_noalloc_entry_point_allocates_no_device_memory():
    """Free device memory (as the driver reports it) and this process's allocator statistics are the same before and
    after a call whose inputs and outputs already exist: the entry point takes nothing from the device heap."""
    from fbamtrain_b200.ops import native as nv
    t_len, b, h = 12, 4, 256
    gates, whh, h0, c0 = _inputs(t_len, b, h, 7)
    y = torch.empty(t_len, b, h, dtype=BF, device="cuda")
    c_all = torch.empty(t_len, b, h, dtype=torch.float32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib = nv.lib()
    lib.fbam_lstm_fwd_noalloc.restype = C.c_int
    args = (nv.ptr(gates), nv.ptr(whh), nv.ptr(h0), nv.ptr(c0), nv.ptr(y), nv.ptr(c_all), nv.ptr(status), t_len, b, h,
            nv.stream_ptr())
    assert lib.fbam_lstm_fwd_noalloc(*args) == 0          # first call on the device: module load
    torch.cuda.synchronize()
    free_before, _ = torch.cuda.mem_get_info()
    reserved_before = torch.cuda.memory_reserved()
    assert lib.fbam_lstm_fwd_noalloc(*args) == 0
    torch.cuda.synchronize()
    free_after, _ = torch.cuda.mem_get_info()
    assert free_after == free_before
    assert torch.cuda.memory_reserved() == reserved_before
    assert int(status.item()) == 0


def test_noalloc_entry_point_rejects_oversize_with_clear_error():
    from fbamtrain_b200.ops import native as nv
    lib = nv.lib()
    lib.fbam_lstm_fwd_noalloc.restype = C.c_int
    lib.fbam_lstm_fwd_noalloc_max_hidden.restype = C.c_int
    lib.fbam_lstm_fwd_noalloc_strerror.restype = C.c_char_p
    limit = lib.fbam_lstm_fwd_noalloc_max_hidden()
    assert limit == 1024
    code = lib.fbam_lstm_fwd_noalloc(None, None, None, None, None, None, None, 4, 2, limit + 16, None)
    assert code == 401
    assert b"exceeds" in lib.fbam_lstm_fwd_noalloc_strerror(code)
