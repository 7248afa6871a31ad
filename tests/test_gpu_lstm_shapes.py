"""The persistent recurrence at the edges of its launch rules — batch rows that fill groups of eight partly, several
groups per block, several launches, hidden sizes on both sides of every block shape — and with a buffer that rules out
the wide loads, against the fp32 PyTorch definition."""
import math

import pytest
import torch

from fbamtrain_b200.ops import reference as ref
from fbamtrain_b200.utils.testing import assert_similar

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _problem(t_len, b, i_dim, h, dtype, per_sample=False):
    g = torch.Generator(device=DEV).manual_seed(t_len * 1000 + b * 10 + h)
    k = 1.0 / math.sqrt(h)

    def uniform(*shape):
        return ((torch.rand(shape, device=DEV, generator=g) * 2 - 1) * k).requires_grad_(True)

    x = torch.randn(t_len, b, i_dim, device=DEV, generator=g).to(dtype).requires_grad_(True)
    state = (b, h) if per_sample else (h,)
    h0, c0 = ((0.1 * torch.randn(state, device=DEV, generator=g)).requires_grad_(True) for _ in range(2))
    return (x, uniform(4 * h, i_dim), uniform(4 * h, h), uniform(4 * h), uniform(4 * h), h0, c0), g


def _rel(a, e):
    return float((a.float() - e).norm() / e.norm().clamp_min(1e-20))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("t_len,b,h", [
    (1, 1, 16), (2, 3, 48), (5, 9, 16), (6, 17, 256), (4, 32, 256), (5, 33, 240),      # 8 units, up to four groups
    (6, 8, 272), (5, 16, 272), (4, 25, 512), (7, 31, 496),                             # 16 units above one group
    (5, 8, 528), (6, 9, 528), (5, 24, 1024), (9, 32, 1024), (4, 41, 1008),             # two groups, one or two turns
    (4, 8, 1040), (5, 13, 1072), (4, 20, 2048), (6, 32, 2048),                         # one group, up to four turns
])
def test_batch_and_hidden_edges(t_len, b, h, dtype):
    from fbamtrain_b200.ops import lstm as L, native as nv
    params, g = _problem(t_len, b, 64, h, dtype)
    assert L.persistent_ok(b, h)
    y, h_n, c_n = L.lstm_sequence(*params, dtype)
    dy = torch.randn(y.shape, device=DEV, generator=g).to(dtype)
    got = torch.autograd.grad((y.float() * dy.float()).sum() + c_n.sum() + h_n.float().sum(), params)
    nv.check_status(y.device)
    fp = [p.detach().float().requires_grad_(True) for p in params]
    yf, hf, cf = ref.lstm_sequence(*fp, torch.float32)
    exp = torch.autograd.grad((yf * dy.float()).sum() + cf.sum() + hf.sum(), fp)
    assert_similar(yf.to(dtype), y, 3e-2)
    assert_similar(cf, c_n, 3e-2)
    # weights, h and the gate gradients are rounded to the 16-bit type once per step (bf16: 2^-9 relative each)
    for name, a, e in zip(["dx", "dw_ih", "dw_hh", "db_ih", "db_hh", "dh0", "dc0"], got, exp):
        assert _rel(a, e) < 4e-2, (name, _rel(a, e))


@pytest.mark.parametrize("t_len,b,h,persistent", [
    (3, 70, 1024, True), (2, 100, 2048, True), (3, 97, 64, True),       # three and four launches, ragged last ones
    (2, 384, 2048, True), (2, 480, 2048, False),                        # both sides of the line with gradients
    (1, 3744, 64, True), (1, 3800, 64, False),
])
def test_batches_of_several_launches(t_len, b, h, persistent):
    from fbamtrain_b200.ops import lstm as L
    assert L.persistent_ok(b, h, t_len) is persistent
    params, g = _problem(t_len, b, 64, h, torch.bfloat16)
    y, _, c_n = L.lstm_sequence(*params, torch.bfloat16)
    dy = torch.randn(y.shape, device=DEV, generator=g).bfloat16()
    got = torch.autograd.grad(y, params, dy)
    fp = [p.detach().float().requires_grad_(True) for p in params]
    yf, _, cf = ref.lstm_sequence(*fp, torch.float32)
    exp = torch.autograd.grad(yf, fp, dy.float())
    assert _rel(y, yf) < 1e-2 and _rel(c_n, cf) < 1e-2
    for name, a, e in zip(["dx", "dw_ih", "dw_hh", "db_ih", "db_hh", "dh0", "dc0"], got, exp):
        assert _rel(a, e) < 4e-2, (name, _rel(a, e))
    # a state per sample is accepted on both sides
    head = [p.detach() for p in params]
    full = [s.expand(b, h).contiguous() for s in head[5:]]
    ys, _, _ = L.lstm_sequence(*head[:5], *full, torch.bfloat16)
    assert _rel(ys, yf) < 1e-2


@pytest.mark.parametrize("b,h", [(3, 64), (12, 528)])
def test_carried_state_per_sample(b, h):
    from fbamtrain_b200.ops import lstm as L
    params, _ = _problem(8, b, 64, h, torch.bfloat16, per_sample=True)
    y, _, c_n = L.lstm_sequence(*params, torch.bfloat16)
    head = [p.detach() for p in params]
    y1, _, c1 = L.lstm_sequence(head[0][:5].contiguous(), *head[1:], torch.bfloat16)
    y2, _, c2 = L.lstm_sequence(head[0][5:].contiguous(), *head[1:5], y1[-1].float(), c1, torch.bfloat16)
    assert torch.equal(torch.cat([y1, y2]), y) and torch.equal(c2, c_n)


def test_output_rows_without_16_byte_alignment():
    """The C entry takes y and dGates at any element offset: two bytes off, the vectors are exchanged element by
    element, with the same bits as a result."""
    from fbamtrain_b200.ops import native as nv
    t_len, b, h = 7, 5, 80
    g = torch.Generator(device=DEV).manual_seed(3)
    pre = torch.randn(t_len, b, 4 * h, device=DEV, generator=g)
    whh = (torch.randn(4 * h, h, device=DEV, generator=g) / math.sqrt(h)).bfloat16()
    h0, c0 = torch.randn(2, h, device=DEV, generator=g).unbind(0)
    dy = torch.randn(t_len, b, h, device=DEV, generator=g).bfloat16()
    status = nv.status_word(pre.device)
    results = []
    for shift in (0, 1):
        gates = pre.clone()
        y = torch.zeros(t_len * b * h + 8, dtype=torch.bfloat16, device=DEV)[shift:shift + t_len * b * h]
        dg = torch.zeros(4 * t_len * b * h + 8, dtype=torch.bfloat16, device=DEV)[shift:shift + 4 * t_len * b * h]
        c_all = torch.empty(t_len, b, h, device=DEV)
        dh0, dc0 = torch.empty(2, b, h, device=DEV).unbind(0)
        assert nv.lib().fbam_lstm_fwd(nv.ptr(gates), nv.ptr(whh), nv.ptr(h0), nv.ptr(c0), nv.ptr(y), nv.ptr(c_all), None,
                                      None, nv.ptr(status), t_len, b, h, nv.stream_ptr()) == 0
        whh_t = whh.t().contiguous()
        assert nv.lib().fbam_lstm_bwd(nv.ptr(gates), nv.ptr(c_all), nv.ptr(c0), nv.ptr(dy), nv.ptr(whh_t), nv.ptr(dg),
                                      nv.ptr(dh0), nv.ptr(dc0), None, None, None, nv.ptr(status), t_len, b, h,
                                      nv.stream_ptr()) == 0
        nv.check_status(pre.device)
        results.append([t.clone() for t in (gates, y, c_all, dg, dh0, dc0)])
    for a, e in zip(results[1], results[0]):
        assert torch.equal(a, e)


def test_nan_travels_through_the_exchange():
    """A NaN hidden value is data, not an unwritten word: the recurrence goes on and the NaN reaches the outputs."""
    from fbamtrain_b200.ops import lstm as L, native as nv
    params, _ = _problem(6, 2, 64, 64, torch.bfloat16)
    params[0].data[2, 1] = float("nan")
    y, _, c_n = L.lstm_sequence(*params, torch.bfloat16)
    nv.check_status(y.device)
    assert torch.isfinite(y[:, 0].float()).all() and torch.isnan(y[2:, 1].float()).all() and torch.isnan(c_n[1]).all()


@pytest.mark.parametrize("b", [3, 9])
def test_operand_layouts_and_sizes(b):
    """Batches above 8 used to run a GEMM per step, which takes a recurrent weight of any row pitch and start and
    broadcasts one-element states and biases: dense copies give the same bits, and sizes that do not fit are refused."""
    from fbamtrain_b200.ops import lstm as L
    h, dtype = 64, torch.bfloat16
    params, g = _problem(4, b, 64, h, dtype)
    x, w_ih, w_hh, b_ih, b_hh, h0, c0 = [p.detach() for p in params]
    w_hh = w_hh.to(dtype)
    expected = L.lstm_sequence(x, w_ih, w_hh, b_ih, b_hh, h0, c0, dtype)[0]
    pitched = torch.zeros(4 * h, h + 8, dtype=dtype, device=DEV)
    pitched[:, :h] = w_hh
    odd = torch.zeros(4 * h * h + 1, dtype=dtype, device=DEV)
    odd[1:] = w_hh.flatten()
    for w in (pitched[:, :h], odd[1:].view(4 * h, h), w_hh.t().contiguous().t()):
        assert torch.equal(L.lstm_sequence(x, w_ih, w, b_ih, b_hh, h0, c0, dtype)[0], expected)
    one = torch.full((1,), 0.25, device=DEV)
    a = L.lstm_sequence(x, w_ih, w_hh, one, one, one, one, dtype)[0]
    full = [torch.full((n,), 0.25, device=DEV) for n in (4 * h, 4 * h, h, h)]
    assert torch.equal(a, L.lstm_sequence(x, w_ih, w_hh, *full, dtype)[0])
    for wrong in ((w_ih, w_hh[:-1], b_ih, b_hh, h0, c0), (w_ih, w_hh, b_ih[:-1], b_hh[:-1], h0, c0),
                  (w_ih, w_hh, b_ih, b_hh, h0[:-1], c0), (w_ih, w_hh, b_ih, b_hh, h0, c0[:-1])):
        with pytest.raises((ValueError, RuntimeError)):
            L.lstm_sequence(x, *wrong, dtype)


@pytest.mark.parametrize("t_len,b,h", [(9, 8, 1024), (10, 4, 1024), (17, 3, 560), (18, 9, 2048), (19, 24, 512), (33, 32, 1024)])
def test_steps_around_the_prefetch_distance_and_many_phases(t_len, b, h):
    """More steps than the distance at which lines are fetched ahead, and enough for every barrier of a backward cluster
    to go through several phases, with groups that share a block and rows that fill a group partly."""
    from fbamtrain_b200.ops import lstm as L, native as nv
    params, g = _problem(t_len, b, 64, h, torch.bfloat16)
    y, _, c_n = L.lstm_sequence(*params, torch.bfloat16)
    dy = torch.randn(y.shape, device=DEV, generator=g).bfloat16()
    got = torch.autograd.grad(y, params, dy)
    nv.check_status(y.device)
    fp = [p.detach().float().requires_grad_(True) for p in params]
    yf, _, cf = ref.lstm_sequence(*fp, torch.float32)
    exp = torch.autograd.grad(yf, fp, dy.float())
    # 16-bit weights, h and gate gradients: 2^-9 relative each, as above
    assert _rel(y, yf) < 1e-2 and _rel(c_n, cf) < 1e-2
    for name, a, e in zip(["dx", "dw_ih", "dw_hh", "db_ih", "db_hh", "dh0", "dc0"], got, exp):
        assert _rel(a, e) < 4e-2, (name, _rel(a, e))


def test_gate_functions_against_64_bits():
    """One step with a recurrent weight of zeros: the activated gates and the cell state are functions of the given
    pre-activations alone.  Bounds, relative: 2^x within 2^-22 of an argument that is off by 2^-24 of |x| log2(e), 1/x
    within 2^-23, and a rounding of 2^-24 for each of the operations around them."""
    from fbamtrain_b200.ops import native as nv
    b, h = 8, 512
    x = torch.cat([torch.linspace(-30, 30, 2 * b * h), torch.linspace(-0.7, 0.7, 2 * b * h)]).to(DEV)
    x[torch.arange(0, 40, 4)] = torch.tensor([0.0, -0.0, 1e-30, -1e-30, 100.0, -100.0, math.inf, -math.inf, math.nan, 1e-8],
                                             device=DEV)
    x = x[torch.randperm(x.numel(), device=DEV, generator=torch.Generator(device=DEV).manual_seed(0))]
    gates = x.view(1, b, 4 * h).clone()
    whh = torch.zeros(4 * h, h, device=DEV, dtype=torch.bfloat16)
    h0 = torch.zeros(h, device=DEV)
    c0 = torch.randn(h, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    y = torch.empty(1, b, h, dtype=torch.bfloat16, device=DEV)
    c_all = torch.empty(1, b, h, device=DEV)
    assert nv.lib().fbam_lstm_fwd(nv.ptr(gates), nv.ptr(whh), nv.ptr(h0), nv.ptr(c0), nv.ptr(y), nv.ptr(c_all), None, None,
                                  nv.ptr(nv.status_word(y.device)), 1, b, h, nv.stream_ptr()) == 0
    pre = x.view(b, 4, h).double()
    expected = torch.sigmoid(pre)
    expected[:, 2] = torch.tanh(pre[:, 2])
    got = gates.view(b, 4, h).double()
    assert torch.equal(got.isnan(), pre.isnan())
    ok = ~pre.isnan()
    bound = expected.abs() * (2.0 ** -22 + 2.0 ** -23 + 3 * 2.0 ** -24 + pre.abs().clamp_max(104.0) * 1.45 * 2.0 ** -24) + 1e-37
    # tanh is 2 s - 1 above 0.6: the error of s counts twice, relative to at least 0.53
    bound[:, 2] *= 2.0
    assert bool(((got - expected).abs() <= bound)[ok].all()), float(((got - expected).abs() / bound)[ok].max())
    c = got[:, 1] * c0.double() + got[:, 0] * got[:, 2]
    live = ~c.isnan()
    assert bool(((c_all[0].double() - c).abs() <= 2.0 ** -23 * (c0.abs() + 1.0))[live].all())


@pytest.mark.parametrize("span,sigmoid,tanh", [(8.0, (4.98e-7, 9.71e-8), (1.96e-7, 2.62e-8)),
                                                (1.0, (1.82e-7, 4.38e-8), (1.96e-7, 5.64e-8))])
def test_gate_functions_are_as_exact_as_their_plain_forms(span, sigmoid, tanh):
    """Relative errors against 64 bits over [-span, span], largest and root mean square.  The bounds are what
    1 / (1 + __expf(-x)) and tanhf leave there, measured over 4 million points; the largest of a sigmoid on [-1, 1], which
    hangs on single arguments of the hardware's 2^x, is that of the uncorrected reciprocal."""
    from fbamtrain_b200.ops import native as nv
    t_len, b, h = 64, 8, 512
    x = (torch.linspace(-span, span, t_len * b * h)).to(DEV).view(t_len, b, 1, h).expand(t_len, b, 4, h).contiguous()
    gates = x.clone().view(t_len, b, 4 * h)
    zeros = torch.zeros(4 * h, h, device=DEV, dtype=torch.bfloat16)
    y = torch.empty(t_len, b, h, dtype=torch.bfloat16, device=DEV)
    c_all = torch.empty(t_len, b, h, device=DEV)
    state = torch.zeros(h, device=DEV)
    assert nv.lib().fbam_lstm_fwd(nv.ptr(gates), nv.ptr(zeros), nv.ptr(state), nv.ptr(state), nv.ptr(y), nv.ptr(c_all), None,
                                  None, nv.ptr(nv.status_word(y.device)), t_len, b, h, nv.stream_ptr()) == 0
    nv.check_status(y.device)
    pre, got = x.double(), gates.view(t_len, b, 4, h).double()
    some = pre.abs() > 1e-6
    for k, of, bounds in ((0, torch.sigmoid, sigmoid), (1, torch.sigmoid, sigmoid), (2, torch.tanh, tanh), (3, torch.sigmoid, sigmoid)):
        off = (got[:, :, k] / of(pre[:, :, k]) - 1)[some[:, :, k]]
        assert float(off.abs().max()) <= bounds[0] and float(off.square().mean().sqrt()) <= bounds[1]
