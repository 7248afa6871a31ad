"""The recurrent weight as the persistent LSTM kernels take it (the kernels themselves are tested on the GPU)."""
import pytest
import torch

from fbamtrain_b200.ops.lstm import recurrent_weight


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_rows_at_four_bytes(dtype):
    h = 16
    w = torch.randn(4 * h, h).to(dtype)
    pitched = torch.zeros(4 * h, h + 3, dtype=dtype)
    pitched[:, :h] = w
    odd = torch.zeros(4 * h * h + 1, dtype=dtype)
    odd[1:] = w.flatten()
    for form in (w, w.float(), pitched[:, :h], odd[1:].view(4 * h, h), w.t().contiguous().t(), w.t().contiguous().t().float()):
        got = recurrent_weight(form, dtype)
        assert torch.equal(got, w) and got.is_contiguous() and got.data_ptr() % 4 == 0
    assert recurrent_weight(w, dtype).data_ptr() == w.data_ptr()          # nothing to do: no copy
    with pytest.raises(ValueError):
        recurrent_weight(w[:-1], dtype)


def test_rule_for_large_batches(monkeypatch):
    """Pure rule (no GPU): the sizes it was measured at, and those no rule is to touch."""
    from fbamtrain_b200.ops import lstm as L

    class Lib:
        fbam_lstm_persistent_max_hidden = staticmethod(lambda: 2048)

    monkeypatch.setattr(L.nv, "lib", lambda *a: Lib)
    for hidden in range(16, 2049, 16):
        for batch in (1, 8, 9, 32, 64, 128):
            for steps in (1, 2, 16, 256):
                for grad in (True, False):
                    assert L.persistent_ok(batch, hidden, steps, grad)
    assert not L.persistent_ok(1, 2064) and not L.persistent_ok(1, 24) and not L.persistent_ok(1, 0)
    # batch, hidden, steps, grad -> persistent was the faster one
    measured = [((512, 1024, 1, False), True), ((2048, 1024, 1, False), False), ((2048, 1024, 16, False), False),
                ((768, 1024, 64, False), True), ((256, 2048, 1, False), True), ((1024, 2048, 1, False), False),
                ((1024, 2048, 16, False), False), ((256, 2048, 64, False), True), ((1536, 256, 1, False), True),
                ((2048, 256, 1, False), False), ((1024, 64, 16, False), True), ((4096, 256, 16, False), False),
                ((1024, 512, 1, False), True), ((1536, 512, 1, False), False), ((1536, 512, 4, False), True),
                ((768, 1024, 1, True), True), ((2048, 1024, 1, True), False), ((1024, 1024, 16, True), True),
                ((768, 1024, 64, True), True), ((320, 2048, 1, True), True), ((1024, 2048, 1, True), False),
                ((1024, 2048, 16, True), False), ((320, 2048, 64, True), True), ((4096, 64, 1, True), False),
                ((1536, 256, 4, True), True), ((2048, 64, 16, False), True), ((4096, 64, 16, False), False)]
    for args, faster in measured:
        assert L.persistent_ok(*args) is faster, args


@pytest.mark.parametrize("steps", [1, 2, 8, 9, 10, 11, 17, 18, 256])
@pytest.mark.parametrize("down", [0, 1])
def test_lines_are_fetched_within_the_sequence(steps, down):
    """Both directions fetch the lines of the step eight behind the published one while there is one: the backward pass used
    to reach the step before the first (T = 10 and more)."""
    from fbamtrain_b200.ops import native as nv
    if not nv.available():
        pytest.skip("kernel library not built")
    ahead = nv.lib().fbam_lstm_step_ahead
    for published in range(steps):
        to = published - 8 if down else published + 8
        assert ahead(published, steps, down) == (to if 0 <= to < steps else -1)
