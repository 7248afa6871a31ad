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
