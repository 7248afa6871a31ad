"""Attention inside a checkpoint: the backward may read its saved tensors only once, because every access runs the unpack
hooks (a non-reentrant checkpoint refuses a second one)."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint


def _attend(fused):
    from fbamtrain_b200.ops import mha
    if fused:
        return lambda x: mha.flash_attention_qkv(x, True)
    return lambda x: mha.flash_attention(x[:, :, 0], x[:, :, 1], x[:, :, 2], True)


@pytest.mark.parametrize("fused", [True, False])
def test_every_saved_tensor_is_unpacked_once(fused, monkeypatch):
    """On the CPU, with the launches replaced: what counts is how often the hooks run."""
    from fbamtrain_b200.ops import mha

    class Lib:
        fbam_attn_fwd = fbam_attn_fwd2 = fbam_attn_bwd = staticmethod(lambda *a: 0)

    monkeypatch.setattr(mha.nv, "lib", lambda *a: Lib)
    monkeypatch.setattr(mha.nv, "stream_ptr", lambda: None)
    monkeypatch.setattr(mha.nv, "status_word", lambda device: torch.zeros(1, dtype=torch.int32))
    unpacked = []

    def unpack(packed):
        unpacked.append(packed[0])
        return packed[1]

    packed = []

    def pack(t):
        packed.append((len(packed), t))
        return packed[-1]

    x = torch.randn(1, 5, 3, 2, 64).bfloat16().requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        y = _attend(fused)(x)
    torch.autograd.grad(y, x, torch.ones_like(y))
    assert sorted(unpacked) == list(range(len(packed))) and len(packed) == 5      # q, k, v, output, log-sum-exp
    y = checkpoint(_attend(fused), x, use_reentrant=False)
    torch.autograd.grad(y, x, torch.ones_like(y))


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_checkpointed_gradients_match(dtype, fused):
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(2, 130, 3, 2, 64, device="cuda", generator=g).to(dtype).requires_grad_(True)
    d_out = torch.randn(2, 130, 2, 64, device="cuda", generator=g).to(dtype)
    plain, kept = _attend(fused)(x), checkpoint(_attend(fused), x, use_reentrant=False)
    assert torch.equal(plain, kept)
    (a,), (b,) = torch.autograd.grad(plain, x, d_out), torch.autograd.grad(kept, x, d_out)
    # two key blocks: dQ is summed in fp32 by reductions in either order, which may move one 16-bit rounding
    assert float((a.float() - b.float()).norm() / a.float().norm()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)


@pytest.mark.gpu
def test_frame_head_with_attention_under_recompute():
    """The model key ``frame_head_recompute`` on a frame head with attention blocks: the same vectors and gradients as
    with the activations kept."""
    import copy
    from test_config import DEBUG_JSON
    from fbamtrain_b200 import RunConfiguration
    from fbamtrain_b200.data import SyntheticBatchSource
    from fbamtrain_b200.models import FbamModel
    d = copy.deepcopy(DEBUG_JSON)
    d["micro_batch_size"] = d["total_batch_size"] = 2
    d["train_sequence_length"] = d["validation_sequence_length"] = 16
    d["frame_rows"], d["frame_cols"], d["tokenizer_file_path"] = 8, 16, ""
    d["model_config"].update({"n_embed": 128, "n_layer": 1, "n_head": 2, "frame_rows": 8, "frame_cols": 16, "dtype": "bf16",
                              "use_fp16_accumulation": False, "action_vocab": 64, "frame_head_recompute": True})
    cfg = RunConfiguration.from_json(d)
    model = FbamModel(cfg.model_config, 64).cuda()
    cells = SyntheticBatchSource(8, 16, 256, 64, seed=0, pin=False).next_batch(2, 16)[0].cuda().view(32, 128, 3)
    params = list(model.frame_head.parameters())
    g = torch.Generator(device="cuda").manual_seed(1)
    results = []
    for recompute in (False, None):                       # None: as configured
        v = model.frame_head_chunk(cells, recompute)
        d_v = torch.randn(v.shape, device="cuda", generator=g.manual_seed(1)).to(v.dtype)
        results.append((v, torch.autograd.grad(v, params, d_v)))
    assert torch.equal(results[0][0], results[1][0])
    # fp32 sums by atomics in any order, rounded to bf16 on their way through a few layers
    for a, e in zip(results[1][1], results[0][1]):
        assert float((a.float() - e.float()).norm()) <= 2.0 ** -7 * float(e.float().norm())
