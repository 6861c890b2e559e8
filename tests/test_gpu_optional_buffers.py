"""Buffers that only make a plan faster do not decide whether it can be made: a batch size whose chunk buffers have no room on the device leaves the
token-by-token prefill, with nothing of them kept, and a batch size beyond the context costs no more than the context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_room_for_the_chunk(pkg):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    shape = S.Shape("llama", 8192, 64, 1, 256, 1, 32, 64, False, 500000.0, 1e-5)  # 32 KB of residual stream and 33 KB of projections per chunk row
    rows = 3_200_000                                                               # 105 GB and 106 GB: the first fits, the second does not
    tensors = S.build_tensors_fast(shape, Q8, seed=4, device="cuda")
    toks = np.arange(1, 8, dtype=np.int32)
    seen = []
    for context, batch in ((rows, rows), (rows, 1), (64, 8)):
        plan = pkg.B200MasterPlan(pkg.loader.model_from_tensors(shape, Q8, dict(tensors), context), prefill_batch_size=batch)
        plan.forward_batch_prefill(toks[:-1], 0)
        assert plan.exact_prefill_info()[:2] == ((8, 1) if context == 64 else (0, 0))
        seen.append((plan.device_bytes, plan.forward_decode(int(toks[-1]), len(toks) - 1)[0].view(np.uint32)))
        plan.free()
    assert seen[0][0] == seen[1][0]  # nothing kept
    for _, logits in seen[1:]:
        assert np.array_equal(logits, seen[0][1])


def test_batch_beyond_the_context(pkg, make_model):
    model = make_model("tiny-llama", pkg.gguf.GGMLType.Q8_0, ctx=64)
    used = []
    for batch in (64, 100_000):
        plan = pkg.B200MasterPlan(model, prefill_batch_size=batch)
        plan.forward_batch_prefill(list(range(64)), 0)
        used.append(plan.device_bytes)
        plan.free()
    assert used[0] == used[1]


def test_refused_tensor_maps(pkg, make_model, monkeypatch):
    """A driver that does not make the tensor maps of the chunk's products: token by token, with nothing kept and the reason said."""
    model = make_model("tiny-llama", pkg.gguf.GGMLType.Q8_0, ctx=64)
    toks = list(range(3, 40))
    seen = []
    for refuse, batch, info in (("", 1, (0, 0)), ("tensor_maps", 64, (0, 0)), ("", 64, (64, 1))):
        monkeypatch.setenv("B200_TEST_REFUSE", refuse)
        plan = pkg.B200MasterPlan(model, prefill_batch_size=batch)
        plan.forward_batch_prefill(toks[:-1], 0)
        assert plan.exact_prefill_info()[:2] == info and ("tensor maps" in plan.exact_prefill_info()[2]) == bool(refuse)
        seen.append((plan.device_bytes, plan.forward_decode(toks[-1], len(toks) - 1)[0].tobytes()))
        plan.free()
    assert seen[0] == seen[1] and seen[0][0] < seen[2][0] and seen[0][1] == seen[2][1]
