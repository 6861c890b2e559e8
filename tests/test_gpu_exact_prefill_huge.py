"""A chunk of more tokens than a launch has blocks in y (65535): one chunk of the exact Q8_0 prefill and the same tokens in two leave the same cache and logits, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_than_65535_tokens(pkg):
    S, Q8, n = pkg.synth, pkg.gguf.GGMLType.Q8_0, 65600
    shape = S.Shape("qwen3", 64, 96, 1, 1, 1, 32, 128, False, 500000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=3), n + 2)
    toks = np.random.default_rng(3).integers(0, shape.vocab, n + 1).astype(np.int32)
    out = []
    for chunks in ([n], [32800, 32800]):
        plan = pkg.B200MasterPlan(model, prefill_batch_size=n)
        at = 0
        for k in chunks:
            plan.forward_batch_prefill(toks[at:at + k], at)
            at += k
        assert plan.exact_prefill_info()[1] == len(chunks)
        cache = [plan.read_buffer(b, n * 32, layer=0).view(np.uint32).copy() for b in ("key_cache", "value_cache")]
        out.append(cache + [plan.forward_decode(int(toks[n]), n)[0].view(np.uint32).copy()])
        plan.free()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
