"""The 32-token tile of the exact Q8_0 prefill's attention in sixteen warps of two tokens (csrc/exact_prefill.cuh, k_xp_attention<HS, 2, 512>: heads of 128 and 256 entries whose score rows leave
no room for 64 tokens): whole and ragged last tiles, key tiles of 64 that end inside, two passes over the elements of a head of 256."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv,hs,chunks", [(32, 8, 128, [520]), (32, 8, 128, [479, 163]), (16, 2, 256, [320]), (16, 4, 256, [301, 290])])
def test_heads(pkg, heads, kv, hs, chunks):
    S, Q8, n = pkg.synth, pkg.gguf.GGMLType.Q8_0, sum(chunks)
    shape = S.Shape("qwen3", 256, 256, 1, heads, kv, hs, 512, False, 500000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=n), n + 4)
    check(pkg, model, np.random.default_rng(n).integers(0, 512, n + 1), chunks, max(chunks))
