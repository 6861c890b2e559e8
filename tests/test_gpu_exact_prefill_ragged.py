"""The 64-token tile of the exact Q8_0 prefill's attention (csrc/exact_prefill.cuh, k_xp_attention) with a last tile of few tokens behind a cache whose length is no
multiple of the 64 keys of a staged tile: the tokens that the tile does not have read no scores.  Bit for bit the token-by-token path's."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu


# (heads, key/value heads, head size, tokens in front, tokens): 1 to 29 tokens in the last tile, which end within the first half of a staged tile, in the second
# half and behind it
@pytest.mark.parametrize("heads,kv,hs,start,n", [(32, 8, 128, 3, 285), (32, 8, 128, 3, 257), (32, 4, 64, 31, 257), (32, 4, 64, 7, 280), (64, 8, 64, 13, 140), (32, 8, 96, 20, 268),
                                                 (32, 8, 128, 40, 270), (32, 8, 128, 60, 261), (64, 4, 32, 67, 157)])
def test_ragged_last_tile(pkg, heads, kv, hs, start, n):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    assert (n + 63) // 64 * heads >= 148  # the 64-token tile
    shape = S.Shape("qwen3", 256, 256, 2, heads, kv, hs, 128, False, 500000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=start), start + n + 2)
    toks = np.random.default_rng(n).integers(0, 128, start + n + 1)
    check(pkg, model, toks, [start, n], 512)
