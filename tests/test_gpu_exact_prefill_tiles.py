"""The token tiles (8, 16, 32, 64) that the product of the exact Q8_0 prefill (csrc/exact_prefill.cuh) chooses from the chunk's length and the matrix, each with a ragged
last tile: the cache and the logits behind the chunk are the token-by-token path's bit for bit."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,chunks", [("mid-llama-1b", [2, 9]), ("mid-llama-1b", [61]), ("mid-qwen3-4b", [29, 17]), ("mid-qwen3-4b", [203]), ("small-llama", [95]), ("mid-llama", [5, 449])])
def test_tiles(pkg, shape, chunks):
    S, Q8, n = pkg.synth, pkg.gguf.GGMLType.Q8_0, sum(chunks)
    model = pkg.loader.model_from_tensors(S.SHAPES[shape], Q8, S.build_tensors_fast(S.SHAPES[shape], Q8, seed=n), n + 4)
    check(pkg, model, np.random.default_rng(n).integers(0, S.SHAPES[shape].vocab, n + 1), chunks, n)
