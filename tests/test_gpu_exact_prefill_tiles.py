"""The token tiles (8, 16, 32, 64) of the exact Q8_0 prefill's product (csrc/exact_prefill.cuh): the cache and the logits behind the chunk are the token-by-token path's bit for
bit.  Once with the tile that the launch chooses from the chunk's length and the matrix, and once with each tile in every product of the layer (B200_XP_TILE), whatever the
choice would be: whole and ragged last tiles, chunks shorter than the tile, row tiles of 64 that the rows do not fill, and rows of fewer columns than a stage."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu


def run(pkg, shape, chunks):
    S, Q8, n = pkg.synth, pkg.gguf.GGMLType.Q8_0, sum(chunks)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=n), n + 4)
    check(pkg, model, np.random.default_rng(n).integers(0, shape.vocab, n + 1), chunks, n)


@pytest.mark.parametrize("shape,chunks", [("mid-llama-1b", [2, 9]), ("mid-llama-1b", [61]), ("mid-qwen3-4b", [29, 17]), ("mid-qwen3-4b", [203]), ("small-llama", [95]), ("mid-llama", [5, 449]),
                                          ("mid-llama", [189]), ("mid-qwen3-4b", [301])])
def test_tiles(pkg, monkeypatch, shape, chunks):
    monkeypatch.delenv("B200_XP_TILE", raising=False)
    run(pkg, pkg.synth.SHAPES[shape], chunks)


# (dim, hidden, heads, key/value heads, head size): rows of three and of seven segments of 27 and 23 blocks; 96 + 2 * 32 rows and rows of 64 and 96 columns, less than the 128 of a stage
@pytest.mark.parametrize("geometry", [(2592, 5152, 8, 2, 128), (64, 96, 3, 1, 32)])
@pytest.mark.parametrize("tile", [8, 16, 32, 64])
def test_forced_tiles(pkg, monkeypatch, geometry, tile):
    dim, hidden, heads, kv, hs = geometry
    monkeypatch.setenv("B200_XP_TILE", str(tile))
    run(pkg, pkg.synth.Shape("qwen3", dim, hidden, 2, heads, kv, hs, 128, False, 500000.0, 1e-5), [3, tile, 2 * tile + tile // 2 + 1])
