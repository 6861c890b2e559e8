"""The attention of the exact Q8_0 prefill where its score rows live in global memory (csrc/exact_prefill.cuh, k_xp_attention): a CTA then walks several (token tile,
head) items over the same slot, q tile and staged tiles.  32 heads take the 32-token tile, 4 heads the 8-token one; the chunk in front of the first such one, in
shared memory, is the other side of each limit.  Everything is the token-by-token path's bit for bit; the second layer's cache holds what the attention of every token
of the chunk gave."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu

SMEM_FLOATS, SMS, SCRATCH_FLOATS = 220 * 1024 // 4, 148, (256 << 20) // 4


def stride(keys):
    return (keys + 31) // 32 * 32 + 4


def fits(head_size, tile, keys):  # the tile's score rows beside its queries, two staged tiles of 64 keys and the row maxima and sums
    return tile * (head_size + 4) + 2 * 64 * (head_size + 4) + tile * stride(keys) + 128 <= SMEM_FLOATS


def variant(heads, head_size, n, keys, context):
    """(tokens per tile, in global memory, items per CTA) of a chunk of n tokens whose last one sees `keys` keys."""
    if (n + 63) // 64 * heads >= SMS and fits(head_size, 64, keys):
        tile = 64
    else:
        tile = 32 if (n + 31) // 32 * heads >= SMS else 8
    items = (n + tile - 1) // tile * heads
    if fits(head_size, tile, keys):
        return tile, False, 1.0
    slot = 32 * stride(context)
    slots = max(min(slot * SMS, SCRATCH_FLOATS), slot) // (tile * stride(keys))
    return tile, True, items / min(items, slots)


# (heads, key/value heads, head size, chunks, context, tile in global memory)
@pytest.mark.parametrize("arch,heads,kv,hs,chunks,context,tile", [
    ("qwen3", 32, 8, 128, [512, 512, 512, 300], 2000, 32),
    ("qwen3", 32, 4, 64, [512, 512, 512, 161], 1700, 32),
    ("qwen3", 4, 2, 256, [512] * 5 + [140, 300], 3100, 8),
])
def test_score_rows_in_global_memory(pkg, arch, heads, kv, hs, chunks, context, tile):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    ends = np.cumsum(chunks)
    taken = [variant(heads, hs, n, int(end), context) for n, end in zip(chunks, ends)]
    assert taken[-1][:2] == (tile, True) and not taken[0][1]
    assert tile == 8 or max(v[2] for v in taken) > 1  # CTAs that walk several items
    shape = S.Shape(arch, 256, 256, 2, heads, kv, hs, 128, False, 500000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=heads + hs), context)
    toks = np.random.default_rng(hs).integers(0, 128, int(ends[-1]) + 1)
    check(pkg, model, toks, chunks, 512)
