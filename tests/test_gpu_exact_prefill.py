"""Batched exact prefill of Q8_0 plans (csrc/exact_prefill.cuh): the KV cache, and the logits of the decode step behind the chunk, are the
token-by-token path's bit for bit.  Sizes sit at the edges of the token tiles (8 / 16 / 32 / 64), of the attention tiles (8 and 32 tokens,
128 keys) and of the weight tiles (rows that are no multiple of 64, segments that are no multiple of 128 columns)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kv(plan, c, n):
    return [plan.read_buffer(name, c.context_length * c.kv_dim, layer=l)[: n * c.kv_dim].view(np.uint32) for l in range(c.n_layers) for name in ("key_cache", "value_cache")]


def token_by_token(pkg, model, toks):
    plan = pkg.B200MasterPlan(model, prefill_batch_size=1)
    for p, t in enumerate(toks[:-1]):
        plan.forward_prefill(int(t), p)
    cache = kv(plan, model.configuration, len(toks) - 1)
    x = plan.read_buffer("x", model.configuration.dim).view(np.uint32)
    logits = plan.forward_decode(int(toks[-1]), len(toks) - 1)[0].view(np.uint32)
    plan.free()
    return cache, x, logits


def check(pkg, model, toks, chunks, batch, why=""):
    """Chunks of more than one token are multiplied at once; with `why` (a word of the reason) they go token by token, as in the plan that they are compared with."""
    cache, x, logits = token_by_token(pkg, model, toks)
    plan = pkg.B200MasterPlan(model, prefill_batch_size=batch)
    at = 0
    for n in chunks:
        plan.forward_batch_prefill(toks[at:at + n], at)
        at += n
    assert at == len(toks) - 1
    rows, multiplied, reason = plan.exact_prefill_info()
    assert (rows, multiplied) == ((0, 0) if why else (min(batch, model.configuration.context_length), sum(n > 1 for n in chunks))) and (why in reason if why else not reason)
    for got, want in zip(kv(plan, model.configuration, at), cache):
        assert np.array_equal(got, want)
    assert np.array_equal(plan.read_buffer("x", model.configuration.dim).view(np.uint32), x)
    assert np.array_equal(plan.forward_decode(int(toks[-1]), at)[0].view(np.uint32), logits)
    plan.free()


@pytest.mark.parametrize("shape,chunks,batch", [
    ("tiny-llama", [2], 2), ("tiny-llama", [7, 8, 9], 16), ("tiny-llama", [15, 17], 32), ("tiny-llama", [31, 33], 64), ("tiny-llama", [63, 65, 2], 128),
    ("tiny-qwen3", [1, 40, 3], 64), ("tiny-qwen3", [127, 2, 128], 128), ("tiny-phi3", [16, 48], 64), ("tiny-phi3-gqa", [64, 1, 36], 64), ("small-llama", [37, 129], 256),
])
def test_chunks(pkg, make_model, shape, chunks, batch):
    model = make_model(shape, pkg.gguf.GGMLType.Q8_0, ctx=sum(chunks) + 3)
    toks = np.random.default_rng(len(chunks) + batch).integers(0, model.configuration.vocab_size, sum(chunks) + 1)
    check(pkg, model, toks, chunks, batch)


# the layer geometries of the models that use this path (segments of 2432, 1536, 2048 columns; the widest token tiles)
@pytest.mark.parametrize("shape,n", [("mid-qwen3-4b", 37), ("mid-phi3-mini", 100), ("mid-llama", 130), ("mid-llama", 300)])
def test_geometries(pkg, shape, n):
    S = pkg.synth
    Q8 = pkg.gguf.GGMLType.Q8_0
    model = pkg.loader.model_from_tensors(S.SHAPES[shape], Q8, S.build_tensors_fast(S.SHAPES[shape], Q8, seed=5), n + 4)
    toks = np.random.default_rng(n).integers(0, S.SHAPES[shape].vocab, n + 1)
    check(pkg, model, toks, [n], n)


# chunks behind a long cache; four heads take the 8-token attention tile, whose score rows of 2093 keys still fit shared memory (test_gpu_exact_prefill_long.py has
# those in global memory)
@pytest.mark.parametrize("shape", ["tiny-llama", "tiny-qwen3"])
def test_long_context(pkg, make_model, shape):
    chunks = [512] * 4 + [40, 5]
    model = make_model(shape, pkg.gguf.GGMLType.Q8_0, ctx=6000)
    toks = np.random.default_rng(9).integers(0, model.configuration.vocab_size, sum(chunks) + 1)
    check(pkg, model, toks, chunks, 512)
