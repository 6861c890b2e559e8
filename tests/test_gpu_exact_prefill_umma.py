"""The tcgen05 product of the exact Q8_0 prefill (csrc/exact_prefill_umma.cuh): the cache and the logits behind the chunk are the token-by-token path's bit for bit.  Every product of
the layer in tiles of 128 tokens x 96 or 128 weight rows (B200_XP_TILE): ragged and whole token tiles, row tiles that the rows do not fill, segments that are no multiple of a stage's
128 columns, more tiles than SMs, and block scales over the whole FP16 range (subnormal, negative, large), on both sides of it at once where results stay finite."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu
CODES = {96: "12896", 128: "128128"}


def run(pkg, shape, chunks, scales=None):
    S, Q8, n = pkg.synth, pkg.gguf.GGMLType.Q8_0, sum(chunks)
    tensors = S.build_tensors_fast(shape, Q8, seed=n)
    if scales is not None:
        for name, (kind, dims, raw) in tensors.items():
            if len(dims) == 2 and name.startswith("blk."):
                raw.reshape(-1, 34)[:, :2] = scales(np.random.default_rng(len(name)), raw.size // 34, name).astype(np.float16).view(np.uint8).reshape(-1, 2)
    model = pkg.loader.model_from_tensors(shape, Q8, tensors, n + 4)
    toks = np.random.default_rng(n).integers(0, shape.vocab, n + 1)
    check(pkg, model, toks, chunks, n)
    return model, toks


# (dim, hidden, heads, key/value heads, head size): rows of three and of seven segments of 27 and 23 blocks; 96 + 2 * 32 rows and rows of 64 and 96 columns
@pytest.mark.parametrize("geometry", [(2592, 5152, 8, 2, 128), (64, 96, 3, 1, 32)])
@pytest.mark.parametrize("rows", [96, 128])
def test_tiles(pkg, monkeypatch, geometry, rows):
    dim, hidden, heads, kv, hs = geometry
    monkeypatch.setenv("B200_XP_TILE", CODES[rows])
    run(pkg, pkg.synth.Shape("qwen3", dim, hidden, 2, heads, kv, hs, 128, False, 500000.0, 1e-5), [3, 128, 257])


@pytest.mark.parametrize("rows", [96, 128])
def test_several_tiles_per_sm(pkg, monkeypatch, rows):
    monkeypatch.setenv("B200_XP_TILE", CODES[rows])
    run(pkg, pkg.synth.SHAPES["mid-llama"], [129, 300])


@pytest.mark.parametrize("rows", [96, 128])
def test_scales(pkg, monkeypatch, rows):
    monkeypatch.setenv("B200_XP_TILE", CODES[rows])
    run(pkg, pkg.synth.SHAPES["tiny-llama"], [130], lambda rng, n, name: np.ldexp(rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n), rng.integers(-26, -2, n)))


@pytest.mark.parametrize("rows", [96, 128])
def test_large_scales(pkg, monkeypatch, rows):
    """Scales up to the largest FP16 numbers in queries, keys, gates and the attention's output, against values and up rows of the smallest, so that the hidden rows'
    scales and the logits stay finite."""
    exponents = {"attn_q": (6, 16), "attn_k": (6, 16), "attn_v": (-24, -14), "attn_output": (6, 16), "ffn_gate": (6, 16), "ffn_up": (-24, -14), "ffn_down": (-12, -4)}
    monkeypatch.setenv("B200_XP_TILE", CODES[rows])

    def scales(rng, n, name):
        lo, hi = exponents[name.split(".")[2]]
        return np.ldexp(rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 1.99, n), rng.integers(lo, hi, n))

    model, toks = run(pkg, pkg.synth.SHAPES["tiny-llama"], [130], scales)
    plan = pkg.B200MasterPlan(model, prefill_batch_size=130)
    plan.forward_batch_prefill(toks[:130], 0)
    assert np.isfinite(plan.forward_decode(int(toks[130]), 130)[0]).all()
    assert np.abs(plan.read_buffer("qkv", 64)).max() > 1e6
    plan.free()


def test_without_its_buffers(pkg, monkeypatch):
    """A driver that does not make its tensor maps: the chunk takes the other product, with none of its buffers."""
    used = []
    for refuse in ("umma", ""):
        monkeypatch.setenv("B200_TEST_REFUSE", refuse)
        run(pkg, pkg.synth.SHAPES["small-llama"], [300])
        S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
        plan = pkg.B200MasterPlan(pkg.loader.model_from_tensors(S.SHAPES["small-llama"], Q8, S.build_tensors_fast(S.SHAPES["small-llama"], Q8, seed=1), 304), prefill_batch_size=300)
        used.append(plan.device_bytes)
        plan.free()
    assert used[0] < used[1]


@pytest.mark.parametrize("side", [0, 1])
def test_swiglu_line(pkg, side):
    """On both sides of the line from which SwiGLU is a launch behind the gate/up product (csrc/plan.cu, XP_SPLIT_UNITS hidden units per SM): 12288 units are 90.3 tokens on 148 SMs."""
    run(pkg, pkg.synth.Shape("qwen3", 256, 12288, 1, 2, 1, 128, 128, False, 500000.0, 1e-5), [90 + side])
