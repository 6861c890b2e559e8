"""Chunks of more tokens than a launch has blocks in y (65535), and than the gate/up rows are kept for at a time (8192; csrc/plan.cu, XP_SLICE): one chunk of the exact Q8_0 prefill and the
same tokens in two leave the same cache and logits, bit for bit, and a plan's buffers grow by the tokens' quants alone beyond a slice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WIDTH, HIDDEN = 64, 96


def make(pkg, n):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    shape = S.Shape("qwen3", WIDTH, HIDDEN, 1, 1, 1, 32, 128, False, 500000.0, 1e-5)
    return pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=3), n + 2)


def compare(pkg, n, halves):
    model = make(pkg, n)
    toks = np.random.default_rng(3).integers(0, 128, n + 1).astype(np.int32)
    out = []
    for chunks in ([n], halves):
        plan = pkg.B200MasterPlan(model, prefill_batch_size=n)
        at = 0
        for k in chunks:
            plan.forward_batch_prefill(toks[at:at + k], at)
            at += k
        assert plan.exact_prefill_info()[1] == len(chunks)
        cache = [plan.read_buffer(b, n * 32, layer=0).view(np.uint32).copy() for b in ("key_cache", "value_cache")]
        hidden = [plan.read_buffer(b, k, d).copy() for b, k, d in (("hb", HIDDEN, np.float32), ("hq", HIDDEN, np.int8), ("hs", HIDDEN // 32, np.float32))]
        out.append(cache + hidden + [plan.read_buffer("x", WIDTH).copy(), plan.forward_decode(int(toks[n]), n)[0].copy()])
        plan.free()
    for a, b in zip(*out):
        assert a.tobytes() == b.tobytes()


def test_more_than_65535_tokens(pkg):
    compare(pkg, 65600, [32800, 32800])


@pytest.mark.parametrize("n", [8193, 8320, 16500])  # a token, a tile of 128 and more than a slice behind the first one
@pytest.mark.parametrize("kernel", ["128128", "64", "16"])
def test_slices(pkg, monkeypatch, n, kernel):
    monkeypatch.setenv("B200_XP_TILE", kernel)
    compare(pkg, n, [4000, n - 4000] if n < 12000 else [8000, 8000, n - 16000])


def test_room(pkg, monkeypatch):
    n, held = 65600, []
    for refuse in ("umma", ""):
        monkeypatch.setenv("B200_TEST_REFUSE", refuse)
        plan = pkg.B200MasterPlan(make(pkg, n), prefill_batch_size=n)
        held.append(plan.device_bytes)
        plan.free()
    assert 0 < held[1] - held[0] <= 2 * n * (WIDTH + HIDDEN) + 8 * 8192 * HIDDEN + 4096
