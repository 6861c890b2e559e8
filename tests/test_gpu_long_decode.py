"""Decode attention of heads that a cluster of CTAs shares (csrc/decode_kernels.cuh, attention_split): logits bit-equal to the CPU oracle at the
edges of the split (128 keys), of the key blocks (32), of the value stages (128 positions) and of the pieces of the sequential sum (1024 and 4096)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AT = [126, 127, 128, 129, 159, 160, 161, 255, 256, 257, 300, 511, 513, 1022, 1023, 1024, 1055, 2047, 2050, 4094, 4095, 4096, 4130]


def run(pkg, orc, model, at, batch):
    c = model.configuration
    toks = np.random.default_rng(c.head_size).integers(0, c.vocab_size, max(at) + 1)
    plan = pkg.B200MasterPlan(model, prefill_batch_size=batch)
    om = orc.OracleModel(model, lanes=16)
    done = 0
    for p in at:
        for q in range(done, p):
            om.forward(int(toks[q]), q, want_logits=False)
        if batch > 1:
            for q in range(done, p, batch):
                plan.forward_batch_prefill(toks[q:min(q + batch, p)], q)
        else:
            for q in range(done, p):
                plan.forward_prefill(int(toks[q]), q)
        got, best = plan.forward_decode(int(toks[p]), p)
        ref = om.forward(int(toks[p]), p)
        assert np.array_equal(got.view(np.uint32), np.asarray(ref, dtype=np.float32).view(np.uint32)), f"position {p}"
        assert best == orc.argmax(ref)
        done = p + 1
    plan.free()


@pytest.mark.parametrize("shape", ["tiny-llama", "tiny-qwen3", "tiny-phi3"])  # head sizes 64, 128, 96
def test_q8(pkg, orc, make_model, shape):
    run(pkg, orc, make_model(shape, pkg.gguf.GGMLType.Q8_0, ctx=max(AT) + 2), AT, 512)


@pytest.mark.parametrize("shape", ["tiny-llama", "tiny-qwen3"])
def test_f16_token_by_token(pkg, orc, make_model, shape):
    run(pkg, orc, make_model(shape, pkg.gguf.GGMLType.F16, ctx=320), [p for p in AT if p <= 300], 1)


def test_head_size_256(pkg, orc, tmp_path):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    shape = S.Shape("llama", 512, 512, 1, 2, 1, 256, 512, False, 500000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=3), 300)
    run(pkg, orc, model, [127, 128, 131, 290], 64)


def test_trace_runs_the_step_s_kernels(pkg, make_model):
    """The traced copy of the step shows the attention that the step runs: shared by a cluster from 128 positions on, where a head's 900 keys take one CTA several
    times as long."""
    plan = pkg.B200MasterPlan(make_model("tiny-qwen3", pkg.gguf.GGMLType.Q8_0, ctx=1000), prefill_batch_size=512)
    toks = np.random.default_rng(1).integers(0, 640, 900).astype(np.int32)
    for p in range(0, 900, 300):
        plan.forward_batch_prefill(toks[p:p + 300], p)

    def attention_us(at):
        best = 1e9
        for _ in range(5):
            rec = plan._native.trace_decode(7, at).astype(np.int64)
            best = min(best, min((x - w) / 1e3 for k, _, w, x in rec if k == 4))
        return best

    deep, single = attention_us(900), attention_us(127)
    traced = plan.read_buffer("logits", 640).view(np.uint32)
    assert np.array_equal(traced, plan.forward_decode(7, 127)[0].view(np.uint32))
    plan.free()
    assert deep < 3 * single, (deep, single)  # a CTA per head: about 5 times the 128-key step's
