"""The norm that the streaming matvecs compute themselves (csrc/fused_norm.cuh, csrc/seqsum3.cuh): the sequential sum on adversarial terms, and logits
bit-equal to the oracle at the edges of the four widths of a thread's share (1024, 2048, 4096, 8192 entries)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def literal(t):
    return np.add.accumulate(np.concatenate(([np.float32(0)], t)), dtype=np.float32)[-1]  # strictly in order


def cases():
    rng = np.random.default_rng(11)
    f = np.float32
    for n in (1, 31, 32, 33, 256, 1000, 1024, 1025, 1056, 2048, 2049, 2560, 4095, 4096, 4097, 8191, 8192):
        x = rng.standard_normal(n).astype(f)
        yield x * x
        yield ((rng.integers(-127, 128, n) * f(np.float16(0.013))) ** 2).astype(f)  # a dequantised row: few significant bits
        yield np.full(n, 0.25, f)                                                    # every add exact, every binade boundary hit
        yield np.where(rng.random(n) < 0.5, 0, x * x).astype(f)
        yield (x * x * np.exp(rng.standard_normal(n) * 4)).astype(f)
        y = np.full(n, 2.0 ** -24, f)
        y[0] = 1.0                                                                   # every later add is a tie
        yield y
    yield np.zeros(4096, f)
    yield np.full(300, 1e-42, f)                                                     # subnormal terms
    yield np.concatenate((np.full(100, 1e30, f), np.full(100, 1e-30, f), np.full(3000, 3e37, f)))  # runs into infinity


def test_sum(pkg):
    with np.errstate(over="ignore"):
        for t in cases():
            got = np.float32(pkg.native.test_seqsum(t, threads=3))
            want = literal(t)
            assert got.view(np.uint32) == np.float32(want).view(np.uint32), (len(t), t[:4], got, want)


@pytest.mark.parametrize("dim", [32, 992, 1024, 1056, 2048, 2080, 4096, 4128, 8192])
def test_q8_widths(pkg, orc, dim):
    check(pkg, orc, dim, pkg.gguf.GGMLType.Q8_0)


@pytest.mark.parametrize("dim", [256, 1024, 1280, 2048, 2304, 4096, 4352, 8192])
def test_f16_widths(pkg, orc, dim):  # inside the matvecs up to 4096, a launch of its own beyond
    check(pkg, orc, dim, pkg.gguf.GGMLType.F16)


def check(pkg, orc, dim, quant):
    S = pkg.synth
    shape = S.Shape("qwen3", dim, 512, 2, 4, 2, 64, 512, True, 1000000.0, 1e-6)
    model = pkg.loader.model_from_tensors(shape, quant, S.build_tensors_fast(shape, quant, seed=dim), 8)
    plan, om = pkg.B200MasterPlan(model), orc.OracleModel(model, lanes=16)
    for pos, tok in enumerate((3, 77, 410)):
        got, _ = plan.forward_decode(tok, pos)
        assert np.array_equal(got.view(np.uint32), np.asarray(om.forward(tok, pos), dtype=np.float32).view(np.uint32)), pos
    plan.free()


# a shallow ring (B200_SMV_BUDGET_KB) is as deep as without the norm: its squares come on top of the budget.  Rows of 4128 to 8192 entries had no stage left at 48 KB.
@pytest.mark.parametrize("dim,kb", [(2080, 40), (4288, 40), (4288, 48), (8192, 48), (8192, 64)])
def test_q8_small_budget(pkg, monkeypatch, dim, kb):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    shape = S.Shape("qwen3", dim, 512, 1, 4, 2, 64, 512, True, 1000000.0, 1e-6)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=dim), 8)

    def logits():
        plan = pkg.B200MasterPlan(model)
        try:
            return [plan.forward_decode(tok, pos)[0].view(np.uint32) for pos, tok in enumerate((3, 77))]
        finally:
            plan.free()

    want = logits()
    monkeypatch.setenv("B200_SMV_BUDGET_KB", str(kb))
    for a, b in zip(want, logits()):
        assert np.array_equal(a, b)


def test_q8_budget_without_a_stage_is_refused(pkg, monkeypatch, make_model):
    monkeypatch.setenv("B200_SMV_BUDGET_KB", "1")
    with pytest.raises(Exception, match="leaves no stage"):
        pkg.B200MasterPlan(make_model("tiny-llama", pkg.gguf.GGMLType.Q8_0, ctx=8))
