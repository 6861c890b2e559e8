"""Plans that the system has no pinned memory for beyond what they need (B200_TEST_REFUSE=pinned: the allocations fail as cudaMallocHost does): they are made all the same and
their steps and rows are the other plans' bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gguf(pkg, make_model):
    plan = pkg.B200MasterPlan(make_model("tiny-llama", pkg.gguf.GGMLType.Q8_0, ctx=32), prefill_batch_size=8)
    plan.forward_batch_prefill([3, 1, 4, 1, 5], 0)
    out = [plan.forward_decode(t, 5 + i) for i, t in enumerate((9, 2, 6))]
    plan.free()
    return [(row.tobytes(), token) for row, token in out]


def layered(pkg, make_model):
    S, n = pkg.synth, 300
    cfg = S.pibidra_config(64, 96, [S.pibidra_layer(4, 2, 16, 16, 6, 96)])
    toks = np.random.default_rng(2).integers(0, 96, n).tolist()
    plan = pkg.B200MasterPlan.initialize_plan(S.pibidra_model(cfg, S.pibidra_weights(cfg, 4), n + 8), prefill_batch_size=n, compute="float32")
    out = [plan.forward_batch_logits(toks, 0, rows)[0].tobytes() for rows in ([n - 1, 0, 7], list(range(n)), [])]
    row, token = plan.forward_decode(5, n)
    plan.free()
    return out + [row.tobytes(), token]


@pytest.mark.parametrize("make", [gguf, layered])
def test_no_pinned_memory(pkg, make_model, monkeypatch, make):
    monkeypatch.delenv("B200_TEST_REFUSE", raising=False)
    want = make(pkg, make_model)
    monkeypatch.setenv("B200_TEST_REFUSE", "pinned")
    assert make(pkg, make_model) == want
