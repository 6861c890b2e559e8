"""The line between the tensor-core attention of a layered BF16 prefill chunk, whose operands are BF16, and the general kernel with FP32 keys and values
(csrc/layered_plan.cuh, ly_mma_fits): windows (which no context cuts short) up to the limit take the one, wider windows the other, which B200_LAYERED_ATT=simt chooses for every layer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMEM = 227 * 1024  # of a CTA


def widest(dk, dv):  # distances of four bytes beside 128 queries and two stages of 64 keys and values
    return (SMEM - ((128 + 128) * (dk + 8) + 128 * (dv + 8)) * 2) // 4


@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64), (192, 128)])
@pytest.mark.parametrize("beyond", [0, 1, 4000])
def test_wide_windows(pkg, monkeypatch, dk, dv, beyond):
    S, n = pkg.synth, 70
    window = widest(dk, dv) + beyond
    cfg = S.pibidra_config(128, 128, [S.pibidra_layer(2, 1, dk, dv, window, 128)])
    weights = S.pibidra_weights(cfg, 9, bias_rows=8)
    toks = np.random.default_rng(dk).integers(0, 128, n).tolist()
    out = []
    for att in ("", "simt"):
        monkeypatch.setenv("B200_LAYERED_ATT", att)
        plan = pkg.B200MasterPlan.initialize_plan(S.pibidra_model(cfg, weights, window), prefill_batch_size=n, compute="bfloat16")
        out.append(plan.forward_batch_logits(toks, 0, list(range(n)))[0].view(np.uint32))
        plan.free()
    assert np.array_equal(out[0], out[1]) == (beyond > 0)
