"""The tensor-core attention of a layered prefill chunk (csrc/layered.cuh, k_window_attention_mma) at the edges of its launches, against the float64 oracle: chunks whose
key tiles two CTAs share (few heads, more than 128 keys) with an even, an odd and a ragged number of tiles, windows inside a tile and beyond several, and enough
heads for tiles of 128 rows.  BF16 operands: relative RMS error of a logits row <= 2e-2, the bound of the layered prefill tests (measured there: 2e-3 .. 6e-3)."""
import numpy as np
import pytest

from pibidra_util import oracle, rel_rms, w64

pytestmark = pytest.mark.gpu


def layers(S):
    L = S.pibidra_layer
    return {
        "narrow": [L(2, 1, 64, 64, 70, 256, bias_max=100.0), L(2, 2, 128, 128, 33, 128, bias_max=40.0)],
        "wide": [L(2, 1, 192, 128, 300, 128, bias_max=90.0), L(3, 1, 128, 128, 200, 256, bias_max=200.0, softcap=4.0)],
        "many_heads": [L(152, 4, 64, 64, 150, 128, bias_max=100.0)],
    }


@pytest.mark.parametrize("name,chunks", [("narrow", [129, 65]), ("narrow", [192, 1, 130]), ("wide", [128, 129]), ("wide", [320]), ("wide", [257, 63]), ("many_heads", [127]),
                                         ("many_heads", [129, 70])])
def test_chunks(pkg, name, chunks):
    S, O = pkg.synth, oracle()
    cfg = S.pibidra_config(256, 256, layers(S)[name])
    w = S.pibidra_weights(cfg, 31, bias_rows=10)
    toks = np.random.default_rng(sum(chunks)).integers(0, cfg["vocab"], sum(chunks)).tolist()
    ref = O.forward(cfg, w64(w), toks)
    plan = pkg.B200MasterPlan.initialize_plan(S.pibidra_model(cfg, w, sum(chunks) + 8), prefill_batch_size=max(chunks), compute="bfloat16")
    try:
        at = 0
        for n in chunks:
            got, _ = plan.forward_batch_logits(toks[at:at + n], at, list(range(n)))
            worst = max(rel_rms(got[i], ref[at + i]) for i in range(n))
            assert worst <= 2e-2, f"rows {at}..{at + n - 1}: {worst:.3g}"
            at += n
    finally:
        plan.free()
