"""Recurrence scans of prefill chunks that have up to a CTA per SM for the whole chunk are not launched programmatically: their CTAs would become resident during the
kernel in front and be spread unevenly.  A chunk with programmatic launches takes no longer than one without (B200_PDL=0); with the SSD scan among them three layers took
1.46 times as long.  Device times, the smallest of ten."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixer", ["mamba2", "rglru"])
def test_chunk_is_not_slower(pkg, monkeypatch, mixer):
    S = pkg.synth
    layer = S.dinuzen_mamba2(64, 64, 128, 1, 4) if mixer == "mamba2" else S.dinuzen_rglru(1024, 8, 4)
    cfg = S.dinuzen_config(1024, 256, [layer] * 3)
    w = S.dinuzen_weights(cfg, 3)
    toks = np.random.default_rng(3).integers(0, 256, 512).tolist()

    def run():
        plan = pkg.B200MasterPlan.initialize_plan(S.dinuzen_model(cfg, w, 520), prefill_batch_size=512, compute="bfloat16")
        try:
            ms = []
            for _ in range(13):
                plan.forward_batch_prefill(toks, 0)
                ms.append(plan.prefill_info()[2])
            return min(ms[3:])
        finally:
            plan.free()

    fast = run()
    monkeypatch.setenv("B200_PDL", "0")
    plain = run()
    assert fast <= 1.05 * plain, (fast, plain)
