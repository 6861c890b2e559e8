"""Kernels of prefill chunks that fill the SMs for long (recurrence scans, the GEMMs of the FP32 mode and of shapes without tensor-core tiles, the tensor-core
attention) are not launched programmatically: their CTAs would become resident during the kernel in front and be spread unevenly.  A chunk with programmatic launches takes
no longer than one without (B200_PDL=0); with the SSD scan among them three layers took 1.46 times as long, with the FP32 GEMM two layers 1.2 times.  Device times, the
smallest of ten."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(pkg, monkeypatch, model, vocab, compute):
    toks = np.random.default_rng(3).integers(0, vocab, 512).tolist()

    def run():
        plan = pkg.B200MasterPlan.initialize_plan(model, prefill_batch_size=512, compute=compute)
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


@pytest.mark.parametrize("mixer", ["mamba2", "rglru"])
def test_scans(pkg, monkeypatch, mixer):
    S = pkg.synth
    layer = S.dinuzen_mamba2(64, 64, 128, 1, 4) if mixer == "mamba2" else S.dinuzen_rglru(1024, 8, 4)
    cfg = S.dinuzen_config(1024, 256, [layer] * 3)
    check(pkg, monkeypatch, S.dinuzen_model(cfg, S.dinuzen_weights(cfg, 3), 520), 256, "bfloat16")


@pytest.mark.parametrize("width,compute", [(1024, "float32"), (1000, "bfloat16"), (1024, "bfloat16")])
def test_gemms(pkg, monkeypatch, width, compute):
    S = pkg.synth
    cfg = S.pibidra_config(width, 1024, [S.pibidra_layer(16, 4, 64, 64, 512, 4096 if width == 1024 else 3000)] * 2)
    check(pkg, monkeypatch, S.pibidra_model(cfg, S.pibidra_weights(cfg, 1, bias_rows=32), 520), 1024, compute)
