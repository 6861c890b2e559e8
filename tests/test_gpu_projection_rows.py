"""The projection rows that stay in registers (csrc/layered.cuh, k_qk_prep_reg) against the kernel that walks the row three times (B200_LAYERED_PREP=general): the
same threads add the same squares in the same order, so caches and logits are equal bit for bit, in a chunk and in a decode step.  Sizes: rows that fill whole
rounds of 256 and of 1024 entries and rows that do not, entries that are no multiple of four, the most rounds that the registers hold and one more."""
import numpy as np
import pytest

from test_gpu_pibidra import make_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv,dk,dv,compute", [(2, 1, 16, 24, "float32"), (3, 1, 10, 7, "float32"), (4, 2, 64, 64, "bfloat16"), (12, 3, 100, 50, "float32"), (16, 4, 64, 64, "bfloat16"),
                                                    (16, 8, 128, 128, "float32"), (32, 8, 128, 128, "bfloat16"), (40, 8, 128, 128, "float32"), (48, 8, 128, 128, "float32"),
                                                    (48, 8, 128, 132, "float32")])
def test_bits(pkg, monkeypatch, heads, kv, dk, dv, compute):
    S = pkg.synth
    cfg = S.pibidra_config(128, 96, [S.pibidra_layer(heads, kv, dk, dv, 12, None), S.pibidra_layer(heads, kv, dk, dv, 12, 64)])
    w = S.pibidra_weights(cfg, heads, bias_rows=4)
    toks = np.random.default_rng(dk).integers(0, 96, 24).tolist()

    def outputs():
        plan = make_plan(pkg, cfg, w, ctx=32, batch=16, compute=compute)
        try:
            out = [plan.forward_batch_logits(toks[:15], 0, list(range(15)))[0], plan.forward_batch_logits(toks[15:16], 15, [0])[0], plan.forward_batch_logits(toks[16:22], 16, [5])[0]]
            out += [plan.forward_decode(t, 22 + i)[0] for i, t in enumerate(toks[22:])]
            out += [plan.read_buffer(name, 24 * kv * size, layer=run) for run in (0, 1) for name, size in (("key_cache", dk), ("value_cache", dv))]
            return out
        finally:
            plan.free()

    got = outputs()
    monkeypatch.setenv("B200_LAYERED_PREP", "general")
    for i, (a, b) in enumerate(zip(got, outputs())):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), i
