"""The decode attention over latent rows (csrc/layered.cuh, k_step_attention<2, true>: values inside the key rows, all rows of a CTA in shared memory at once): logits against the same
position's from a prompt that goes through the chunk attention, in FP32.  Positions at the edges of the groups of rows (4), of the keys that a part is worth (32) and of the eight parts, and a
context whose rows do not fit, which takes the ring.  Both sides sum FP32 products of at most 320 terms in other orders: a relative error of sqrt(320) * 2^-24 per sum, 1e-6, over a
handful of sums behind one another; 2e-5 of the logits' norm bounds it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("positions,context", [([1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 127, 128, 255, 256, 257], 264), ([40, 300], 4000)])
def test_against_the_prompt(pkg, positions, context):
    cfg = pkg.synth.latusun_config(256, 512, [pkg.synth.latusun_layer("latent_attention", 8, 48, 16, 64, 256, experts=4, top=2, ff=128)])
    weights = pkg.synth.latusun_weights(cfg, 3)
    toks = np.random.default_rng(5).integers(0, 512, max(positions) + 1).astype(np.int32)
    plan = pkg.B200MasterPlan.initialize_plan(pkg.synth.latusun_model(cfg, weights, context), prefill_batch_size=512, compute="float32")
    want = plan.forward_batch_logits(toks, 0, positions)[0]
    for row, p in enumerate(positions):
        got = plan.forward_decode(int(toks[p]), p)[0]
        assert np.linalg.norm(got - want[row]) <= 2e-5 * np.linalg.norm(want[row]), p
    plan.free()
