"""The delta rule in blocks of four tokens (csrc/delta.cuh, k_delta_coef / k_delta_rule_blocks) against the float64 oracle: every register shape (key sizes of
1, 2, 4 and 8 entries a lane, whole and ragged), portions that end inside a block of four and inside a staged block, and the single-row kernel in between.

Tolerance: FP32 compute mode differs from the oracle in the order of FP32 sums only; 3e-5 relative RMS is the bound of every other Lerosun test."""
import numpy as np
import pytest

from lerosun_util import oracle, w64
from test_gpu_lerosun import assert_rows, make_plan, portions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dk,dv", [(2, 1, 16, 16), (3, 3, 13, 9), (4, 2, 32, 24), (5, 5, 20, 70), (2, 2, 64, 64), (4, 1, 50, 8), (2, 1, 128, 130), (6, 2, 100, 33), (1, 1, 4, 4)])
def test_portions(pkg, heads, kv_heads, dk, dv):
    S = pkg.synth
    cfg = S.lerosun_config(48, 64, [S.lerosun_delta(heads, kv_heads, dk, dv, 3, None)])
    w = S.lerosun_weights(cfg, dk)
    toks = np.random.default_rng(dv).integers(0, 64, 75).tolist()
    ref = oracle().forward(cfg, w64(w), toks)
    plan = make_plan(pkg, cfg, w, batch=64)
    try:
        for sizes in ([3, 4, 5, 7, 8, 9, 2, 1, 16, 17], [63, 11], [64, 3, 1]):
            assert_rows(portions(plan, toks, sizes, 64), ref, 3e-5, f"portions {sizes}")
    finally:
        plan.free()
