"""The decode step's attention over a cluster (csrc/layered.cuh, k_step_attention) where a CTA's keys and values take more tiles than its ring has stages (4), so that
stages are filled again: windows of 1000 keys and more, rows of 128, 256 and 576 entries, a ring that has wrapped.  Against the float64 oracles; tolerances are those
of the other tests of these plans (the order of FP32 sums)."""
import numpy as np
import pytest

import latusun_util
import test_gpu_latusun as latusun
from test_gpu_pibidra import TOL_DECODE, assert_rows
from test_gpu_step_attention import decode_behind

pytestmark = pytest.mark.gpu

STAGES, STAGE_FLOATS, SMS, MOST_PARTS = 4, 4096, 148, 8


def tiles(keys, heads, row):
    parts = max(1, min(SMS // heads, MOST_PARTS))
    return -(-(-(-keys // parts)) // min(64, STAGE_FLOATS // row))


# (heads, key/value heads, key size, value size, window, tokens in front): within the window and behind it, where the ring (a window and a chunk) has wrapped
@pytest.mark.parametrize("heads,kv,dk,dv,window,n", [(40, 8, 128, 128, 1000, 700), (40, 8, 128, 128, 1000, 1300), (16, 4, 256, 256, 1100, 1400), (48, 6, 64, 256, 1024, 1200)])
def test_windows_of_many_tiles(pkg, heads, kv, dk, dv, window, n):
    assert min(tiles(min(n, window), heads, dk), tiles(min(n, window), heads, dv)) > STAGES
    S = pkg.synth
    cfg = S.pibidra_config(64, 96, [S.pibidra_layer(heads, kv, dk, dv, window, 64, softcap=6.0)])
    w = S.pibidra_weights(cfg, dk + n, bias_rows=32)
    got, ref = decode_behind(pkg, cfg, w, n, 5, 128)
    assert_rows(got, ref, TOL_DECODE)


# one shared key/value row of 512 + 64 entries per token: seven rows a tile
def test_latent_rows(pkg):
    S, O, n = pkg.synth, latusun_util.oracle(), 500
    assert tiles(n, 16, 576) > STAGES
    cfg = S.latusun_config(64, 96, [S.latusun_layer("latent_attention", 16, 32, 64, 32, 512, experts=None), S.latusun_layer("latent_attention_2", 8, 32, 64, 32, 512, experts=None)])
    w = S.latusun_weights(cfg, 3)
    toks = np.random.default_rng(3).integers(0, 96, n + 5).tolist()
    ref = O.forward(cfg, latusun_util.w64(w), toks)
    plan = latusun.make_plan(pkg, cfg, w, ctx=n + 8, batch=128)
    try:
        latusun.prefill_all(plan, toks[:n], 128)
        got = np.stack([plan.forward_decode(t, n + i)[0] for i, t in enumerate(toks[n:])])
    finally:
        plan.free()
    latusun.assert_rows(got, ref[n:], latusun.TOL_DECODE)
