"""The decode step's attention over a cluster of CTAs (csrc/layered.cuh, k_step_attention), the row kernel in registers and the wide argmax, against the float64
oracles: windows at the edges of a key tile (64 keys) and of the parts of a head (32 keys and more), rings that wrap, key sizes whose tiles hold fewer rows, and
logits rows that are no multiple of four.  Tolerance: the FP32 bound of every other Pibidra test (only the order of sums differs)."""
import numpy as np
import pytest

from pibidra_util import oracle, w64
from test_gpu_pibidra import TOL_DECODE, assert_rows, make_plan, prefill_all

pytestmark = pytest.mark.gpu


def decode_behind(pkg, cfg, w, n, steps, batch):
    """`n` tokens in chunks, then `steps` decode steps: the logits of the steps and the oracle's."""
    toks = np.random.default_rng(n).integers(0, cfg["vocab"], n + steps).tolist()
    ref = oracle().forward(cfg, w64(w), toks)
    plan = make_plan(pkg, cfg, w, ctx=n + steps + 1, batch=batch)
    try:
        prefill_all(plan, toks[:n], batch)
        return np.stack([plan.forward_decode(t, n + i)[0] for i, t in enumerate(toks[n:])]), ref[n:]
    finally:
        plan.free()


@pytest.mark.parametrize("window", [1, 31, 32, 63, 64, 65, 127, 128, 129, 255, 256, 257, 600])
def test_windows(pkg, window):
    S = pkg.synth
    cfg = S.pibidra_config(64, 96, [S.pibidra_layer(4, 2, 16, 24, window, 96), S.pibidra_layer(2, 1, 64, 32, max(1, window - 1), 96)])
    w = S.pibidra_weights(cfg, window, bias_rows=16)
    got, ref = decode_behind(pkg, cfg, w, 290, 12, 37)
    assert_rows(got, ref, TOL_DECODE)


# (heads, key/value heads, key size, value size): one lane to 32 lanes a row, tiles of 64 down to 16 rows, values over more threads than a warp; sizes that are
# no multiple of four keep the general kernel
@pytest.mark.parametrize("heads,kv,dk,dv", [(2, 1, 4, 4), (3, 1, 12, 20), (5, 5, 32, 128), (2, 2, 128, 8), (1, 1, 256, 256), (40, 8, 16, 16), (3, 3, 10, 6)])
def test_head_shapes(pkg, heads, kv, dk, dv):
    S = pkg.synth
    cfg = S.pibidra_config(64, 97, [S.pibidra_layer(heads, kv, dk, dv, 150, 64, softcap=6.0)])
    w = S.pibidra_weights(cfg, dk, bias_rows=12)
    got, ref = decode_behind(pkg, cfg, w, 180, 6, 64)
    assert_rows(got, ref, TOL_DECODE)


# a single row of up to 4096 entries stays in registers, with the steps of a loop and without
@pytest.mark.parametrize("width", [4, 1020, 1024, 1028, 2048, 2052, 4096, 4100, 1030])
def test_norm_rows(pkg, width):
    S = pkg.synth
    cfg = S.pibidra_config(width, 50, [S.pibidra_layer(2, 1, 8, 8, 5, 16), S.pibidra_layer(2, 1, 8, 8, 5, None), S.pibidra_layer(1, 1, 8, 8, 5, 16)], loop=(1, 2, 3), embedding_scale=2.0)
    w = S.pibidra_weights(cfg, 5, bias_rows=4)
    got, ref = decode_behind(pkg, cfg, w, 9, 4, 4)
    assert_rows(got, ref, TOL_DECODE)


# the device-side argmax of the layered step: equal to the first maximum of the logits it returns; 32768 logits and the remainders behind them
@pytest.mark.parametrize("vocab", [1, 2, 3, 5, 4095, 4098, 32767, 32768, 32771, 70001])
def test_argmax(pkg, vocab):
    S = pkg.synth
    cfg = S.pibidra_config(16, vocab, [S.pibidra_layer(1, 1, 8, 8, 4, 8)])
    w = S.pibidra_weights(cfg, 3, bias_rows=4)
    for name in list(w):  # rows of the classifier repeat, so that the maximum is shared: the first one has to win
        if w[name].ndim == 2 and w[name].shape[0] == vocab and vocab > 8:
            w[name][vocab // 2:] = w[name][: vocab - vocab // 2]
    plan = make_plan(pkg, cfg, w, ctx=16, batch=4)
    try:
        for p in range(5):
            lg, am = plan.forward_decode(p % vocab, p)
            assert am == int(np.argmax(lg))
    finally:
        plan.free()


# q | k | v of a row in registers (k_qk_prep_reg): 2048, 4096 and 8192 entries, one step more, which takes the next kernel or the general one
@pytest.mark.parametrize("heads,kv,dk,dv", [(14, 1, 128, 128), (14, 1, 128, 132), (16, 8, 128, 128), (16, 8, 128, 132), (48, 8, 128, 128), (48, 8, 128, 132)])
def test_projection_rows(pkg, heads, kv, dk, dv):
    S = pkg.synth
    cfg = S.pibidra_config(64, 96, [S.pibidra_layer(heads, kv, dk, dv, 12, None)])
    w = S.pibidra_weights(cfg, heads, bias_rows=4)
    got, ref = decode_behind(pkg, cfg, w, 20, 3, 8)
    assert_rows(got, ref, TOL_DECODE)
