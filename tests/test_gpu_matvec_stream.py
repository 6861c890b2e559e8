"""Decode projections of layered plans at the edges of the streaming kernel (csrc/layered.cuh, k_matvec_stream_bf16), against the float64 oracle.  On 148 SMs its 296 CTAs have
2368 warps, and matrices of fewer than 585 rows take a CTA per row.  Rows of one, of several and of a ragged number of 2048-column segments; several rows a warp, of one segment
and of three; warps without a row; gated pairs, one and two a warp; experts' and heads' views of stacked matrices; and widths that keep a warp per row.  Tolerance: the FP32
bound of every other decode test (only the order of sums differs)."""
import numpy as np
import pytest

import latusun_util
import test_gpu_latusun
from pibidra_util import oracle, w64
from test_gpu_pibidra import TOL_DECODE, assert_rows, make_plan

pytestmark = pytest.mark.gpu


# (width, feed-forward width, vocabulary): the feed-forward width is the down projection's row, the width every other projection's.  The last three: warps of the last CTA without
# a row; 2504 rows of three segments, so that warps go on to a second row; 2408 gated pairs of three segments, likewise
@pytest.mark.parametrize("width,ff,vocab", [(1024, 1024, 2500), (1032, 2056, 300), (1016, 4104, 64), (2048, 1048, 5000), (2056, 2048, 33), (4096, 1024, 96), (4104, 1096, 50), (1024, 1024, 2003),
                                           (2504, 4104, 64), (4104, 2408, 40)])
def test_projections(pkg, width, ff, vocab):
    S = pkg.synth
    cfg = S.pibidra_config(width, vocab, [S.pibidra_layer(2, 1, 16, 24, 8, ff)])
    w = S.pibidra_weights(cfg, width, bias_rows=8)
    toks = np.random.default_rng(ff).integers(0, vocab, 4).tolist()
    ref = oracle().forward(cfg, w64(w), toks)
    plan = make_plan(pkg, cfg, w, ctx=16, batch=1)
    try:
        assert_rows(np.stack([plan.forward_decode(t, i)[0] for i, t in enumerate(toks)]), ref, TOL_DECODE)
    finally:
        plan.free()


# The down projection of the chosen experts (rows of 1048 columns of a stack of three, two of them a step, 600 and 1032 rows each) and the value expansion of heads with a latent of
# 1024 entries (three heads' rows of a stack)
@pytest.mark.parametrize("width,heads,rank", [(600, 3, 16), (1032, 3, 1024)])
def test_views(pkg, width, heads, rank):
    S, O = pkg.synth, latusun_util.oracle()
    cfg = S.latusun_config(width, 96, [S.latusun_layer("latent_attention", heads, 8, 4, 16, rank, experts=3, top=2, ff=1048)], logit_softcap=None)
    w = test_gpu_latusun.weights(S, cfg, width, "float32")
    toks = np.random.default_rng(width).integers(0, 96, 5).tolist()
    ref = O.forward(cfg, latusun_util.w64(w), toks)
    plan = test_gpu_latusun.make_plan(pkg, cfg, w, ctx=16, batch=1)
    try:
        assert_rows(np.stack([plan.forward_decode(t, i)[0] for i, t in enumerate(toks)]), ref, test_gpu_latusun.TOL_DECODE)
    finally:
        plan.free()


# An infinite first entry of the activation is infinite in every result and in no other way: lanes of a warp's last load that lie behind the row (1032, 2504 columns) take part in
# no product.  1016 columns keep a warp per row, 1280 have no such lanes.
@pytest.mark.parametrize("width", [1016, 1032, 1280, 2504])
def test_infinite_activation(pkg, width):
    S, vocab = pkg.synth, 2500
    cfg = S.pibidra_config(width, vocab, [S.pibidra_layer(2, 1, 16, 24, 8, 64)])
    w = S.pibidra_weights(cfg, width, bias_rows=8)
    w["embed"][:, 0] = 50.0
    w["final.norm"][0] = 3e38
    w["head"][:, 0] = np.where(np.arange(vocab) % 3 == 0, -1.0, 1.0)
    plan = make_plan(pkg, cfg, w, ctx=16, batch=1)
    logits = plan.forward_decode(7, 0)[0]
    plan.free()
    assert np.array_equal(logits, np.where(np.arange(vocab) % 3 == 0, -np.inf, np.inf).astype(np.float32))
