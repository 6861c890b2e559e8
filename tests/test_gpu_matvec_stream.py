"""Decode projections of layered plans at the edges of the streaming kernel (csrc/layered.cuh, k_matvec_stream_bf16): rows of one, of several and of a ragged number of
2048-column segments, fewer rows than warps and several rows a warp, gated pairs, and widths that keep a warp per row, against the float64 oracle.  Tolerance: the FP32
bound of every other decode test (only the order of sums differs)."""
import numpy as np
import pytest

from pibidra_util import oracle, w64
from test_gpu_pibidra import TOL_DECODE, assert_rows, make_plan

pytestmark = pytest.mark.gpu


# (width, feed-forward width, vocabulary): the feed-forward width is the down projection's row, the width every other projection's
@pytest.mark.parametrize("width,ff,vocab", [(1024, 1024, 2500), (1032, 2056, 300), (1016, 4104, 64), (2048, 1048, 5000), (2056, 2048, 33), (4096, 1024, 96), (4104, 1096, 50)])
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
