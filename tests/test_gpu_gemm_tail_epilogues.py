"""The narrow tiles of the persistent CTA-pair GEMM's last round (csrc/prefill_gemm.cuh, cut_tiles) under the epilogues that compute something: the gated pair of FP16
GGUF plans and of BF16 layered plans, and the squared ReLU.  74 CTA pairs walk tiles of 256 columns (gated: 128 of each matrix); the counts below leave one tile of the
last round, the most that 64-wide tiles take, and what 128-wide tiles take.  Tolerances are those of the other tests of each path (operands rounded to 16 bits)."""
import numpy as np
import pytest

import test_gpu_pibidra as pibidra
import test_gpu_zulesun as zulesun
from pibidra_util import oracle, w64
from test_gpu_prefill import _prefill_and_compare

pytestmark = pytest.mark.gpu

CLUSTERS = 74


def narrow(pairs, tiles):  # width of the tiles of the last round, as cut_tiles chooses it
    wide = CLUSTERS * (pairs * tiles // CLUSTERS) // pairs
    left = (tiles - wide) * 256
    return next((w for w in (64, 128) if wide and left and -(-left // w) * pairs <= CLUSTERS), 256)


# two layers: the second one's cache shows every row of the first one's feed-forward
@pytest.mark.parametrize("tokens,tiles,width", [(200, 75, 64), (200, 92, 64), (130, 93, 128), (400, 38, 64), (300, 46, 64), (300, 50, 128)])
def test_gated_f16(pkg, orc, tokens, tiles, width):
    assert narrow(-(-tokens // 256), tiles) == width
    S, F16 = pkg.synth, pkg.gguf.GGMLType.F16
    shape = S.Shape("llama", 256, 128 * tiles, 2, 4, 2, 64, 256, False, 10000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, F16, S.build_tensors_fast(shape, F16, seed=tiles), tokens + 8)
    _prefill_and_compare(pkg, orc, model, tokens, tokens)


@pytest.mark.parametrize("tokens,tiles,width", [(150, 75, 64), (256, 93, 128), (300, 38, 64)])
def test_gated_bf16(pkg, tokens, tiles, width):
    assert narrow(-(-tokens // 256), tiles) == width
    S = pkg.synth
    cfg = S.pibidra_config(128, 96, [S.pibidra_layer(2, 1, 64, 64, 40, 128 * tiles)])
    w = S.pibidra_weights(cfg, tiles, bias_rows=32)
    toks = np.random.default_rng(tiles).integers(0, 96, tokens).tolist()
    ref = oracle().forward(cfg, w64(w), toks)
    plan = pibidra.make_plan(pkg, cfg, w, ctx=tokens + 8, batch=tokens, compute="bfloat16")
    try:
        pibidra.assert_rows(pibidra.prefill_all(plan, toks, tokens), ref, pibidra.TOL["bfloat16"])
    finally:
        plan.free()


@pytest.mark.parametrize("tokens,tiles,width", [(150, 75, 64), (256, 93, 128), (300, 38, 64)])
def test_squared_relu_bf16(pkg, tokens, tiles, width):
    assert narrow(-(-tokens // 256), tiles) == width
    S, O = pkg.synth, zulesun.oracle()
    cfg = S.zulesun_config(128, 96, [S.zulesun_lightning(1, 64, 64, S.zulesun_dense(256 * tiles))], side=None)
    toks = np.random.default_rng(tiles).integers(0, 96, tokens).tolist()
    w = S.zulesun_weights(cfg, tiles)
    w["l0.norm1b"][:] = -1.0  # the mixer adds nothing: the feed-forward alone
    w = zulesun.bf16_values(w)
    ref = O.forward(cfg, zulesun.w64(w), toks)
    plan = zulesun.make_plan(pkg, cfg, w, ctx=tokens + 8, batch=tokens, compute="bfloat16")
    try:
        zulesun.assert_rows(zulesun.prefill_all(plan, toks, tokens), ref, zulesun.tol("bfloat16", cfg))
    finally:
        plan.free()
