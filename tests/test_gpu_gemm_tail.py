"""The last, partial round of the persistent CTA-pair GEMM in narrower tiles (csrc/prefill_gemm.cuh, cut_tiles), against an fp32 matmul of the same operands.
74 CTA pairs walk tiles of 256 x 256: the column counts leave no partial round, one tile of it, the most that 64-wide and 128-wide tiles take, and one more than
that (which stays wide); K down to a single stage.  Tolerance: that of the other GEMM test (the order of the fp32 sums), 1e-4 of the largest value."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resid", [0, 1])
@pytest.mark.parametrize("m,tiles,k", [(256, 73, 64), (256, 74, 128), (256, 75, 64), (256, 92, 192), (256, 93, 64), (256, 111, 320), (256, 112, 64), (512, 38, 64),
                                       (512, 46, 448), (512, 56, 128), (768, 25, 64), (768, 37, 192)])
def test_matches_fp32(pkg, m, tiles, k, resid):
    n = 256 * tiles
    rng = np.random.default_rng(m + n + k)
    a = (rng.standard_normal((m, k)) * 0.5).astype(np.float16)
    b = (rng.standard_normal((n, k)) * 0.5).astype(np.float16)
    ref = a.astype(np.float32) @ b.astype(np.float32).T
    env = {"B200_GEMM_2CTA": "1256", **({"B200_GEMM_RESID": "1"} if resid else {})}
    os.environ.update(env)
    try:
        c, _ = pkg.native.gemm_f16(a, b, iters=2)
    finally:
        for key in env:
            del os.environ[key]
    assert np.max(np.abs(c - ref)) <= 1e-4 * np.max(np.abs(ref))
