"""Q8_0 plans whose query and key heads of one token are wider than the shared memory that the batched exact prefill rotates them in (220 KB): the chunk goes token by
token.  The shape in front of the limit is multiplied at once; both leave the token-by-token path's bits.  Rows of 218 heads of 128 have no segments of
whole 32-column blocks that the streaming path takes: that plan is off it."""
import numpy as np
import pytest

from test_gpu_exact_prefill import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv,why", [(216, 216, ""), (218, 218, "streaming"), (219, 219, "wider"), (224, 224, "wider"), (256, 256, "wider")])
def test_wide_rows(pkg, heads, kv, why):
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    assert ((heads + kv) * 129 * 4 <= 220 * 1024) == (heads <= 218)
    shape = S.Shape("qwen3", 128, 128, 2, heads, kv, 128, 64, False, 500000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=heads), 24)
    toks = np.random.default_rng(heads).integers(0, 64, 16)
    check(pkg, model, toks, [9, 6], 16, why)
