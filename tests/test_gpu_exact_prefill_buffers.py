"""What b200_read_buffer finds behind an exact prefill chunk of a Q8_0 plan: every single-token buffer holds what the last token's own step leaves there, the
quantised activations included.  Shapes: attention output as wide as the model, wider (its tail stays in xq / xs behind the norms' row) and three layers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffers(plan, c):
    wide = max(c.dim, c.n_heads * c.head_size)
    sizes = {"x": (c.dim, np.float32), "qkv": (c.n_heads * c.head_size + 2 * c.kv_dim, np.float32), "hb": (c.hidden_dim, np.float32), "xq": (wide, np.int8), "xs": (wide // 32, np.float32),
             "hq": (c.hidden_dim, np.int8), "hs": (c.hidden_dim // 32, np.float32)}
    return {name: plan.read_buffer(name, n, dtype) for name, (n, dtype) in sizes.items()}


@pytest.mark.parametrize("shape", ["tiny-llama", "tiny-qwen3", "tiny-phi3", "small-llama"])
@pytest.mark.parametrize("n", [2, 9, 64, 70])
def test_buffers(pkg, make_model, shape, n):
    model = make_model(shape, pkg.gguf.GGMLType.Q8_0, ctx=n + 4)
    c = model.configuration
    toks = np.random.default_rng(n).integers(0, c.vocab_size, n + 1).astype(np.int32)
    out = []
    for batch in (1, 96):
        plan = pkg.B200MasterPlan(model, prefill_batch_size=batch)
        plan.forward_decode(int(toks[n]), 0)  # something else in every buffer
        if batch == 1:
            for p in range(n):
                plan.forward_prefill(int(toks[p]), p)
        else:
            plan.forward_batch_prefill(toks[:n], 0)
        out.append(buffers(plan, c))
        plan.free()
    for name in out[0]:
        assert out[0][name].tobytes() == out[1][name].tobytes(), name
