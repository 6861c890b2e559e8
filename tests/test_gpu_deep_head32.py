"""Decode at depth with a CTA per head (csrc/decode_kernels.cuh, k_attention): heads of 32 entries are not shared by a cluster, so they keep the kernel's several
passes over scores and values from 128 keys on, the parallel softmax sum from 512 keys on and, with a long context, the score row in global memory.  Logits against
the CPU path bit for bit on both sides of every switch-over, the cache at the end."""
import numpy as np
import pytest

from test_gpu_parity import assert_bit_equal, set_mode

pytestmark = pytest.mark.gpu

CHECK = {0, 126, 127, 128, 129, 255, 256, 257, 383, 384, 510, 511, 512, 513, 639, 640, 641, 698, 699}


@pytest.mark.parametrize("arch,quant,context", [("llama", "Q8_0", 704), ("qwen3", "Q8_0", 20000), ("llama", "F16", 20000)])
def test_head_size_32(pkg, orc, arch, quant, context):
    S = pkg.synth
    quant = getattr(pkg.gguf.GGMLType, quant)
    shape = S.Shape(arch, 256, 256, 2, 8, 2, 32, 256, False, 10000.0, 1e-5)
    model = pkg.loader.model_from_tensors(shape, quant, S.build_tensors_fast(shape, quant, seed=context), context)
    c, n = model.configuration, 700
    plan = pkg.B200MasterPlan.initialize_plan(model)
    set_mode(pkg, plan, "graph")
    om = orc.OracleModel(model, lanes=16)
    toks = orc.bench_tokens(c.vocab_size, n)
    try:
        for pos in range(n):
            tok = int(toks[pos])
            if pos in CHECK:
                assert_bit_equal(plan.forward_decode(tok, pos)[0], om.forward(tok, pos), f"logits at position {pos}")
            else:
                plan.forward_prefill(tok, pos)
                om.forward(tok, pos, want_logits=False)
        for l in range(c.n_layers):
            for name, ref in (("key_cache", om.key_cache(l)), ("value_cache", om.value_cache(l))):
                assert_bit_equal(plan.read_buffer(name, c.context_length * c.kv_dim, layer=l)[: n * c.kv_dim], np.asarray(ref)[: n * c.kv_dim], f"{name} {l}")
    finally:
        plan.free()
        om.close()
