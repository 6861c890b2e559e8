"""b200_forward_decode into pinned and pageable buffers, at vocabularies on both sides of the line from which a pinned buffer is written without a copy on the host
(csrc/plan.cu, logits_direct): the logits and the greedy token are the same bit for bit, and nothing is written behind the row."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [4096, 24575, 24576, 128256])
def test_buffers(pkg, vocab):
    import torch

    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    shape = S.Shape("llama", 256, 512, 1, 4, 2, 64, vocab, False, 500000.0, 1e-5)
    plan = pkg.B200MasterPlan(pkg.loader.model_from_tensors(shape, Q8, S.build_tensors_fast(shape, Q8, seed=vocab), 32), prefill_batch_size=1)
    seen = []
    for pinned in (False, True):
        row = torch.full((vocab + 8,), -7.0)
        row = row.pin_memory() if pinned else row
        for position, token in enumerate((5, 9, 11)):
            got = ctypes.c_int32(-1)
            rc = pkg.native.lib().b200_forward_decode(plan._native._p, token, position, row.data_ptr(), ctypes.byref(got))
            assert rc == 0 and got.value == int(np.argmax(row[:vocab].numpy())) and bool((row[vocab:] == -7.0).all())
            seen.append((got.value, row[:vocab].numpy().tobytes()))
    assert seen[:3] == seen[3:]
    plan.free()
