"""Two plans that prefill at the same time from two threads, in chunks whose products have rings of different depth (csrc/exact_prefill.cuh: a chunk of few tiles has deep ones), with the
same kernel instance: every chunk goes through, and each plan's cache is the one that it has alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_plans(pkg, monkeypatch):
    monkeypatch.setenv("B200_XP_TILE", "16")
    S, Q8 = pkg.synth, pkg.gguf.GGMLType.Q8_0
    plans, toks, want = [], [], []
    for shape, n, seed in (("tiny-llama", 16, 1), ("small-llama", 96, 2)):
        model = pkg.loader.model_from_tensors(S.SHAPES[shape], Q8, S.build_tensors_fast(S.SHAPES[shape], Q8, seed=seed), n + 4)
        plans.append((pkg.B200MasterPlan(model, prefill_batch_size=n), model.configuration))
        toks.append(np.random.default_rng(seed).integers(0, S.SHAPES[shape].vocab, n).astype(np.int32))

    def cache(i):
        plan, c = plans[i]
        return plan.read_buffer("key_cache", len(toks[i]) * c.kv_dim, layer=c.n_layers - 1).view(np.uint32).copy()

    for i in range(2):
        plans[i][0].forward_batch_prefill(toks[i], 0)
        want.append(cache(i))
    errors = []

    def work(i):
        try:
            for _ in range(600):
                plans[i][0].forward_batch_prefill(toks[i], 0)
                if errors:
                    break
            assert np.array_equal(cache(i), want[i])
        except Exception as e:
            errors.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for plan, _ in plans:
        plan.free()
