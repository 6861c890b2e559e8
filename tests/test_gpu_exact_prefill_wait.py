"""The bounded waits of the exact prefill's products (csrc/exact_prefill.cuh, xp_wait; csrc/exact_prefill_umma.cuh): a tile whose operands arrive in part only (its
stages never fill) ends with the error word set, every warp of it, and the context goes on as before."""
import pytest

pytestmark = pytest.mark.gpu


def test_operands_that_do_not_arrive(pkg, make_model):
    before, starved, after = pkg.native.test_exact_prefill_wait()
    assert before[0] == 0 and before[1] < 900
    assert starved[0] == 200 and 1000 <= starved[1] < 1100  # the first wait in full, the drained stages a tenth of a millisecond each
    assert after[0] == 0 and after[1] < 10
    model = make_model("tiny-llama", pkg.gguf.GGMLType.Q8_0, ctx=32)
    plan = pkg.B200MasterPlan(model, prefill_batch_size=16)
    plan.forward_batch_prefill(list(range(3, 14)), 0)
    assert plan.exact_prefill_info()[1] == 1
    plan.free()


@pytest.mark.parametrize("form", [1, 2, 3, 4])
def test_other_tiles(pkg, form):
    """1, 2 and 4: the fetching warp has issued every chunk when the others give up, and waits for their copies, as long as a copy takes and no longer than a wait's
    limit; 3: on tcgen05, every role waits."""
    before, starved, after = pkg.native.test_exact_prefill_wait(form)
    assert before[0] == 0 and before[1] < 900
    assert starved[0] == 200 and 1000 <= starved[1] < 1100
    assert after[0] == 0 and after[1] < 10
