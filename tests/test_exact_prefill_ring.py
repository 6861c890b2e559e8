"""CPU model of the operand ring of the exact Q8_0 prefill's product (csrc/exact_prefill.cuh, k_xp_gemm) with the kernel's own stage and phase expressions, under random
interleavings of its four warps and its copies, where waits may give up at any time: no copy lands in a stage that a warp has still to read, every warp ends, and a product without
a wait that gave up has read every chunk from its own stage.  A thread 0 that does not wait for a stage to come free (planted here, wait=False) is found out."""
import random

import pytest

STAGES, WARPS = 3, 4


class Hazard(Exception):
    pass


def product(n_chunks, rng, give_up, wait=True):
    """One CTA.  Returns whether a wait gave up; raises Hazard where a copy lands in a stage that is still read, or a warp reads another chunk than its own."""
    holds = [None] * STAGES                      # the chunk that a stage's copies brought (None: nothing yet, or on their way)
    filled, freed = [0] * STAGES, [0] * STAGES   # completed phases of the full and of the empty barriers
    arrived = [0] * STAGES
    in_flight = []                               # (stage, chunk)
    reading = [None] * WARPS                     # the stage that a warp is in
    failed = []
    place = {"chunk": 0, "stage": 0}             # thread 0's

    def fetch():
        stage, chunk = place["stage"], place["chunk"]
        holds[stage] = None
        in_flight.append((stage, chunk))
        if stage in reading:
            raise Hazard("a copy into a stage that a warp reads")
        place["chunk"], place["stage"] = chunk + 1, (stage + 1) % STAGES

    def waits(barrier, stage, phase):
        while barrier[stage] <= phase:           # (phase completed: its parity has flipped)
            if failed or rng.random() < give_up:
                return False
            yield
        return True

    def warp(w):
        dead = False
        for c in range(n_chunks):
            stage, phase = c % STAGES, c // STAGES
            ok = (not dead) and (yield from waits(filled, stage, phase))
            if not ok:
                failed.append(w)
                return
            reading[w] = stage
            if holds[stage] != c:
                raise Hazard("a warp reads another chunk")
            for _ in range(rng.randrange(4)):
                yield
                if holds[stage] != c:
                    raise Hazard("the stage changed under a warp")
            reading[w] = None
            arrived[stage] += 1
            if arrived[stage] == WARPS:
                arrived[stage], freed[stage] = 0, freed[stage] + 1
            if w == 0 and c + STAGES < n_chunks:
                dead = wait and not (yield from waits(freed, stage, phase))
                if not dead:
                    fetch()

    for _ in range(min(STAGES, n_chunks)):
        fetch()
    running = {w: warp(w) for w in range(WARPS)}
    while running:
        if in_flight and rng.random() < 0.5:
            stage, chunk = in_flight.pop(rng.randrange(len(in_flight)))
            holds[stage] = chunk
            filled[stage] += 1
            continue
        w = rng.choice(list(running))
        try:
            next(running[w])
        except StopIteration:
            del running[w]
    return bool(failed)


@pytest.mark.parametrize("give_up", [0.0, 0.002, 0.02])
def test_ring(give_up):
    rng = random.Random(5)
    ended = [product(rng.randrange(1, 24), rng, give_up) for _ in range(3000)]
    assert any(ended) == (give_up > 0)


def test_a_missing_wait_is_found():
    rng = random.Random(6)
    with pytest.raises(Hazard):
        for _ in range(100):
            product(rng.randrange(6, 24), rng, 0.0, wait=False)
