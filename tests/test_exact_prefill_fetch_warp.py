"""CPU model of the operand ring of the exact Q8_0 prefill's product (csrc/exact_prefill.cuh, k_xp_gemm) as a warp of its own fills it, with the kernel's stage and phase
expressions, for rings of 3 to 8 stages under random interleavings, where waits may give up at any time: no copy lands in a stage that a warp has still to read, every warp ends, and
a product without a wait that gave up has read every chunk.  A fetching warp that does not wait for a stage to come free (planted here) is found out."""
import random

import pytest

WARPS = 4


class Hazard(Exception):
    pass


def product(n_chunks, stages, rng, give_up, wait=True):
    holds, reading = [None] * stages, [None] * WARPS
    filled, freed, arrived = [0] * stages, [0] * stages, [0] * stages  # completed phases of the full and the empty barriers
    in_flight, failed, seen = [], [], [0] * WARPS

    def waits(barrier, stage, parity):  # mbarrier.try_wait.parity: true once the phase of that parity is over
        while barrier[stage] % 2 == parity:
            if failed or rng.random() < give_up:
                return False
            yield
        return True

    def fetcher():
        stage, ph = 0, 1
        for c in range(n_chunks):
            if wait and not (yield from waits(freed, stage, ph)):
                failed.append("fetch")
                return
            if stage in reading:
                raise Hazard("a copy into a stage that a warp reads")
            holds[stage] = None
            in_flight.append((stage, c))
            stage += 1
            if stage == stages:
                stage, ph = 0, ph ^ 1
            yield

    def warp(w):
        stage, ph = 0, 0
        for c in range(n_chunks):
            if not (yield from waits(filled, stage, ph)):
                failed.append(w)
                return
            reading[w] = stage
            for _ in range(1 + rng.randrange(3)):
                if holds[stage] != c:
                    raise Hazard("a warp reads another chunk")
                yield
            reading[w] = None
            seen[w] += 1
            arrived[stage] += 1
            if arrived[stage] == WARPS:
                arrived[stage], freed[stage] = 0, freed[stage] + 1
            stage += 1
            if stage == stages:
                stage, ph = 0, ph ^ 1

    running = [fetcher()] + [warp(w) for w in range(WARPS)]
    for _ in range(100000):
        if not running:
            break
        if in_flight and rng.random() < 0.3:
            stage, c = in_flight.pop(rng.randrange(len(in_flight)))
            holds[stage], filled[stage] = c, filled[stage] + 1
        r = rng.choice(running)
        try:
            next(r)
        except StopIteration:
            running.remove(r)
    assert not running
    return bool(failed), seen


@pytest.mark.parametrize("stages", range(3, 9))
def test_ring(stages):
    for seed in range(120):
        rng = random.Random(seed * 8 + stages)
        n = rng.randrange(1, 30)
        failed, seen = product(n, stages, rng, rng.choice((0.0, 0.0, 0.002)))
        assert failed or seen == [n] * WARPS


def test_a_missing_wait_is_found():
    with pytest.raises(Hazard):
        for seed in range(200):
            product(12, 3, random.Random(seed), 0.0, wait=False)
