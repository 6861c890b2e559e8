"""CPU model of the operand ring of the exact Q8_0 prefill's product (csrc/exact_prefill.cuh, k_xp_gemm) as a warp of its own fills it, with the kernel's stage and
phase expressions, for rings of 3 to 8 stages under random interleavings, where waits may give up at any time: no copy lands in a stage that a warp has still to
read, every warp ends, a product without a wait that gave up has read every chunk, and no copy is on its way where the gate/up form takes the ring for its hidden
units or the block ends.  Found out where planted: a fetching warp that does not wait for a stage to come free, and one that waits for its last copies only if a wait
of its own gave up, or not at all."""
import random

import pytest

WARPS = 4


class Hazard(Exception):
    pass


def product(n_chunks, stages, rng, give_up, wait=True, drain="always", gateup=False):
    holds, reading = [None] * stages, [None] * WARPS
    filled, freed, arrived = [0] * stages, [0] * stages, [0] * stages  # completed phases of the full and the empty barriers
    in_flight, failed, seen, at_barrier = [], [], [0] * WARPS, [0]

    def waits(barrier, stage, parity):  # mbarrier.try_wait.parity: true once the phase of that parity is over
        while barrier[stage] % 2 == parity:
            if failed or rng.random() < give_up:
                return False
            yield
        return True

    def epilogue():  # the gate/up form: a barrier, then the ring is the hidden units'
        if not gateup:
            return
        at_barrier[0] += 1
        while at_barrier[0] <= WARPS:
            yield
        if in_flight:
            raise Hazard("a copy into the hidden units")

    def fetcher():
        stage, ph, issued, ok = 0, 1, 0, True
        for c in range(n_chunks):
            if wait and not (yield from waits(freed, stage, ph)):
                failed.append("fetch")
                ok = False
                break
            if stage in reading:
                raise Hazard("a copy into a stage that a warp reads")
            holds[stage] = None
            in_flight.append((stage, c))
            issued += 1
            stage += 1
            if stage == stages:
                stage, ph = 0, ph ^ 1
            yield
        if drain == "always" or (drain == "own" and not ok):
            for _ in range(min(issued, stages)):
                if stage == 0:
                    stage, ph = stages, ph ^ 1
                stage -= 1
                while filled[stage] % 2 == ph ^ 1:  # (its limit is far above the time of a copy)
                    if not any(s == stage for s, _ in in_flight):
                        raise Hazard("waits for what was never issued")
                    yield
        yield from epilogue()

    def warp(w):
        stage, ph = 0, 0
        for c in range(n_chunks):
            if not (yield from waits(filled, stage, ph)):
                failed.append(w)
                break
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
        yield from epilogue()

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
    if in_flight:
        raise Hazard("a copy into the memory of a block that has ended")
    return bool(failed), seen


@pytest.mark.parametrize("stages", range(3, 9))
def test_ring(stages):
    for seed in range(120):
        rng = random.Random(seed * 8 + stages)
        n = rng.randrange(1, 30)
        failed, seen = product(n, stages, rng, rng.choice((0.0, 0.0, 0.002, 0.02)), gateup=seed % 2 == 0)
        assert failed or seen == [n] * WARPS


def test_a_missing_wait_is_found():
    with pytest.raises(Hazard):
        for seed in range(200):
            product(12, 3, random.Random(seed), 0.0, wait=False)


@pytest.mark.parametrize("drain", ["own", "never"])
@pytest.mark.parametrize("gateup", [False, True])
@pytest.mark.parametrize("n", [2, 12])  # fewer chunks than stages; several laps
def test_copies_left_behind_are_found(drain, gateup, n):
    with pytest.raises(Hazard, match="hidden" if gateup else "ended"):
        for seed in range(2000):
            product(n, 4, random.Random(seed), 0.02, drain=drain, gateup=gateup)
