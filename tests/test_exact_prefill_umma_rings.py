"""CPU model of the rings of the exact Q8_0 prefill's tcgen05 product (csrc/exact_prefill_umma.cuh, k_xt_gemm) with the kernel's stage and phase expressions: weights
as bytes with both scales, activations, weights as FP16, the scales' operands and the sums' columns, under random interleavings of the fetching lane, the operand
warps, the product warp, the summing warps, the copies and the products, where waits may give up at any time.  Nothing is overwritten that has still to be read,
everything that is read is the chunk's, half's or block's own, every role ends, a run without a wait that gave up has summed every block, and no copy or product is
in flight when the block ends, nor is one waited for that was never issued.  Found out where planted: a fetching lane or a product warp that looks back only if a
wait of its own gave up, a look back over more activation stages than there are, and waits that are left out."""
import random

import pytest

W_STAGES, OPERAND_WARPS, SUM_WARPS = 3, 2, 2  # (four and eight in the kernel; what they share is counted the same way)


class Hazard(Exception):
    pass


class Barrier:
    def __init__(self, count):
        self.count, self.arrived, self.phases = count, 0, 0

    def arrive(self):
        self.arrived += 1
        if self.arrived == self.count:
            self.arrived, self.phases = 0, self.phases + 1

    def over(self, parity):  # mbarrier.try_wait.parity: true once the phase of that parity is over
        return self.phases % 2 != parity


def product(segments, nbs, tiles, rng, give_up, left_out=(), drain="always", fin="always", look_back="issued"):
    cps = (nbs + 3) // 4
    chunks = [min(4, nbs - 4 * c) for _ in range(segments) for c in range(cps)]  # blocks of each
    n_chunks = len(chunks)
    wfull, wempty = [Barrier(1) for _ in range(W_STAGES)], [Barrier(OPERAND_WARPS) for _ in range(W_STAGES)]
    afull, aempty = [Barrier(1) for _ in range(2)], [Barrier(1) for _ in range(2)]
    hfull, hempty = [Barrier(OPERAND_WARPS) for _ in range(2)], [Barrier(1) for _ in range(2)]
    tfull, tempty = [Barrier(1) for _ in range(2)], [Barrier(SUM_WARPS) for _ in range(2)]
    end = Barrier(1)
    weights, acts = [None] * W_STAGES, [None] * 2
    halves, scales = ([[None] * OPERAND_WARPS for _ in range(2)] for _ in range(2))
    columns = [None] * 2
    converting, adding = [None] * OPERAND_WARPS, [None] * SUM_WARPS  # the stage that a warp reads, the columns
    copies, queue = [], []  # (memory, stage, chunk, barrier); products and commits in order
    failed, summed = [], [0] * SUM_WARPS

    def waits(name, barrier, parity):
        if name in left_out:
            return True
        while not barrier.over(parity):
            if failed or rng.random() < give_up:
                return False
            yield
        return True

    def waits_to_the_end(barrier, parity, pending):  # (its limit is far above the time of a copy or a product)
        while not barrier.over(parity):
            if not pending():
                raise Hazard("waits for what was never issued")
            yield

    def in_use(kind, stage):
        return any(op[0] == "mma" and op[1][kind] == stage for op in queue)

    def copy(memory, stage, chunk, barrier):
        memory[stage] = None
        copies.append((memory, stage, chunk, barrier))

    def fetcher():
        it = n_weights = n_acts = 0
        ok = True
        for tile in range(tiles):
            for c in range(n_chunks):
                ws, a = it % W_STAGES, it & 1
                if it >= W_STAGES and not (yield from waits("wempty", wempty[ws], (it // W_STAGES - 1) & 1)):
                    ok = False
                    break
                if ws in converting:
                    raise Hazard("weights that are read")
                copy(weights, ws, (tile, c), wfull[ws])
                n_weights = it + 1
                yield
                if it >= 2 and not (yield from waits("aempty", aempty[a], ((it >> 1) - 1) & 1)):
                    ok = False
                    break
                if in_use("a", a):
                    raise Hazard("activations of a product")
                copy(acts, a, (tile, c), afull[a])
                n_acts = it + 1
                it += 1
                yield
            if not ok:
                break
        if not ok:
            failed.append("fetch")
        if drain == "always" or (drain == "own" and not ok):
            if look_back == "three":  # (as if there were three stages, and the last one issued)
                n_acts = n_weights
            for q in range(max(0, n_weights - W_STAGES), n_weights):
                bar = wfull[q % W_STAGES]
                yield from waits_to_the_end(bar, (q // W_STAGES) & 1, lambda: any(cp[3] is bar for cp in copies))
            for q in range(max(0, n_acts - (3 if look_back == "three" else 2)), n_acts):
                bar = afull[q & 1]
                yield from waits_to_the_end(bar, (q >> 1) & 1, lambda: any(cp[3] is bar for cp in copies))

    def operand(w):
        ws = h = sb = 0
        ph_w, ph_h = 0, 1
        for tile in range(tiles):
            for c in range(n_chunks):
                if not (yield from waits("wfull", wfull[ws], ph_w)):
                    failed.append("operand")
                    return
                converting[w] = ws
                for half in range(2):
                    if 2 * half >= chunks[c]:
                        break
                    if weights[ws] != (tile, c):
                        raise Hazard("another chunk's weights")
                    yield
                    if not (yield from waits("hempty", hempty[h], ph_h)):
                        failed.append("operand")
                        converting[w] = None
                        return
                    if in_use("h", h):
                        raise Hazard("FP16 weights of a product")
                    halves[h][w] = (tile, c, half)
                    if half == 0:
                        if in_use("s", sb):
                            raise Hazard("scales of a product")
                        scales[sb][w] = (tile, c)
                    if weights[ws] != (tile, c):
                        raise Hazard("another chunk's weights")
                    hfull[h].arrive()
                    h += 1
                    if h == 2:
                        h, ph_h = 0, ph_h ^ 1
                    yield
                converting[w] = None
                wempty[ws].arrive()
                ws += 1
                if ws == W_STAGES:
                    ws, ph_w = 0, ph_w ^ 1
                sb ^= 1

    def mma():
        a = h = buf = 0
        ph_a, ph_h, ph_t = 0, 0, 1

        def walk():
            nonlocal a, h, buf, ph_a, ph_h, ph_t
            for tile in range(tiles):
                for c in range(n_chunks):
                    if not (yield from waits("afull", afull[a], ph_a)):
                        return False
                    for half in range(2):
                        if 2 * half >= chunks[c]:
                            break
                        if not (yield from waits("hfull", hfull[h], ph_h)):
                            return False
                        for b in range(2 * half, min(2 * half + 2, chunks[c])):
                            if not (yield from waits("tempty", tempty[buf], ph_t)):
                                return False
                            if buf in adding:
                                raise Hazard("columns that are added up")
                            columns[buf] = None
                            queue.append(("mma", {"a": a, "h": h, "s": a, "t": buf}, (tile, c, half, b)))
                            queue.append(("commit", tfull[buf]))
                            buf += 1
                            if buf == 2:
                                buf, ph_t = 0, ph_t ^ 1
                            yield
                        queue.append(("commit", hempty[h]))
                        h += 1
                        if h == 2:
                            h, ph_h = 0, ph_h ^ 1
                    queue.append(("commit", aempty[a]))
                    a += 1
                    if a == 2:
                        a, ph_a = 0, ph_a ^ 1
            return True

        ok = yield from walk()
        if not ok:
            failed.append("mma")
        if fin == "always" or (fin == "own" and not ok):
            queue.append(("commit", end))
            yield from waits_to_the_end(end, 0, lambda: queue)

    def sums(w):
        buf = ph = 0
        for tile in range(tiles):
            for c in range(n_chunks):
                for b in range(chunks[c]):
                    if not (yield from waits("tfull", tfull[buf], ph)):
                        failed.append("sums")
                        return
                    adding[w] = buf
                    for _ in range(1 + rng.randrange(2)):
                        if columns[buf] != (tile, c, b):
                            raise Hazard("another block's columns")
                        yield
                    adding[w] = None
                    summed[w] += 1
                    tempty[buf].arrive()
                    buf += 1
                    if buf == 2:
                        buf, ph = 0, ph ^ 1

    def advance():  # a copy lands, or the oldest product or commit is done
        if copies and (not queue or rng.random() < 0.5):
            memory, stage, chunk, barrier = copies.pop(rng.randrange(len(copies)))
            memory[stage] = chunk
            barrier.arrive()
        elif queue:
            kind, *op = queue.pop(0)
            if kind == "commit":
                op[0].arrive()
                return
            at, (tile, c, half, b) = op
            if acts[at["a"]] != (tile, c) or any(x != (tile, c, half) for x in halves[at["h"]]) or any(x != (tile, c) for x in scales[at["s"]]):
                raise Hazard("another block's operands")
            columns[at["t"]] = (tile, c, b)

    running = [fetcher(), mma()] + [operand(w) for w in range(OPERAND_WARPS)] + [sums(w) for w in range(SUM_WARPS)]
    slow = rng.choice((0.05, 0.3, 0.7))
    for _ in range(200000):
        if not running:
            break
        if rng.random() < slow:
            advance()
        r = rng.choice(running)
        try:
            next(r)
        except StopIteration:
            running.remove(r)
    assert not running
    if copies:
        raise Hazard("a copy into the memory of a block that has ended")
    if any(op[0] == "mma" for op in queue):
        raise Hazard("a product into columns that were given back")
    return bool(failed), summed, tiles * sum(chunks)


@pytest.mark.parametrize("nbs", [1, 2, 3, 4, 7, 12])
def test_rings(nbs):
    for seed in range(100):
        rng = random.Random(100 * nbs + seed)
        failed, summed, blocks = product(rng.randrange(1, 4), nbs, rng.randrange(1, 4), rng, rng.choice((0.0, 0.0, 0.001, 0.01)))
        assert failed or summed == [blocks] * SUM_WARPS


@pytest.mark.parametrize("planted,what", [
    ({"left_out": ("wempty",)}, "weights"), ({"left_out": ("aempty",)}, "activations|operands"), ({"left_out": ("hempty",)}, "FP16|scales|operands"), ({"left_out": ("tempty",)}, "columns"),
    ({"left_out": ("wfull",)}, "weights"), ({"left_out": ("afull",)}, "operands"), ({"left_out": ("hfull",)}, "operands|FP16|scales"), ({"left_out": ("tfull",)}, "columns"),
])
def test_a_missing_wait_is_found(planted, what):
    with pytest.raises(Hazard, match=what):
        for seed in range(300):
            product(2, 7, 2, random.Random(seed), 0.0, **planted)


@pytest.mark.parametrize("planted,what,shape", [  # (segments, blocks of each, tiles): no more chunks than stages; a stage twice
    ({"drain": "own"}, "a copy", (1, 4, 1)), ({"drain": "own"}, "a copy", (2, 7, 1)), ({"drain": "never"}, "a copy", (1, 4, 1)), ({"fin": "own"}, "a product", (1, 4, 1)),
    ({"fin": "own"}, "a product", (2, 3, 1)), ({"fin": "never"}, "a product", (1, 4, 1)), ({"look_back": "three"}, "never issued", (3, 7, 2)),
])
def test_what_is_left_behind_is_found(planted, what, shape):
    with pytest.raises(Hazard, match=what):
        for seed in range(6000):
            product(*shape, random.Random(seed), 0.005, **planted)
