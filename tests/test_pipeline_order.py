"""The barrier protocols of the gathered-row pipelines, restated with a random scheduler that may hold back any
role for any time: a ring of stages, warps that fill them by turns, a thread that issues the MMAs, whose completions
come later but in order per issuing thread.

A parity wait sees only whether the phase before the running one had that parity: a waiter more than one phase off,
on either side, reads the wrong answer.  Two rules keep the waiters within a phase:
 - k_oz_apply (csrc/ozgemm.cu): `empty` has to complete in the order of the chunks.  The issuing thread of a group
   without states frees a stage by a commit, behind its own earlier MMAs, and not by an arrival of its own.
 - k_cheb_umma (csrc/spmm_umma.cu): a stage of a tile's last chunks has slots without one.  Their warps arrive for
   them as for the others; where the copying thread does so in their place, the MMAs can run past a warp that is late,
   and the phase that it waits for is then read as not yet there."""
import random

import pytest


class Barrier:
    def __init__(self, count):
        self.count = self.left = count
        self.phases = 0                                   # completed

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phases = self.count, self.phases + 1

    def test(self, parity):
        return (self.phases & 1) != (parity & 1)


def run(agents, rng):
    """Agents yield a condition to wait for, or None.  True: all ended; False: nobody can go on."""
    waits = {a: None for a in agents}
    speed = {a: rng.choice([1, 1, 5, 40]) for a in agents}
    while waits:
        ready = [a for a, w in waits.items() if w is None or w()]
        if not ready:
            return False
        a = rng.choices(ready, [speed[x] for x in ready])[0]
        if rng.random() < 0.01:
            speed[a] = rng.choice([0.01, 1, 40])
        try:
            waits[a] = next(a)
        except StopIteration:
            del waits[a]
    return True


def completions(queue, last):
    """The tensor pipe behind one issuing thread: commits arrive in order, each after some time."""
    while True:
        yield lambda: queue or last["ended"]
        if not queue:
            return
        queue.pop(0).arrive()


def apply_pipeline(rng, blocks, chunks, commit):
    """k_oz_apply on one CTA: column blocks of `chunks` chunks, the second group absent in some."""
    stages, warps = 5, 4
    full, empty = [Barrier(2) for _ in range(stages)], [Barrier(2) for _ in range(stages)]
    work = [(b, c) for b in range(len(blocks)) for c in range(chunks)]
    landed, early = [0], []

    def copies():
        for q in range(len(work)):
            if q >= stages:
                par = q // stages - 1
                yield lambda s=q % stages: empty[s].test(par)
            full[q % stages].arrive()
            yield

    def gather(w):
        for q in range(w, len(work), warps):
            if q >= stages:
                par = q // stages - 1
                yield lambda s=q % stages: empty[s].test(par)
            if empty[q % stages].phases < q // stages:
                early.append(q)
            yield
            full[q % stages].arrive()

    def waiter():
        for q in range(len(work)):
            yield lambda s=q % stages, p=q // stages: full[s].test(p)
            landed[0] = q + 1

    queues, last = [[], []], [{"ended": False}, {"ended": False}]

    def issue(h):
        for q, (b, _) in enumerate(work):
            yield lambda: landed[0] > q
            if h == 0 or blocks[b] or commit:
                queues[h].append(empty[q % stages])
            else:
                empty[q % stages].arrive()
        last[h]["ended"] = True

    agents = [copies(), waiter()] + [gather(w) for w in range(warps)] + [issue(h) for h in (0, 1)]
    agents += [completions(queues[h], last[h]) for h in (0, 1)]
    return run(agents, rng) and not early


def filter_pipeline(rng, items, stages, sc, warps, own):
    """k_cheb_umma on one CTA: tiles of items[i] chunks, stages of sc chunks."""
    full, done = [Barrier(1 + sc) for _ in range(stages)], [Barrier(1) for _ in range(stages)]
    slots = []                                            # chunk or no chunk, whole stages an item
    for n in items:
        slots += [True] * n + [False] * (-n % sc)
    early, queue, last = [], [], {"ended": False}

    def copies():
        for g in range(len(slots) // sc):
            if g >= stages:
                yield lambda s=g % stages, p=g // stages - 1: done[s].test(p)
            if not own:
                for j in range(sc):
                    if not slots[g * sc + j]:
                        full[g % stages].arrive()
            full[g % stages].arrive()
            yield

    def gather(w):
        for t in range(w, len(slots), warps):
            g = t // sc
            if g >= stages:
                yield lambda s=g % stages, p=g // stages - 1: done[s].test(p)
            if done[g % stages].phases < g // stages:
                early.append(t)
            yield
            if slots[t] or own:
                full[g % stages].arrive()

    def mma():
        for g in range(len(slots) // sc):
            yield lambda s=g % stages, p=g // stages: full[s].test(p)
            queue.append(done[g % stages])
        last["ended"] = True

    agents = [copies(), mma(), completions(queue, last)] + [gather(w) for w in range(warps)]
    return run(agents, rng) and not early


BLOCKS = [[True, False], [True, True, False], [False, True, False, True]]


@pytest.mark.parametrize("blocks", BLOCKS)
def test_absent_group_frees_stages_in_order(blocks):
    assert all(apply_pipeline(random.Random(i), blocks, 23, commit=True) for i in range(150))


def test_absent_group_without_a_commit_is_read_too_early():
    assert not all(apply_pipeline(random.Random(i), b, 23, commit=False) for b in BLOCKS for i in range(150))


# FP32 (two chunks a stage) and BF16 (four) rings; tiles of nine chunks give a warp two empty slots in a row
RINGS = [(5, 2, 10, [9] * 12), (4, 2, 8, [7, 7, 1, 15, 7, 7, 7, 30]), (5, 4, 10, [9, 5, 17, 1, 2, 3, 13, 13, 13])]


@pytest.mark.parametrize("stages, sc, warps, items", RINGS)
def test_empty_slots_are_filled_by_their_warps(stages, sc, warps, items):
    assert all(filter_pipeline(random.Random(i), items, stages, sc, warps, own=True) for i in range(150))


def test_empty_slots_filled_by_the_copies_can_stop_a_late_warp():
    assert not all(filter_pipeline(random.Random(i), r[3], *r[:3], own=False) for r in RINGS for i in range(150))
