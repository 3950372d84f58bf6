"""CPU model of conv32_ys_kernel's protocol (csrc/cnn.cu; no GPU): the ring of row
sets, the barriers' counts and parities, and the accumulator cycle -- eight slots of
each plane, a window of three that moves on by one a step and jumps back every
sixth, rows whose sum lies in two slots.

An event simulation with random interleavings: a producer, two MMA issuers whose MMAs
and commits take effect later and in order, and sixteen epilogue warps.  Checked are
that every MMA finds its row set in the ring, that every stored output row holds
exactly its three steps' terms when it is read, that no barrier counts past a phase,
and that every role ends.
"""
import random

import pytest

Y_R, Y_NT, Y_ROWS = 4, 2, 8


class Barrier:
    def __init__(self, count):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        assert self.left >= 0
        if self.left == 0:
            self.phase += 1
            self.left = self.count

    def passed(self, parity):   # mbarrier.try_wait.parity
        return (self.phase & 1) != parity


def run(items, planes, seed, lag=6):
    """items: the row counts of one CTA's runs; planes: issuers with MMAs; step T
    waits for row T - lag to have been read."""
    rng = random.Random(seed)
    full = [Barrier(1) for _ in range(Y_R)]
    empty = [Barrier(2) for _ in range(Y_R)]
    accf = [Barrier(2) for _ in range(Y_ROWS)]
    acce = [Barrier(8) for _ in range(Y_ROWS)]
    ring = [None] * Y_R
    slots = [[None] * 8 for _ in range(2)]
    queues = [[], []]           # each issuer's MMAs and commits, in order
    stored = []

    def producer():
        T = 0
        for ly in items:
            for _ in range(ly + 2):
                s = T % Y_R
                if T >= Y_R:
                    yield lambda s=s, T=T: empty[s].passed((T // Y_R - 1) & 1)
                ring[s] = None      # the copy is under way
                yield lambda: rng.random() < 0.5
                ring[s] = T
                full[s].arrive()
                T += 1

    def issuer(p):
        T = w = 0
        q = queues[p]

        def step(T, w, s):
            def go():
                assert ring[s] == T, "row set gone"
                for k, dy in ((0, 2), (1, 1), (2, 0)):
                    if w == 0 or k == 2:
                        slots[p][w + k] = [(T, dy)]
                    else:
                        slots[p][w + k] = slots[p][w + k] + [(T, dy)]
            return go

        for ly in items:
            for _ in range(ly + 2):
                s = T % Y_R
                if T >= lag:
                    yield lambda T=T: acce[(T - lag) % Y_ROWS].passed(((T - lag) // Y_ROWS) & 1)
                yield lambda s=s, T=T: full[s].passed((T // Y_R) & 1)
                if p < planes:
                    q.append(step(T, w, s))
                q.append(empty[s].arrive)
                if T >= 2:
                    q.append(accf[(T - 2) % Y_ROWS].arrive)
                w = (w + 1) % 6
                T += 1
        for r in range(max(T - 2, 0), T):
            q.append(accf[r % Y_ROWS].arrive)

    def epilogue(warp):
        p, tset = (warp >> 2) & 1, warp >> 3
        T = w = 0
        for n, ly in enumerate(items):
            for i in range(ly + 2):
                wt, t = w, T
                w = (w + 1) % 6
                T += 1
                if t % Y_NT != tset:
                    continue
                yield lambda t=t: accf[t % Y_ROWS].passed((t // Y_ROWS) & 1)
                if i < ly and p < planes:
                    got = list(slots[p][wt + 2])
                    if wt >= 4:
                        got += slots[p][wt - 4]
                    assert sorted(got) == [(t, 0), (t + 1, 1), (t + 2, 2)], (t, got)
                    stored.append((warp, n, i))
                acce[t % Y_ROWS].arrive()

    def tensor(p, steps):       # drains issuer p's queue
        for _ in range(steps):
            yield lambda: len(queues[p]) > 0
            queues[p].pop(0)()

    total = sum(ly + 2 for ly in items)
    roles = [producer()] + [issuer(p) for p in range(2)] + [epilogue(w) for w in range(16)]
    roles += [tensor(p, total * (3 if p < planes else 2)) for p in range(2)]
    waiting = [(g, next(g, None)) for g in roles]
    waiting = [(g, c) for g, c in waiting if c is not None]
    idle = 0
    while waiting:
        k = rng.randrange(len(waiting))
        g, cond = waiting[k]
        if not cond():
            idle += 1
            assert idle < 20000, "no role can go on"
            continue
        idle = 0
        nxt = next(g, None)
        if nxt is None:
            waiting.pop(k)
        else:
            waiting[k] = (g, nxt)
    rows = sum(items)
    assert len(stored) == len(set(stored)) == 4 * planes * rows  # four warps a row and plane
    for b in full + empty:
        assert b.left == b.count


@pytest.mark.parametrize("planes", [2, 1])
@pytest.mark.parametrize("items", [[1], [2, 1], [1] * 7, [4, 4, 3], [23], [6, 5, 4, 3, 2, 1],
                                   [32, 9, 17]], ids=str)
def test_accumulator_cycle(items, planes):
    for seed in range(6):
        run(items, planes, seed)


def test_a_slot_reused_a_step_early_is_found():
    with pytest.raises(AssertionError):
        for seed in range(50):
            run([23], 2, seed, lag=7)
