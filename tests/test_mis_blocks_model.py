"""A CPU model of mis_kernel's blocks under random interleavings: each goes through its own
undecided vertices pass after pass, with no round and no barrier between blocks, and ends
with the oracle's set (the greedy MIS in descending (priority, id) order).

Modelled at the level that matters for correctness: a vertex keeps the position of the first
outranking neighbour that is not out, and who that is; scans and pushes that are too long for a
thread go to the block's warps, longer ones to the block, a part a pass, and wait for the next
pass where a list is full; a joiner's push may so come passes after it joined, with other blocks
joining between its parts; a block reads states as they were when it last looked (L1) or as
they are, which of the two at random for every read. No GPU is involved."""
import numpy as np
import pytest

import oracle
from test_batch_sssp_model import _random_graph

UNDECIDED, IN, OUT = 0, 1, 2
THREAD, WARP, PART = 2, 4, 3  # entries a thread and a warp scan, entries of a block's part
LONG, HUGE, TILE = 2, 1, 2    # room in the lists; vertices of a tile


class _Block:
    def __init__(self, model, vertices):
        self.m = model
        self.lists = [[], [(v, None, None) for v in vertices]]  # to go through next: lists[1]
        self.view = model.state.copy()

    def read(self, v):
        """A state from L1, which may hold an older one, or from memory."""
        if self.m.rng.random() < 0.5:
            self.view[v] = self.m.state[v]
        return self.view[v]

    def scan(self, v, e, lim, first=False):
        """(stop, state there) of the entries [e, lim), or None."""
        for k in range(e, lim):
            u = self.m.ci[k]
            if u != v and self.m.outranks(u, v):
                s = UNDECIDED if first else self.read(u)
                if s == UNDECIDED and self.m.mistake == "an undecided neighbour is passed by":
                    continue
                if s != OUT:
                    return k, s
        return None

    def push(self, v, e, lim):
        for k in range(e, lim):
            u = self.m.ci[k]
            if u != v and self.read(u) == UNDECIDED:
                yield
                self.m.state[u] = OUT

    def passes(self):
        """Steps of the block until nothing is left."""
        m, rp = self.m, self.m.rp
        first = True
        while self.lists[1]:
            now, nxt = self.lists[1], []
            self.view = m.state.copy()  # the acquire at the end of a pass
            long_, huge = [], []

            def keep(v, pos, by):
                nxt.append((v, pos, by))

            def hand_on(v, pos, item):
                if len(long_) < LONG:
                    long_.append((v, item))
                    return True
                keep(v, pos, -1)
                return False

            def to_block(v, item, by):
                if len(huge) < HUGE:
                    huge.append((v, item))
                else:
                    keep(v, item, by)

            for i in m.rng.permutation(len(now)):
                v, pos, by = now[i]
                yield
                if by == v:  # a push that goes on
                    to_block(v, pos, v)
                    continue
                r1 = rp[v + 1]
                if first:
                    e = rp[v]
                else:
                    if self.read(v) == OUT:
                        continue
                    s = OUT if by < 0 else self.read(by)
                    if s == UNDECIDED and m.mistake != "an undecided neighbour is passed by":
                        keep(v, pos, by)
                        continue
                    if s == IN:
                        m.state[v] = OUT
                        continue
                    e = pos + 1
                lim = min(r1, e + THREAD)
                stop = self.scan(v, e, lim, first)
                yield
                if stop is not None:
                    if stop[1] == IN:
                        m.state[v] = OUT
                    else:
                        keep(v, stop[0], m.ci[stop[0]])
                elif lim < r1:
                    hand_on(v, lim - 1, lim - 1)
                elif r1 - rp[v] > THREAD:
                    if hand_on(v, r1 - 1, "push"):
                        m.state[v] = IN
                else:
                    m.state[v] = IN
                    yield from self.push(v, rp[v], r1)
            for v, item in long_:
                yield
                r0, r1 = rp[v], rp[v + 1]
                if item == "push":
                    if r1 - r0 > WARP:
                        to_block(v, -2 - r0, v)
                    else:
                        yield from self.push(v, r0, r1)
                    continue
                e = item + 1
                lim = min(r1, e + WARP)
                stop = self.scan(v, e, lim)
                if stop is not None:
                    if stop[1] == IN:
                        m.state[v] = OUT
                    else:
                        keep(v, stop[0], m.ci[stop[0]])
                elif lim >= r1:
                    keep(v, r1 - 1, -1)
                else:
                    to_block(v, lim - 1, -1)
            for v, item in huge:
                yield
                r1 = rp[v + 1]
                if item < -1:
                    e = -2 - item
                    lim = min(r1, e + PART)
                    yield from self.push(v, e, lim)
                    if lim < r1:
                        keep(v, -2 - lim, v)
                    continue
                e = item + 1
                lim = min(r1, e + PART)
                stop = self.scan(v, e, lim)
                if stop is None:
                    keep(v, lim - 1, -1)
                else:
                    keep(v, stop[0], m.ci[stop[0]])
            self.lists[1] = nxt
            first = False


class _Model:
    def __init__(self, rp, ci, prio, rng, mistake=None):
        self.rp, self.ci, self.prio = [int(x) for x in rp], [int(x) for x in ci], [int(x) for x in prio]
        self.rng, self.mistake = rng, mistake
        self.state = np.full(len(self.prio), UNDECIDED)

    def outranks(self, u, v):
        return (self.prio[u], u) > (self.prio[v], v)

    def run(self, blocks):
        n = len(self.prio)
        tiles = range(0, n, TILE)
        running = [_Block(self, [v for t in tiles[b::blocks] for v in range(t, min(n, t + TILE))]).passes()
                   for b in range(blocks)]
        for _ in range(400000):
            if not running:
                return self.state
            b = int(self.rng.integers(0, len(running)))
            for _ in range(int(self.rng.integers(1, 12))):  # a block may run ahead of the others
                if next(running[b], "end") == "end":
                    running.pop(b)
                    break
        raise AssertionError("no progress")


@pytest.mark.parametrize("seed", range(40))
def test_every_schedule_gives_the_greedy_set(seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 40))
    rp, ci = _random_graph(rng, n, int(rng.integers(0, 7)))[:2]
    prio = rng.integers(0, 1 + int(rng.integers(1, 50)), n).astype(np.uint32)  # ties among them
    state = _Model(rp, ci, prio, rng).run(int(rng.integers(1, 6)))
    np.testing.assert_array_equal(state == IN, oracle.mis_greedy(rp, ci, prio).astype(bool))
    assert (state != UNDECIDED).all()


def test_a_planted_mistake_is_found():
    wrong = 0
    for seed in range(30):
        rng = np.random.default_rng(seed)
        rp, ci = _random_graph(rng, 25, 4)[:2]
        prio = rng.integers(0, 1000, 25).astype(np.uint32)
        try:
            state = _Model(rp, ci, prio, rng, "an undecided neighbour is passed by").run(3)
        except AssertionError:
            wrong += 1
            continue
        wrong += not np.array_equal(state == IN, oracle.mis_greedy(rp, ci, prio).astype(bool))
    assert wrong > 0
