"""A CPU model of grid_begin and grid_barrier (common.cuh) as blocks run them: the phase, bit 31
of the counter, is read once before a block's first arrival and then kept and flipped by the
block itself; an arrival's addition returns nothing. Under random orders no block leaves an
episode before all have arrived at it, and all leave, also when blocks read the phase while
others have arrived already or start from either phase."""
import numpy as np
import pytest

MASK, FLIP = 0xFFFFFFFF, 0x80000000


def _simulate(n, episodes, rng, start=0, mistake=None):
    bar = start
    phase = [None] * n  # None: not begun
    waiting = [False] * n
    ep = [0] * n
    arrived = [0] * episodes
    left = []
    running = list(range(n))
    for _ in range(400 * n * episodes):
        if not running:
            return left
        b = running[int(rng.integers(0, len(running)))]
        if phase[b] is None or (mistake == "read again" and not waiting[b] and rng.random() < 0.5):
            phase[b] = bar & FLIP  # grid_begin
        elif not waiting[b]:
            bar = (bar + (FLIP - (n - 1) if b == 0 else 1)) & MASK
            arrived[ep[b]] += 1
            waiting[b] = True
            if mistake == "read after arriving":
                phase[b] = bar & FLIP
        elif (bar ^ phase[b]) & FLIP:
            left.append(arrived[ep[b]])
            phase[b] ^= FLIP
            waiting[b] = False
            ep[b] += 1
            if ep[b] == episodes:
                running.remove(b)
    raise AssertionError("no progress")


@pytest.mark.parametrize("start", [0, FLIP])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 148])
def test_no_block_leaves_before_all_arrive(n, start):
    rng = np.random.default_rng(n)
    episodes = 3 if n > 100 else 20
    left = _simulate(n, episodes, rng, start)
    assert len(left) == n * episodes and all(count == n for count in left)


def test_reading_the_phase_again_before_an_arrival_changes_nothing():
    # bit 31 cannot flip until the block itself has arrived
    assert all(count == 8 for count in _simulate(8, 10, np.random.default_rng(1), mistake="read again"))


def test_a_phase_read_after_the_arrival_traps_the_last_block():
    with pytest.raises(AssertionError):
        _simulate(4, 6, np.random.default_rng(2), mistake="read after arriving")
