"""The exchange of the shared-memory cluster kernel (resident.cuh) when a wait
gives up, restated as a simulation on the CPU.

Every block sends its share of a vector to every other block twice per
iteration with stores that land some time after they are issued and complete
only on the receiver's barrier.  A block waits, with a limit, for all bytes of
a half; a warp that gives up still sends, the block leaves its loop at the end
of that iteration, and all blocks meet at the cluster barrier, which does not
wait for stores under way.  One message never arrives.  No store may land in a
block that has retired: blocks that finished all iterations may retire at the
barrier, blocks that gave up only after the drain."""
import numpy as np
import pytest

BLOCKS, WARPS, ITERS, LIMIT, DELAY = 4, 3, 6, 1000.0, 5.0


def simulate(seed, drain):
    """(latest landing after retirement over all blocks, whether any block gave up)."""
    rng = np.random.default_rng(seed)
    lost = (rng.integers(2), rng.integers(ITERS), rng.integers(BLOCKS), rng.integers(BLOCKS - 1))
    lost = (*lost[:3], lost[3] + (lost[3] >= lost[2]))               # (half, iteration, sender, receiver)
    now = rng.uniform(0, 3, (BLOCKS, WARPS))
    running, ok = np.ones(BLOCKS, bool), np.ones(BLOCKS, bool)
    arrived = [0.0] * BLOCKS                                         # at the cluster barrier
    lands = [[] for _ in range(BLOCKS)]
    complete = np.zeros(BLOCKS)                                      # the phase the next wait is for
    for it in range(ITERS):
        for half in range(2):
            failed = np.zeros(BLOCKS, bool)
            if it > 0 or half == 1:
                for b in np.flatnonzero(running):
                    gave_up = now[b] + LIMIT < complete[b]
                    now[b] = np.where(gave_up, now[b] + LIMIT, np.maximum(now[b], complete[b]))
                    failed[b] = gave_up.any()
            ok &= ~failed
            now += np.where(running[:, None], rng.uniform(0.5, 3, now.shape), 0.0)
            complete = np.where(running, 0.0, np.inf)
            if half == 1 and it == ITERS - 1:
                continue                                             # the last half sends nothing
            for b in range(BLOCKS):
                for r in range(BLOCKS):
                    if r == b:
                        continue
                    if not running[b]:
                        complete[r] = np.inf
                        continue
                    at = now[b] + rng.uniform(0.1, DELAY, WARPS)
                    if (half, it, b, r) == lost:
                        complete[r] = np.inf
                        continue
                    lands[r].extend(at)
                    complete[r] = max(complete[r], at.max())
        for b in np.flatnonzero(running):
            now[b] = now[b].max()                                    # the block barrier
            if not ok[b] or it == ITERS - 1:
                running[b], arrived[b] = False, now[b].max()
    barrier = max(arrived)
    late = [max(lands[b]) - (barrier + (0.0 if ok[b] else drain)) for b in range(BLOCKS)]
    return max(late), bool((~ok).any())


@pytest.mark.parametrize("seed", range(200))
def test_no_store_lands_in_a_retired_block(seed):
    late, _ = simulate(seed, drain=2 * DELAY)
    assert late <= 0.0


def test_the_barrier_alone_is_not_enough():
    runs = [simulate(seed, drain=0.0) for seed in range(200)]
    assert any(late > 0.0 for late, gave_up in runs if gave_up)
