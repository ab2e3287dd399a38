"""The split of small launches (fewer worlds per group, the latency list of
operations) gives the same worlds as groups of 32 in the throughput list."""

import numpy as np
import pytest

from arc_demo_b200.native import KERNEL_WARPS, Sim

pytestmark = pytest.mark.gpu

BIG = 9601  # more than two groups of 32 per SM, the last one partly filled


def _states(n: int, fp64: bool, queue: bool, steps: int = 3):
    rng = np.random.default_rng(5)
    seeds = np.arange(BIG, dtype=np.uint32) * 13 + 3
    diffs = rng.uniform(0.0, 1.0, BIG)
    acts = rng.uniform(-1.0, 1.0, (steps, BIG, 12))
    s = Sim(n, fp64=fp64)
    s.set_kernel(KERNEL_WARPS)
    s.set_work_queue(queue)
    s.reset(np.arange(n), seeds[:n], diffs[:n])
    for k in range(steps):
        s.step(s.default_angles + 0.6 * acts[k, :n])
    out = s.get_state(np.arange(min(n, 4800)))
    s.close()
    return out


@pytest.mark.parametrize("fp64", [False, True])
def test_small_batches_equal_large(fp64):
    # bitwise: a world's arithmetic does not depend on its group or list.
    # 74 groups of 1; 75, 149: groups of 2 and 3, the last partly filled;
    # 2,367-2,369: the split's end; 4,737: the first with a second group on an SM
    whole = _states(BIG, fp64, True)
    for n in (1, 74, 75, 149, 1000, 2367, 2369, 4737):
        for queue in (False, True):
            got = _states(n, fp64, queue)
            assert np.array_equal(got, whole[: len(got)]), (n, queue)
