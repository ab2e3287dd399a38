"""The task state's rows as the device gathers them, and a step's results."""

import numpy as np
import pytest

from arc_demo_b200.task import CAUSE, REWARD, TASK_STATE_SIZE, TERMINATED, TRUNCATED, ArcTask, TaskConfig

pytestmark = pytest.mark.gpu


# one world, a partly filled CTA of eight, copies below and above 256 KB
@pytest.mark.parametrize("n", [1, 9, 1400])
def test_rows_and_results(n):
    t = ArcTask(n, TaskConfig(curriculum=False, max_steps=2), seed=3)
    t.reset(np.arange(n))
    rng = np.random.default_rng(n)
    rows = rng.integers(0, 1000, (n, TASK_STATE_SIZE)).astype(np.float64)  # whole numbers: exact in every type
    rows[:, 22] = rng.integers(0, 2, n)
    t.gpu.set_state(rows)
    assert np.array_equal(t.gpu.get_state(), rows)
    ids = rng.permutation(n)[: n // 2 + 1]
    assert np.array_equal(t.gpu.get_state(ids), rows[ids])
    assert t.gpu.get_state(np.zeros(0, dtype=np.int32)).shape == (0, TASK_STATE_SIZE)
    t.reset(np.arange(n))
    for _ in range(2):  # every episode ends at the second step
        t.step(rng.uniform(-1.0, 1.0, (n, 12)).astype(np.float32))
        st, *rest = t.gpu.results()
        assert np.array_equal(st, t.gpu.get_state())
        for got, which in zip(rest, (REWARD, TERMINATED, TRUNCATED, CAUSE)):
            want = t.gpu.download(which)
            assert got.dtype == want.dtype and np.array_equal(got, want)
    assert rest[2].all() or rest[1].any()
    t.close()
