"""Task rows at the edge of a page-locked copy, more of them than the sim has
worlds, and read by several threads."""

import threading

import numpy as np
import pytest

from arc_demo_b200.task import OBS, REWARD, TASK_STATE_SIZE, ArcTask, TaskConfig

pytestmark = pytest.mark.gpu


# the results of 1,266 worlds are the most that one page-locked copy holds
@pytest.mark.parametrize("n", [1266, 1267, 2600])
def test_rows_beyond_a_small_copy(n):
    t = ArcTask(n, TaskConfig(curriculum=False), seed=3)
    rows = np.random.default_rng(n).integers(0, 1000, (n, TASK_STATE_SIZE)).astype(np.float64)
    rows[:, 22] = np.arange(n) % 2
    t.gpu.set_state(rows)
    reward = np.random.default_rng(1).normal(size=n).astype(np.float32)
    t.gpu.upload(REWARD, reward)
    assert np.array_equal(t.gpu.get_state(), rows)
    ids = np.random.default_rng(2).integers(0, n, n + 5)  # some twice; more than the staging's rows
    assert np.array_equal(t.gpu.get_state(ids), rows[ids])
    got = t.gpu.results()
    assert np.array_equal(got[0], rows) and np.array_equal(got[1], reward)
    t.close()


def test_two_threads():
    t = ArcTask(200, TaskConfig(curriculum=False), seed=3)
    t.reset(np.arange(200))
    calls = [lambda: t.gpu.download(OBS), lambda: t.gpu.get_state(), lambda: t.gpu.get_state(np.arange(7)),
             lambda: t.gpu.results()[0]]
    want = [c() for c in calls]
    wrong = []

    def read(k):
        for _ in range(200):
            if not np.array_equal(calls[k](), want[k]):
                wrong.append(k)
    threads = [threading.Thread(target=read, args=(k,)) for k in range(len(calls))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
    t.close()
