"""The cooperative reset at the edges of its cell blocks (16, 32 and 64
columns wide, 4 and 8 rows) and of its RNG slices: terrain bitwise equal to
the oracle's generator, poses equal to the oracle's reset."""

import numpy as np
import pytest

from arc_demo_b200.native import Sim
from oracle.oracle import OracleSim, oracle_terrain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [1, 2, 7, 8, 15, 16, 17, 31, 32, 33, 47, 63, 64])
def test_terrain_bitwise(grid):
    diffs = np.array([0.0, 0.02, 0.5, 1.0])
    seeds = np.array([0, 1, 0x80000001, 0xFFFFFFFF], dtype=np.uint32)
    s = Sim(len(seeds), fp64=True, grids=np.full(len(seeds), grid))
    f = Sim(len(seeds), grids=np.full(len(seeds), grid))
    for sim in (s, f):
        sim.reset(np.arange(len(seeds)), seeds, diffs)
    for i in range(len(seeds)):
        want, _ = oracle_terrain(grid, 0.4, diffs[i], int(seeds[i]))
        assert np.array_equal(s.get_terrain(i)[0], want)
        assert np.array_equal(f.get_terrain(i)[0], want.astype(np.float32).astype(np.float64))
    s.close()
    f.close()


@pytest.mark.parametrize("n", [1, 2, 1185])
def test_poses(n):
    # 1,185: more worlds than resident CTAs, so a CTA resets several in turn.
    # The bound: the oracle's libm and the GPU's differ by a few FP64 ulps
    rng = np.random.default_rng(n)
    seeds = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    diffs = rng.uniform(0.0, 1.0, n)
    s, o = Sim(n, fp64=True, grid=24), OracleSim(n, grid=24)
    for sim in (s, o):
        sim.reset(np.arange(n), seeds, diffs)
    assert np.abs(s.get_state() - o.get_state()).max() <= 1e-12
    s.close()
