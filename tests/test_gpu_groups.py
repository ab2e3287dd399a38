"""The split of small launches (fewer worlds per group, the latency list of
operations) gives the same worlds as groups of 32 in the throughput list."""

import ctypes

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


@pytest.mark.parametrize("fp64,n,cell", [
    # three groups per SM; whole waves of four per SM; one world over, split
    # over the SMs; a tail of groups of 32 in the latency list, and one in the
    # other; contact lists at the reference's cap (their own list)
    (False, 14208, 0.4), (False, 18944, 0.4), (False, 18945, 0.4), (False, 26000, 0.4), (False, 33000, 0.4),
    (False, 14300, 0.05), (True, 9472, 0.4), (True, 9473, 0.4), (True, 12001, 0.4), (True, 16384, 0.4)])
def test_aligned_groups_equal_groups_of_their_own(fp64, n, cell):
    # bitwise; without the work queue every group has a CTA of its own
    rng = np.random.default_rng(n)
    seeds, diffs = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32), rng.uniform(0.0, 1.0, n)
    acts = rng.uniform(-1.0, 1.0, (2, n, 12))
    states = []
    for queue in (True, False):
        s = Sim(n, fp64=fp64, cell=cell, grid=32)
        s.set_kernel(KERNEL_WARPS)
        s.set_work_queue(queue)
        s.reset(np.arange(n), seeds, diffs)
        for k in range(2):
            s.step(s.default_angles + 0.6 * acts[k])
        states.append(s.get_state())
        s.close()
    assert np.array_equal(*states)


@pytest.mark.parametrize("fp64", [False, True])
def test_task_rows_do_not_depend_on_the_batch(fp64):
    # the task kernel takes 32 worlds per CTA, four at a time: one world, a
    # partly filled CTA, one world in the last CTA; and the row that a step
    # writes is the row that an observation of the same state gives. Bitwise
    import torch
    from arc_demo_b200.task import TaskConfig
    from arc_demo_b200.torch_env import DeviceVecEnv

    acts = torch.rand((2, 97, 12), generator=torch.Generator().manual_seed(3)).mul_(2).sub_(1).cuda()

    def rows(n):
        env = DeviceVecEnv(n, TaskConfig(curriculum=False, max_steps=2), seed=11, fp64=fp64)
        env.set_levels(np.linspace(0.0, 1.0, 97)[:n])
        env.reset()
        out = []
        for k in range(2):  # every episode ends at the second step
            obs, reward, _, truncated = env.step(acts[k, :n])
            out += [obs.clone(), reward.clone(), truncated.clone()]
            if k == 0:
                env.sim._check(env.gpu.lib.arc_env_observe(env.sim.ptr, None))
                env.sim.synchronize()
                assert torch.equal(env.obs, out[0])
        out.append(env.terminal_obs.clone())
        assert int(env.done_count[0]) == n
        torch.cuda.synchronize()
        env.close()
        return out

    whole = rows(97)
    for n in (1, 31, 32, 33, 65):
        for a, b in zip(rows(n), whole):
            assert torch.equal(a, b[:n])


def leg_contacts(s, i):
    """The most contacts of one tibia in world i's last substep."""
    w = s._lib.arc_sim_world(s.ptr, i).contents
    bodies = [w.contacts[k].body for k in range(w.n_contacts)]
    return max(bodies.count(3 * leg + 3) for leg in range(4))


@pytest.mark.parametrize("fp64", [False, True])
def test_split_groups_equal_whole_groups(fp64):
    # bitwise; recording contacts keeps a leg on one warp. Robots dropped into
    # columns of random heights touch many: some leg's list must outgrow the
    # split group's on-chip records (2), or the spill is not tested
    from oracle.oracle import World

    n, steps = 70, 8
    rng = np.random.default_rng(9)
    acts = rng.uniform(-1.0, 1.0, (steps, n, 12))
    states, longest = [], 0
    for record in (False, True):
        s = Sim(n, fp64=fp64)
        s.set_kernel(KERNEL_WARPS)
        s.reset(np.arange(n), np.arange(n, dtype=np.uint32), np.full(n, 0.5))
        terrain = np.random.default_rng(4)
        for i in range(n):
            s.set_terrain(i, terrain.uniform(-0.3, 0.9, (64, 64)), 0.4)
        s._lib.arc_sim_world.restype = ctypes.POINTER(World)
        s._lib.arc_sim_world.argtypes = [ctypes.c_void_p, ctypes.c_int]
        s._check(s._lib.arc_sim_set_record_contacts(s.ptr, int(record)))
        for k in range(steps):
            s.step(s.default_angles + 0.6 * acts[k])
            if record:
                longest = max([longest] + [leg_contacts(s, i) for i in range(n)])
        states.append(s.get_state())
        s.close()
    assert np.array_equal(*states)
    assert longest > 2


@pytest.mark.parametrize("fp64", [False, True])
def test_both_lists_of_a_split_leg_spill(fp64):
    # bitwise, substep by substep. World i has the femur sphere of leg i % 4 in
    # the corner of a pit: its floor and two walls are three contacts, one more
    # than a split group's upper warps keep on chip, while the leg's tibia,
    # inside the walls' columns, has as many in the same room of the spill
    from oracle.oracle import World

    n, steps, cell = 16, 3, 0.4
    states, femurs, both = [], [0] * 4, [0] * 4
    for record in (False, True):
        s = Sim(n, substeps=1, fp64=fp64, cell=cell)
        s.set_kernel(KERNEL_WARPS)
        s._lib.arc_sim_world.restype = ctypes.POINTER(World)
        s._lib.arc_sim_world.argtypes = [ctypes.c_void_p, ctypes.c_int]
        s.reset(np.arange(n), np.arange(n, dtype=np.uint32), np.zeros(n))
        state = s.get_state()
        for i in range(n):
            leg, sx, sy = i % 4, 1 - 2 * (i // 4 % 2), 1 - 2 * (i // 8)
            w = s._lib.arc_sim_world(s.ptr, i).contents
            ball = w.spheres[5 * leg + 1]
            assert ball.body == 3 * leg + 2
            rot = np.array(w.bodies[ball.body].rot.m).reshape(3, 3)
            at = state[i, 13 * ball.body:][:3] + rot @ [ball.pos.x, ball.pos.y, ball.pos.z]
            # its centre 0.3 radii from the walls at x = 0 and y = 0
            shift = 0.3 * ball.radius * np.array([sx, sy]) - at[:2]
            for b in range(13):
                state[i, 13 * b: 13 * b + 2] += shift
            heights = np.full((64, 64), at[2] + 0.05)
            heights[(slice(32, None) if sy > 0 else slice(None, 32)), (slice(32, None) if sx > 0 else slice(None, 32))] \
                = at[2] - 0.8 * ball.radius
            s.set_terrain(i, heights, cell)
        s.set_state(state)
        s._check(s._lib.arc_sim_set_record_contacts(s.ptr, int(record)))
        for _ in range(steps):
            s.step(np.tile(s.default_angles, (n, 1)))
            states.append((record, s.get_state()))
            for i in range(n if record else 0):
                w = s._lib.arc_sim_world(s.ptr, i).contents
                bodies = [w.contacts[k].body for k in range(w.n_contacts)]
                for leg in range(4):
                    upper, lower = bodies.count(3 * leg + 2), bodies.count(3 * leg + 3)
                    femurs[leg], both[leg] = max(femurs[leg], upper), max(both[leg], min(upper, lower))
        s.close()
    for a, b in zip((x for r, x in states if not r), (x for r, x in states if r)):
        assert np.array_equal(a, b)
    assert min(femurs) > 2 and min(both) > 2, (femurs, both)
