#!/usr/bin/env python
"""Throughput of the B200 batched world step (arc-demo's quadruped task).

Workload (the configuration the headline metric is quoted on): 65,536
worlds of the quadruped, terrain difficulty uniform in {0, 0.1, ..., 1.0}
per world, seeded synthetic terrain from the reference's generator,
checkpoints drawn as the reference draws them, auto-reset on termination or
after 1,000 steps, actions from a random-init MLP policy (195 -> 256 -> 256
-> 12, tanh, FP32) that reads the observations in place. One step = one
control step (20 XPBD substeps of 1/600 s) of every world: actuation,
physics, rewards, terminations, checkpoints, curriculum bookkeeping,
observations, resets; plus the policy forward that produces its actions.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Prints one JSON line (rank 0). `value` is device-resident throughput: either
the policy, then the step as one CUDA graph of the library's kernels, or the
worlds in 2, 4 or 8 ranges on their own streams, each range's policy then its
step (DeviceVecEnv.step_parts), whichever a short timing picks; `e2e` is the
same loop through the host-buffer API (actions copied
in, observations/rewards/dones copied out every step). `--impl reference`
times the reference's own CPU path (its csrc/ built by oracle/Makefile, run
with OpenMP on every host core) plus the task layer, over all the worlds.
"""

from __future__ import annotations

import argparse
import ctypes
import json
import os
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "env-steps/s at 65536 worlds vs plain GPU kernel and OpenMP; p50/p99 step lat"
WORLDS = 65536
FLOP_PER_ENV_STEP = 415.6e3   # scalar FP ops of one control step, counted on the reference
HBM_BYTES_PER_ENV_STEP = 3.9e3  # algorithmic HBM traffic of one env-step (state, actions, obs)
LAT_STEPS = 300  # control steps of the step-latency sample
# DRAM bytes (read + write) one world costs a launch of the warp-per-leg step
# kernel: ncu's dram__bytes_read.sum + dram__bytes_write.sum over a
# 16,384-world launch (42.24 MB + 0.00 MB), divided by the worlds; each world
# reads its own record and terrain cells, so the traffic scales with them.
WARPS_DRAM_BYTES_PER_WORLD = (42.242e6 + 192.0) / 16384

# the renderer's workload: frames of the reference's rgb_array size
# (arc/env.py:43), 4 rays per pixel, for a batch of worlds per launch
RENDER_METRIC = "frames/s at 640x360, 4 samples per pixel"
RENDER_WORLDS = 256
RENDER_W, RENDER_H, RENDER_SAMPLES = 640, 360, 4
# Work and DRAM traffic of k_render per frame of this workload, from one ncu
# capture of a 16-frame launch: 683.1 M warp instructions, 1.65 MB read +
# 61.00 MB written, over 16 frames. The kernel is bound by instruction issue
# (4 warp instructions per SM per cycle).
RENDER_WARP_INST_PER_FRAME = 683.050e6 / 16
RENDER_DRAM_BYTES_PER_FRAME = (1.6502e6 + 60.9956e6) / 16


def parse():
    p = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=300)
    p.add_argument("--warmup", type=int, default=5)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--worlds", type=int, default=WORLDS)
    p.add_argument("--cpu-seconds", type=float, default=12.0, help="CPU baseline sample length (all worlds)")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--wpc", type=int, default=0, help="worlds per CTA (0: autotune)")
    p.add_argument("--no-plain", action="store_true")
    p.add_argument("--kernel", choices=["auto", "warps"], default="auto")
    p.add_argument("--parts", type=int, default=0,
                   help="policy + step in this many world ranges on their own streams (0: autotune over 1, 2, 4, 8)")
    p.add_argument("--workload", choices=["step", "render"], default="step",
                   help="step: the world step (the headline); render: frames of the headless renderer")
    p.add_argument("--render-worlds", type=int, default=RENDER_WORLDS)
    p.add_argument("--no-workloads", action="store_true",
                   help="skip the other workloads' short legs (uneven OU batch, grid sizes, FP64, serving)")
    return p.parse_args()


def levels_for(n: int, seed: int) -> np.ndarray:
    """Difficulty uniform in {0, 0.1, ..., 1.0} per world."""
    return np.random.default_rng(seed).integers(0, 11, n) / 10.0


# ---------------------------------------------------------------------------
# clocks during the timed region

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=self.file, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        # nvidia-smi needs a moment before its first sample: start timing
        # only once it samples, so that the window is covered
        deadline = time.time() + 3.0
        while self.proc and self.proc.poll() is None and time.time() < deadline:
            self.file.flush()
            if Path(self.file.name).stat().st_size > 0:
                break
            time.sleep(0.02)
        self.skip = sum(1 for _ in open(self.file.name))
        return self

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        self.file.flush()
        rows = []
        for line in Path(self.file.name).read_text().splitlines()[self.skip:]:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        os.unlink(self.file.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}

        def num(x):
            try:
                return float(x)
            except ValueError:
                return None
        sm = [num(r[1]) for r in rows if num(r[1])]
        loaded = [v for v, r in zip(sm, rows) if (num(r[3]) or 0) > 300] or sm
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        reasons = sorted({n for r in rows for n, v in zip(names, r[5:9]) if v.strip().lower() == "active"})
        return {"sm_mhz": float(np.median(loaded)) if loaded else None,
                "sm_max_mhz": num(rows[0][2]), "reasons": reasons, "samples": len(rows)}


# ---------------------------------------------------------------------------
# our arm

def make_policy(torch, seed: int):
    """Random-init MLP 195-256-256-12 (torch.nn.Linear's uniform init): the
    weights are kept transposed (in x out) and the hidden activations in
    buffers reused every step."""
    g = torch.Generator(device="cpu").manual_seed(seed)

    def lin(i, o):
        bound = 1.0 / np.sqrt(i)
        w = (torch.rand(o, i, generator=g) * 2 - 1) * bound
        b = (torch.rand(o, generator=g) * 2 - 1) * bound
        return w.t().contiguous().cuda(), b.cuda().contiguous()
    return {"layers": [lin(195, 256), lin(256, 256), lin(256, 12)], "hidden": {}}


def policy_forward(torch, params, obs, out):
    """MLP 195-256-256-12 with tanh, FP32; writes the actions into `out`."""
    (w1, b1), (w2, b2), (w3, b3) = params["layers"]
    n = obs.shape[0]
    h = params["hidden"].get(n)
    if h is None:
        h = params["hidden"][n] = (torch.empty(n, 256, device=obs.device), torch.empty(n, 256, device=obs.device))
    # x @ W, then + b in place: the same numbers as addmm, without the
    # separate bias kernel cuBLAS adds to its FP32 (non-tensor) GEMMs
    torch.mm(obs, w1, out=h[0]).add_(b1).tanh_()
    torch.mm(h[0], w2, out=h[1]).add_(b2).tanh_()
    torch.mm(h[1], w3, out=out).add_(b3)


def apply_candidate(env, cand):
    """Puts the env's step kernel in the form a candidate names: "warps" (one
    CTA per group of 32 worlds), "warps+queue" (one wave of resident CTAs
    taking groups from a work queue), "tileK" (warps+queue, K substeps per
    launch) or an int (the leg-parallel kernel at that many worlds per CTA)."""
    from arc_demo_b200.native import KERNEL_LEGS, KERNEL_WARPS
    c = str(cand)
    env.sim.set_substep_tile(int(c[4:]) if c.startswith("tile") else 0)
    env.sim.set_work_queue(c == "warps+queue" or c.startswith("tile"))
    if c.startswith("warps") or c.startswith("tile"):
        env.set_kernel(KERNEL_WARPS)
    else:
        env.set_kernel(KERNEL_LEGS, int(c))


def autotune(env, torch, stream,
             candidates=("warps", "warps+queue", "tile10", "tile5", "tile2", 1, 2, 4, 8, 16), steps=4):
    """Step kernel, worlds per CTA and substep tiling, by timing the step
    kernel: the warp-per-leg kernel (32 worlds per CTA; one CTA per group, or
    one wave of resident CTAs taking groups from a work queue; the whole
    control step in one launch, or in launches of 10, 5 or 2 substeps with
    the state through device memory in between) and the leg-parallel kernel
    at 1, 2, 4, 8 and 16 worlds per CTA. Every candidate starts from the same
    world states: the step's cost grows over the first steps after a reset,
    as the robots settle and their contacts multiply, so timing the
    candidates one after another from a running state would favour the
    first."""
    lib, ptr = env.sim._lib, env.sim.ptr
    best, table = None, {}
    stream.synchronize()
    start = env.sim.get_state()
    for cand in candidates:
        env.sim.set_state(start)
        torch.cuda.synchronize()
        apply_candidate(env, cand)
        a = ctypes.c_void_p(env.actions.data_ptr())
        st = ctypes.c_void_p(stream.cuda_stream)
        for _ in range(2):
            lib.arc_sim_step_actions(ptr, a, st)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(steps):
            lib.arc_sim_step_actions(ptr, a, st)
        e1.record(stream)
        e1.synchronize()
        ms = e0.elapsed_time(e1) / steps
        table[str(cand)] = round(ms, 4)
        if best is None or ms < table[str(best)]:
            best = cand
    env.sim.set_state(start)
    torch.cuda.synchronize()
    apply_candidate(env, best)
    return best, table


FORMS = {0: "step kernel, then task and reset kernels",
         1: "step and task layer fused per group of 32 worlds, then the reset kernel",
         2: "step, task layer and resets fused: one launch per control step"}


def autotune_parts(env, torch, stream, one_step,
                   candidates=((1, 0), (1, 1), (1, 2), (2, 0), (2, 1), (4, 0), (4, 1), (8, 0)), steps=6):
    """How the control step runs, by timing whole control steps (policy
    included), each candidate from the same world and task states: (ranges,
    form). Ranges 1: the policy, then env.step() as one CUDA graph; 2, 4, 8: the
    worlds in that many ranges on their own streams (DeviceVecEnv.step_parts),
    each range's policy then its step. Forms (DeviceVecEnv.set_fused): 0 the
    step kernel, then the task and reset kernels; 1 the step and the task
    layer fused per group of 32 worlds, then the reset kernel; 2 the
    resets fused too."""
    table = {}
    stream.synchronize()
    start, tstart = env.sim.get_state(), env.gpu.get_state()
    for parts, form in candidates:
        env.set_fused(form)
        env.sim.set_state(start)
        env.gpu.set_state(tstart)
        torch.cuda.synchronize()
        for _ in range(2):
            one_step(parts)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(steps):
            one_step(parts)
        e1.record(stream)
        e1.synchronize()
        table[f"{parts} ranges, form {form}"] = round(e0.elapsed_time(e1) / steps, 4)
    env.sim.set_state(start)
    env.gpu.set_state(tstart)
    torch.cuda.synchronize()
    parts, form = min(candidates, key=lambda c: table[f"{c[0]} ranges, form {c[1]}"])
    env.set_fused(form)
    return parts, form, table


def max_over_ranks(torch, dist, x: float) -> float:
    """The largest x over all ranks, on every rank (x itself without a
    process group): multi-GPU times are the slowest rank's."""
    if dist is None:
        return x
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([float(x)], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_rate(world: int, worlds_per_rank: int, steps: int, ms: float) -> float:
    """env-steps/s of the whole job: every rank's worlds over the slowest
    rank's time (weak scaling: each rank owns worlds_per_rank worlds)."""
    return world * worlds_per_rank * steps / (ms * 1e-3)


def run_ours(args) -> dict | None:
    import torch
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    torch.backends.cuda.matmul.allow_tf32 = False
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))

    from arc_demo_b200.native import KERNEL_LEGS, KERNEL_PLAIN, KERNEL_WARPS, sim_lib
    from arc_demo_b200.task import TaskConfig
    from arc_demo_b200.torch_env import DeviceVecEnv

    n = args.worlds
    cfg = TaskConfig(curriculum=False)
    env = DeviceVecEnv(n, cfg, seed=1000 + rank)
    env.set_levels(levels_for(n, 17 + rank))
    stream = torch.cuda.Stream()
    params = make_policy(torch, 1234)
    with torch.cuda.stream(stream):
        env.reset()
        torch.nn.init.uniform_(env.actions, -1.0, 1.0)
        if args.wpc:
            env.set_kernel(KERNEL_LEGS, args.wpc)
            best_wpc, tune = args.wpc, None
        elif args.kernel == "warps":
            apply_candidate(env, "warps+queue")
            best_wpc, tune = "warps+queue", None
        else:
            best_wpc, tune = autotune(env, torch, stream)
        part_params = [{"layers": params["layers"], "hidden": {}} for _ in range(16)]  # one set per stream

        def part_policy(p, obs, actions):
            policy_forward(torch, part_params[p], obs, actions)

        def one_step(parts=1):
            if parts == 1:
                policy_forward(torch, params, env.obs, env.actions)
                env.step()
            else:
                env.step_parts(part_policy, parts)

        if args.parts:
            parts, form, parts_tune = args.parts, 0, None
            env.set_fused(0)
        else:
            parts, form, parts_tune = autotune_parts(env, torch, stream, one_step)
        env.reset()

        for _ in range(max(args.warmup, 3)):
            one_step(parts)
        stream.synchronize()
        if dist:
            dist.barrier()
        K = args.steps
        starts = [torch.cuda.Event(enable_timing=True) for _ in range(K)]
        ends = [torch.cuda.Event(enable_timing=True) for _ in range(K)]
        with ClockSampler(local) as clocks:
            torch.cuda.synchronize()
            t0 = torch.cuda.Event(enable_timing=True)
            t1 = torch.cuda.Event(enable_timing=True)
            t0.record(stream)
            for k in range(K):
                starts[k].record(stream)
                one_step(parts)
                ends[k].record(stream)
            t1.record(stream)
            t1.synchronize()
            torch.cuda.synchronize()
            ended = int(env.done_count.item())
            # step latency from a longer sample than the timed steps (a p99 of
            # 20 samples is their maximum): LAT_STEPS control steps, each
            # between CUDA events, right after the timed region; the clock
            # samples cover both, the same load
            lat_ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                      for _ in range(LAT_STEPS)]
            for s0, s1 in lat_ev:
                s0.record(stream)
                one_step(parts)
                s1.record(stream)
            stream.synchronize()
        if dist:
            dist.barrier()
        ms_total = max_over_ranks(torch, dist, t0.elapsed_time(t1))
        lat = np.array([s.elapsed_time(e) for s, e in zip(starts, ends)])
        clock = clocks.summary()
        clock["window"] = f"the {K} timed control steps and the {LAT_STEPS}-step latency sample after them"
        lat_long = np.array([s0.elapsed_time(s1) for s0, s1 in lat_ev])

        # the dominant kernel alone: the leg-parallel step, same stream
        lib, ptr = env.sim._lib, env.sim.ptr
        a = ctypes.c_void_p(env.actions.data_ptr())
        st = ctypes.c_void_p(stream.cuda_stream)
        # the worlds in the order the env's step hands them to the kernels
        # (by difficulty band, hardest first), which both kernels are timed in
        order = torch.from_numpy(env.step_order()).to("cuda")
        ids = ctypes.c_void_p(order.data_ptr())

        def step_kernel():
            if env.sim.kernel()[0] in (KERNEL_WARPS, KERNEL_PLAIN):
                lib.arc_sim_step_ids(ptr, ids, n, None, a, st)
            else:  # the leg-parallel kernel steps whole batches, in index order
                lib.arc_sim_step_actions(ptr, a, st)
        M = 10
        k0, k1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        k0.record(stream)
        for _ in range(M):
            step_kernel()
        k1.record(stream)
        k1.synchronize()
        step_kernel_ms = k0.elapsed_time(k1) / M

        # the plain per-world kernel on the same loop (the baseline form)
        plain = None
        if rank == 0 and not args.no_plain:
            # the baseline in whichever step order suits it better (by
            # difficulty band, as ours, or world index)
            env.set_kernel(KERNEL_PLAIN)
            Kp = max(3, min(10, K))
            plain_ms, plain_kernel_ms, plain_order = None, None, None
            for order_mode in (1, 0):
                env.set_step_order(order_mode)
                for _ in range(2):
                    one_step()
                p0, p1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                p0.record(stream)
                for _ in range(Kp):
                    one_step()
                p1.record(stream)
                p1.synchronize()
                ms = p0.elapsed_time(p1) / Kp
                q0, q1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                q0.record(stream)
                for _ in range(3):
                    if order_mode:
                        step_kernel()
                    else:
                        lib.arc_sim_step_actions(ptr, a, st)
                q1.record(stream)
                q1.synchronize()
                kms = q0.elapsed_time(q1) / 3
                if plain_ms is None or ms < plain_ms:
                    plain_ms, plain_order = ms, ("by difficulty band" if order_mode else "world index")
                plain_kernel_ms = kms if plain_kernel_ms is None else min(plain_kernel_ms, kms)
            env.set_step_order(1)
            plain = {"ms_per_step": round(plain_ms, 3), "env_steps_per_s": round(n / plain_ms * 1e3),
                     "step_kernel_ms": round(plain_kernel_ms, 3), "step_order": plain_order,
                     "loop": "the same policy and env.step() graph with the plain per-world kernel (one thread "
                             "per world) and the separate task and reset kernels; the loop and the "
                             "kernel each in the faster of the two step orders"}
            apply_candidate(env, best_wpc)

        # the whole env step alone (no policy): the fused control-step launch
        # (or the separate kernels) over every world, as the graph replays it
        c0, c1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        c0.record(stream)
        for _ in range(M):
            env.step()
        c1.record(stream)
        c1.synchronize()
        control_step_ms = c0.elapsed_time(c1) / M

        e2e = None
        if not args.no_e2e:
            e2e = run_e2e(torch, env, params, stream, max(3, min(K, 50)))
            e2e["ms_per_step"] = round(max_over_ranks(torch, dist, e2e["ms_per_step"]), 4)
            e2e["value"] = round(whole_job_rate(world, n, 1, e2e["ms_per_step"]), 1)
            e2e_abi = run_e2e_reference_abi(env.sim, max(3, min(K, 20)))
            e2e_abi["ms_per_step"] = round(max_over_ranks(torch, dist, e2e_abi["ms_per_step"]), 4)
            e2e_abi["value"] = round(whole_job_rate(world, n, 1, e2e_abi["ms_per_step"]), 1)

    peak = ctypes.c_double(0.0)
    sim_lib().arc_probe_fp32_peak(ctypes.byref(peak), None)
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return None

    value = whole_job_rate(world, n, K, ms_total)
    achieved = n * FLOP_PER_ENV_STEP / (step_kernel_ms * 1e-3)
    cand = str(best_wpc)
    kernel_name = ("warp-per-leg" + (", work queue" if cand != "warps" else "") +
                   (f", {cand[4:]} substeps per launch" if cand.startswith("tile") else "")
                   if cand.startswith(("warps", "tile")) else "leg-parallel")
    form = form if cand.startswith("warps") else 0  # the fused forms need the warp-per-leg kernel
    # our launches per control step and range: the step order's two kernels
    # (with the warp-per-leg kernel), then the step, task and reset kernels
    # (form 0), the fused step and the reset kernel (1), the fused step alone
    # (2); the ranges' merge; the memset of the ended-world count is no kernel
    per_part = {0: 3, 1: 2, 2: 1}[form] + (2 if cand.startswith(("warps", "tile")) else 0)
    launches = (per_part * parts + (1 if parts > 1 else 0)) * K
    out = {
        "metric": METRIC, "value": round(value, 1), "unit": "env-steps/s", "n_gpus": world, "steps": K,
        "warmup": args.warmup, "ms_per_step": round(ms_total / K, 4), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": f"{n} worlds of the quadruped per GPU, difficulty uniform in {{0,...,1.0}}, "
                               "checkpoints, auto-reset, random-init MLP policy 195-256-256-12 tanh FP32 in the loop",
                   "worlds_per_gpu": n, "substeps": 20, "dt": 1 / 30,
                   "kernel": kernel_name,
                   "worlds_per_cta": 32 if cand.startswith(("warps", "tile")) else best_wpc,
                   "substeps_per_launch": int(cand[4:]) if cand.startswith("tile") else 20,
                   "autotune_step_kernel_ms": tune,
                   "parts": parts,
                   "control_step": FORMS[form],
                   "step_order": "each range's worlds by difficulty band, hardest first (arc_env_set_step_order)",
                   "autotune_control_step_ms": parts_tune,
                   "loop": ("policy then env.step() (one CUDA graph) per control step" if parts == 1 else
                            f"policy and step of {parts} world ranges, each on its own stream "
                            "(DeviceVecEnv.step_parts), joined every control step"),
                   "l2": "inputs larger than L2 (world records + 64x64 terrains: ~1.2 GB per GPU)"},
        "latency_ms": {"p50": round(float(np.percentile(lat_long, 50)), 4),
                       "p99": round(float(np.percentile(lat_long, 99)), 4), "max": round(float(lat_long.max()), 4),
                       "samples": int(len(lat_long)),
                       "timed_steps": {"p50": round(float(np.percentile(lat, 50)), 4),
                                       "max": round(float(lat.max()), 4), "samples": int(len(lat))}},
        "plain_kernel": plain,
        "speedup_vs_plain": round(plain["ms_per_step"] / (ms_total / K), 2) if plain else None,
        "speedup_vs_plain_step_kernel": round(plain["step_kernel_ms"] / step_kernel_ms, 2) if plain else None,
        "speedup_vs_plain_meaning": ("speedup_vs_plain: the whole control step, the FP32 MLP policy and the task "
                                     "kernels included (the same in both loops); speedup_vs_plain_step_kernel: "
                                     "the batched step kernel alone against the plain per-world kernel, both on "
                                     "the states after their loops, each in its faster step order"),
        "control_step_ms_without_policy": round(control_step_ms, 4),
        "roofline": {"bound": "fp32", "achieved": round(achieved / 1e12, 3),
                     "peak": round(peak.value / 1e12, 3), "unit": "TFLOP/s",
                     "frac": round(achieved / peak.value, 4) if peak.value else None,
                     "traffic": round(n * WARPS_DRAM_BYTES_PER_WORLD) if cand.startswith("warps") else None,
                     "traffic_unit": "bytes per launch (ncu, scaled from 16,384 worlds)",
                     "kernel": kernel_name + " step",
                     "kernel_ms": round(step_kernel_ms, 4),
                     "flop_per_env_step": FLOP_PER_ENV_STEP,
                     "peak_source": "measured FP32 FMA probe (arc_probe_fp32_peak) on this GPU",
                     "hbm_gbs_algorithmic": round(n * HBM_BYTES_PER_ENV_STEP / (step_kernel_ms * 1e-3) / 1e9, 1)},
        "gpu_launches": launches,
        "ended_in_last_step": ended,
        "clocks": clock,
    }
    if e2e:
        out["e2e"] = e2e
        out["e2e_reference_abi"] = e2e_abi
    if world == 1 and not args.no_workloads:
        out["workloads"] = run_workloads(torch, n)
    if world == 1 and not args.no_cpu:
        out["cpu_baseline"] = cpu_baseline(args.cpu_seconds, n)
    return out


def run_e2e(torch, env, params, stream, K) -> dict:
    """The same loop through host buffers, with the library's host-buffer
    step (arc_env_step_host). Every step: the policy reads the last
    observations and its actions are copied to pinned host memory (as the
    reference's loop, whose policy runs on the host, is also timed with its
    policy), then the step copies those actions in and the observations,
    rewards and done flags out to pinned host memory, the worlds in ranges
    whose copies overlap the next range's step; the number of ranges is the
    fastest of 1, 2, 3, 4 on a few steps."""
    n = env.num_envs
    host_act = torch.empty((n, 12), dtype=torch.float32, pin_memory=True)
    stream.synchronize()
    torch.cuda.synchronize()

    def one(chunks):
        with torch.cuda.stream(stream):
            policy_forward(torch, params, env.obs, env.actions)
            host_act.copy_(env.actions, non_blocking=True)
        stream.synchronize()
        env.step_host(host_act, chunks)

    def run(chunks, k):
        t = time.perf_counter()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(k):
            one(chunks)
        e1.record(stream)
        e1.synchronize()
        return e0.elapsed_time(e1) / k, (time.perf_counter() - t) / k * 1e3

    tried = {}
    for chunks in (1, 2, 3, 4):
        run(chunks, 2)
        tried[chunks] = round(run(chunks, 4)[0], 4)
    best = min(tried, key=tried.get)
    ms, wall = run(best, K)
    h2d = n * 12 * 4
    d2h = n * 12 * 4 + n * 195 * 4 + n * 4 + 2 * n
    return {"value": round(n / (ms * 1e-3), 1), "unit": "env-steps/s", "h2d_bytes_per_step": h2d,
            "d2h_bytes_per_step": d2h, "ms_per_step": round(ms, 4), "wall_ms_per_step": round(wall, 4),
            "chunks": best, "ms_per_chunks": tried,
            "path": "policy on the device, its actions to pinned host memory, then DeviceVecEnv.step_host "
                    "(arc_env_step_host): the actions in, observations, rewards and done flags out to pinned "
                    "host memory, synchronised every step"}


def run_e2e_reference_abi(sim, K) -> dict:
    """The drop-in figure: the calls the reference's task layer makes on its
    simulation every control step (arc/task.py:155-170, 231-259), through the
    reference's C ABI with host float64 buffers: arc_sim_step with the
    targets, arc_sim_observe and arc_sim_heights at the 143 observation
    offsets, each synchronous like the reference's. Physics and its I/O
    only: the task arithmetic, which the reference does in numpy, is not in
    it."""
    from arc_demo_b200.task import HEIGHT_OFFSETS
    n = sim.num_worlds
    rng = np.random.default_rng(5)
    targets = np.ascontiguousarray(np.tile(sim.default_angles, (n, 1)) + 0.6 * rng.uniform(-1, 1, (n, 12)))
    offsets = np.ascontiguousarray(HEIGHT_OFFSETS, dtype=np.float64)
    heights = np.empty((n, len(offsets)))

    def one():
        sim.step(targets)
        sim.observe()
        sim.heights(offsets, heights)

    for _ in range(2):
        one()
    t = time.perf_counter()
    for _ in range(K):
        one()
    ms = (time.perf_counter() - t) / K * 1e3
    h2d = n * 12 * 8 + offsets.nbytes
    d2h = n * (13 + 9 + 36 + 6) * 8 + n * 4 + heights.nbytes
    return {"value": round(n / (ms * 1e-3), 1), "unit": "env-steps/s", "h2d_bytes_per_step": h2d,
            "d2h_bytes_per_step": d2h, "ms_per_step": round(ms, 4),
            "path": "arc_sim_step + arc_sim_observe + arc_sim_heights with host float64 buffers (the reference's "
                    "C ABI, as arc/task.py calls it), wall clock, physics and its I/O only"}


# ---------------------------------------------------------------------------
# the other workloads, short legs beside the headline (one GPU, rank 0)

def ou_update(torch, ou, actions, gen, theta=0.15, sigma=0.3):
    """One control step of a per-joint Ornstein-Uhlenbeck process (dt = one
    control step), clipped to [-1, 1] into `actions`."""
    ou.mul_(1.0 - theta).add_(torch.randn(ou.shape, device=ou.device, generator=gen), alpha=sigma)
    torch.clamp(ou, -1.0, 1.0, out=actions)


def timed_loop(torch, stream, one, k):
    """k calls of one() on `stream`, each bracketed by CUDA events: total ms
    and per-call ms."""
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(k)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    stream.synchronize()
    t0.record(stream)
    for a, b in ev:
        a.record(stream)
        one()
        b.record(stream)
    t1.record(stream)
    t1.synchronize()
    return t0.elapsed_time(t1), np.array([a.elapsed_time(b) for a, b in ev])


def leg_uneven_ou(torch, n=4096, steps=300, warmup=20) -> dict:
    """4,096 worlds, difficulty U[0, 1] per world, per-joint OU actions
    (theta 0.15, sigma 0.3, clipped, seed 1), auto-reset on termination or
    after 1,000 steps; each control step is the OU update (three torch
    kernels) and the env's CUDA graph of the library's kernels."""
    from arc_demo_b200.task import TaskConfig
    from arc_demo_b200.torch_env import DeviceVecEnv
    env = DeviceVecEnv(n, TaskConfig(curriculum=False), seed=21)
    env.set_levels(np.random.default_rng(1).uniform(0.0, 1.0, n))
    stream = torch.cuda.Stream()
    gen = torch.Generator(device="cuda").manual_seed(1)
    with torch.cuda.stream(stream):
        env.reset()
        ou = torch.zeros((n, 12), device="cuda")

        def one():
            ou_update(torch, ou, env.actions, gen)
            env.step()
        for _ in range(warmup):
            one()
        # a batch this small fills a fraction of the GPU: the kernel and
        # worlds per CTA are the autotuner's choice for it
        best, tune = autotune(env, torch, stream)
        for _ in range(3):
            one()
        ms, lat = timed_loop(torch, stream, one, steps)
        ended = int(env.done_count.item())
    env.close()
    return {"worlds": n, "steps": steps, "env_steps_per_s": round(n * steps / (ms * 1e-3), 1),
            "step_kernel": str(best), "autotune_step_kernel_ms": tune,
            "ms_per_step": round(ms / steps, 4),
            "latency_ms": {"p50": round(float(np.percentile(lat, 50)), 4),
                           "p99": round(float(np.percentile(lat, 99)), 4), "max": round(float(lat.max()), 4)},
            "ended_in_last_step": ended,
            "loop": "OU actions on the device, then DeviceVecEnv.step() (one CUDA graph: step, task, "
                    "reset of ended worlds)"}


def leg_grid_sizes(torch, n=16384, steps=40, warmup=5) -> dict:
    """16,384 worlds whose grids are 16..64 columns a side (uniform per
    world), block heights U(0, 0.3 * difficulty * stand_height) written
    per column, difficulty U[0, 1], OU actions; every control step is one
    launch of the step kernel over all sizes (work queue)."""
    import ctypes
    from arc_demo_b200.native import KERNEL_WARPS, Sim
    rng = np.random.default_rng(4)
    grids = rng.integers(16, 65, n).astype(np.int32)
    diffs = rng.uniform(0.0, 1.0, n)
    sim = Sim(n, grids=grids, cell=0.4)
    sim.set_kernel(KERNEL_WARPS)
    sim.set_work_queue(True)
    sim.reset(np.arange(n), rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32), diffs)
    for i in range(n):
        sim.set_terrain(i, rng.uniform(0.0, 0.3 * diffs[i] * sim.stand_height, (grids[i], grids[i])), 0.4,
                        outside=-100.0)
    st = sim.get_state()
    st[:, : 13 * 13].reshape(n, 13, 13)[:, :, 2] += 0.2  # drop every robot onto its blocks
    sim.set_state(st)
    stream = torch.cuda.Stream()
    gen = torch.Generator(device="cuda").manual_seed(1)
    ou = torch.zeros((n, 12), device="cuda")
    actions = torch.zeros((n, 12), device="cuda")
    lib, ptr = sim._lib, sim.ptr
    a, h = ctypes.c_void_p(actions.data_ptr()), ctypes.c_void_p(stream.cuda_stream)

    def one():
        ou_update(torch, ou, actions, gen)
        lib.arc_sim_step_actions(ptr, a, h)
    with torch.cuda.stream(stream):
        for _ in range(warmup):
            one()
        ms, lat = timed_loop(torch, stream, one, steps)
    sim.close()
    return {"worlds": n, "steps": steps, "env_steps_per_s": round(n * steps / (ms * 1e-3), 1),
            "ms_per_step": round(ms / steps, 4), "grid_sizes": "16..64 columns a side, uniform per world",
            "columns_mean": round(float((grids.astype(np.float64) ** 2).mean()), 1),
            "loop": "OU actions on the device, then arc_sim_step_actions: one launch of the warp-per-leg kernel "
                    "over every world size through the work queue (physics step; no task layer)"}


def leg_fp64(torch, n, steps=6, warmup=3) -> dict:
    """The step in FP64 (the reference's precision) at the headline's world
    count: the leg-parallel FP64 kernel at 8 and 16 worlds per CTA and the
    FP64 warp-per-leg kernel (one CTA per group, work queue), each timed alone
    from the same settled states; then the control step with the fastest."""
    import ctypes
    from arc_demo_b200.native import KERNEL_LEGS, KERNEL_WARPS
    from arc_demo_b200.task import TaskConfig
    from arc_demo_b200.torch_env import DeviceVecEnv
    env = DeviceVecEnv(n, TaskConfig(curriculum=False), seed=3, fp64=True)
    env.set_levels(levels_for(n, 17))
    stream = torch.cuda.Stream()
    names = {"legs8": "leg-parallel FP64, 8 worlds per CTA", "legs16": "leg-parallel FP64, 16 worlds per CTA",
             "warps": "warp-per-leg FP64", "warps+queue": "warp-per-leg FP64, work queue"}

    def apply(cand):
        env.sim.set_work_queue(cand == "warps+queue")
        if cand.startswith("legs"):
            env.set_kernel(KERNEL_LEGS, int(cand[4:]))
        else:
            env.set_kernel(KERNEL_WARPS)
    with torch.cuda.stream(stream):
        env.reset()
        torch.nn.init.uniform_(env.actions, -1.0, 1.0)
        apply("legs8")
        for _ in range(warmup):
            env.step()
        stream.synchronize()
        start, tstart = env.sim.get_state(), env.gpu.get_state()
        lib, ptr = env.sim._lib, env.sim.ptr
        a, h = ctypes.c_void_p(env.actions.data_ptr()), ctypes.c_void_p(stream.cuda_stream)
        table = {}
        for cand in names:
            env.sim.set_state(start)
            torch.cuda.synchronize()
            apply(cand)
            lib.arc_sim_step_actions(ptr, a, h)  # first launch: per-device set-up
            env.sim.set_state(start)
            torch.cuda.synchronize()
            ms, _ = timed_loop(torch, stream, lambda: lib.arc_sim_step_actions(ptr, a, h), steps)
            table[cand] = round(ms / steps, 4)
        best = min(table, key=table.get)
        env.sim.set_state(start)
        env.gpu.set_state(tstart)
        torch.cuda.synchronize()
        apply(best)
        step_ms, _ = timed_loop(torch, stream, lambda: env.step(), steps)
    env.close()
    ms = table[best] * steps
    return {"worlds": n, "kernel": names[best], "step_kernel_ms_by_kernel": table,
            "step_kernel_ms": table[best], "env_steps_per_s_step_kernel": round(n * steps / (ms * 1e-3), 1),
            "control_step_ms": round(step_ms / steps, 4),
            "env_steps_per_s_control_step": round(n * steps / (step_ms * 1e-3), 1),
            "note": "actions fixed (uniform random); every kernel from the same states 3 steps after a reset; "
                    "control step = step, task, reset in one graph"}


def leg_serving(seconds=3.0, clients=8, rates=(200.0, 50.0), tick_cap=131072) -> dict:
    """The serving engine with 8 Poisson clients (each request steps one of
    the client's resident sessions of 1..8,192 worlds, log-uniform, for
    1..32 control steps with the task layer; worlds reset in place when their
    episode ends), the pool sized by a 40 GB budget, at 200 requests/s per
    client (more than one GPU steps: the latency includes queueing) and at
    50 (below saturation)."""
    from arc_demo_b200.serve import WORLD_BYTES, Server, run_load
    capacity = int(40e9 // WORLD_BYTES)
    out = {"clients": clients, "capacity": capacity, "tick_cap": tick_cap, "offered_seconds": seconds,
           "bytes_per_world": WORLD_BYTES}
    with Server(capacity, tick_cap=tick_cap) as sv:
        sid = sv.open(np.zeros(64))
        sv.wait(sv.request(sid, 2))
        sv.close_session(sid)
        for rate in rates:
            r = run_load(sv, clients, rate, seconds, seed=int(rate))
            out[f"rate_{int(rate)}"] = {k: (round(v, 4) if isinstance(v, float) else v) for k, v in r.items()}
    return out


def run_workloads(torch, n) -> dict:
    legs = {}
    for name, fn in (("uneven_4096_ou", lambda: leg_uneven_ou(torch)),
                     ("grid_sizes_16384", lambda: leg_grid_sizes(torch)),
                     ("fp64", lambda: leg_fp64(torch, n)),
                     ("serving", lambda: leg_serving())):
        t = time.perf_counter()
        try:
            legs[name] = fn()
        except Exception as e:  # a leg that fails is reported, the headline stands
            legs[name] = {"error": f"{type(e).__name__}: {e}"}
        legs[name]["wall_s"] = round(time.perf_counter() - t, 1)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
    return legs


# ---------------------------------------------------------------------------
# the reference's CPU path

REF_BUILD = {"": "-O3 -march=x86-64-v3 -ffp-contract=fast -fno-math-errno -fno-trapping-math -fopenmp (AVX2)",
             "_v4": "-O3 -march=x86-64-v4 -ffp-contract=fast -fno-math-errno -fno-trapping-math -fopenmp (AVX-512)"}


NO_REFERENCE = "oracle/_ref/libarcsim_ref.so not built (needs the reference sources)"


def reference_loop(n: int, seconds: float | None, steps: int | None, warmup: int, threads: int,
                   variant: str | None = None) -> dict:
    """The reference's OpenMP step/observe/heights (its csrc/, oracle/_ref) with
    the task layer (obs, reward, done, auto-reset) in numpy, over n worlds of
    the workload, the same MLP policy on the host (torch, all threads)."""
    import torch
    from oracle.oracle import RefSim, fastest_ref_variant, ref_available
    from oracle.task_oracle import TaskConfig, TaskOracle
    if not ref_available():
        raise RuntimeError(NO_REFERENCE)
    variant = fastest_ref_variant() if variant is None else variant
    torch.set_num_threads(threads)
    sim = RefSim(n, threads=threads, variant=variant)
    task = TaskOracle(sim, TaskConfig(curriculum=False), seed=5)
    task.level[:] = levels_for(n, 17)
    task.reset(np.arange(n))
    obs = task.observe()
    g = torch.Generator().manual_seed(1234)

    def lin(i, o):
        bound = 1.0 / np.sqrt(i)
        return (torch.rand(o, i, generator=g) * 2 - 1) * bound, (torch.rand(o, generator=g) * 2 - 1) * bound
    (w1, b1), (w2, b2), (w3, b3) = lin(195, 256), lin(256, 256), lin(256, 12)

    def one(obs):
        with torch.no_grad():
            x = torch.from_numpy(obs)
            a = torch.addmm(b3, torch.tanh(torch.addmm(b2, torch.tanh(torch.addmm(b1, x, w1.t())), w2.t())), w3.t())
        _, te, tr, _ = task.step(a.numpy())
        obs = task.observe()
        ended = np.flatnonzero(te | tr)
        if len(ended):
            task.reset(ended)
            obs[ended] = task.observe()[ended]
        return obs

    for _ in range(warmup):
        obs = one(obs)
    lat = []
    t0 = time.perf_counter()
    k = 0
    while True:
        s = time.perf_counter()
        obs = one(obs)
        lat.append(time.perf_counter() - s)
        k += 1
        el = time.perf_counter() - t0
        if (steps is not None and k >= steps) or (seconds is not None and el >= seconds):
            break
    sim.close()
    return {"value": n * k / el, "steps": k, "seconds": el, "lat": np.array(lat) * 1e3, "variant": variant}


def cpu_baseline(seconds: float, full_n: int) -> dict:
    """The reference's path over every world of the workload (like for
    like), plus a 4,096-world sample and one thread on 1,024 worlds."""
    import torch
    from oracle.oracle import ref_available
    if not ref_available():
        return {"unavailable": NO_REFERENCE}
    threads = os.cpu_count() or 1
    torch_threads = torch.get_num_threads()
    r = reference_loop(full_n, seconds, None, 1, threads)
    small_n = 4096
    rs = reference_loop(small_n, seconds / 3, None, 2, threads)
    # the same loop on one thread (OpenMP and torch), a shorter sample
    one_n = 1024
    r1 = reference_loop(one_n, seconds / 3, None, 1, 1)
    torch.set_num_threads(torch_threads)
    return {"value": round(r["value"], 1), "unit": "env-steps/s", "cores": threads, "kind": "reference",
            "sample": f"all {full_n} worlds (same difficulty mix), {r['steps']} control steps "
                      f"in {r['seconds']:.1f} s: reference csrc/ step+observe+heights with OpenMP x{threads}, "
                      "numpy task layer with auto-reset, MLP policy in torch on the host",
            "build": REF_BUILD[r["variant"]], "threads": threads,
            "latency_ms": {"p50": round(float(np.percentile(r["lat"], 50)), 3),
                           "p99": round(float(np.percentile(r["lat"], 99)), 3)},
            "sample_4096": {"value": round(rs["value"], 1), "unit": "env-steps/s", "cores": threads,
                            "sample": f"{small_n} worlds, {rs['steps']} control steps in {rs['seconds']:.1f} s"},
            "single_thread": {"value": round(r1["value"], 1), "unit": "env-steps/s", "cores": 1,
                              "sample": f"{one_n} worlds, {r1['steps']} control steps in {r1['seconds']:.1f} s, "
                                        "OpenMP and torch on one thread"}}


def run_reference(args) -> dict | None:
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return None
    from oracle.oracle import ref_available
    if not ref_available():
        return {"impl": "reference", "unavailable": NO_REFERENCE}
    threads = os.cpu_count() or 1
    n = args.worlds
    r = reference_loop(n, None, max(args.steps, 1), max(args.warmup, 0), threads)
    cpu = {"value": round(r["value"], 1), "unit": "env-steps/s", "cores": threads, "kind": "reference",
           "sample": f"all {n} worlds of the workload, {r['steps']} control steps", "build": REF_BUILD[r["variant"]]}
    return {"metric": METRIC, "value": round(r["value"], 1), "unit": "env-steps/s", "impl": "reference",
            "n_gpus": int(os.environ.get("WORLD_SIZE", "1")), "steps": r["steps"], "warmup": args.warmup,
            "ms_per_step": round(float(r["lat"].mean()), 3), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"{n} worlds of the quadruped, difficulty uniform in {{0,...,1.0}}, "
                                   "checkpoints, auto-reset, MLP policy 195-256-256-12 tanh on the host",
                       "worlds": n, "threads": threads, "build": REF_BUILD[r["variant"]]},
            "latency_ms": {"p50": round(float(np.percentile(r["lat"], 50)), 3),
                           "p99": round(float(np.percentile(r["lat"], 99)), 3)},
            "cpu_baseline": cpu,
            "e2e": {"value": round(r["value"], 1), "unit": "env-steps/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}


# ---------------------------------------------------------------------------
# the renderer

def render_scene(n: int, seed: int):
    """n worlds of the step workload's terrain mix, each robot a few steps
    into random drive targets, one checkpoint marker per world drawn as the
    task draws them, half of them in view."""
    from arc_demo_b200.native import Sim
    rng = np.random.default_rng(seed)
    sim = Sim(n)
    sim.reset(np.arange(n), rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32), levels_for(n, seed))
    targets = np.tile(sim.default_angles, (n, 1)) + rng.uniform(-0.5, 0.5, (n, 12))
    for _ in range(10):
        sim.step(targets)
    half = 0.5 * sim.grid * sim.cell - 1.0
    markers = np.zeros((n, 1, 4), dtype=np.float32)
    markers[:, 0, :2] = rng.uniform(-half, half, (n, 2))
    markers[:, 0, 3] = 0.5
    active = np.where(rng.random(n) < 0.5, 0, -1).astype(np.int32)
    return sim, markers, active


def render_cpu_baseline(sim, markers, active) -> dict:
    """The renderer's CPU restatement (brute force, one core) on one
    160 x 90 frame with one sample, scaled to a 640 x 360 frame of 4 samples
    by the number of rays."""
    from oracle.oracle import RenderOracle
    lib = sim._lib
    from oracle.oracle import World
    lib.arc_sim_world.restype = ctypes.POINTER(World)
    lib.arc_sim_world.argtypes = [ctypes.c_void_p, ctypes.c_int]
    w = lib.arc_sim_world(sim.ptr, 0).contents
    ora = RenderOracle(160, 90, samples=1)
    t = time.perf_counter()
    ora.frame(w, markers[0].astype(np.float64), int(active[0]))
    el = time.perf_counter() - t
    scale = (RENDER_W * RENDER_H * RENDER_SAMPLES) / (160 * 90)
    return {"value": round(1.0 / (el * scale), 4), "unit": "frames/s", "cores": 1, "kind": "port",
            "sample": f"one 160x90 frame with 1 sample in {el:.2f} s, scaled by rays to 640x360 with 4 samples "
                      "(oracle/render_oracle.c: every column and visual tested against every ray)"}


def render_roofline(torch, frames_per_s: float, clock: dict, frames_per_launch: int) -> dict:
    """Issue roofline of k_render: warp instructions per second (the frames
    rendered per second of one GPU times the instructions of a frame, from
    ncu) against 4 per SM per cycle at the SM clock sampled during the run."""
    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    mhz = clock.get("sm_mhz") or clock.get("sm_max_mhz") or 1965.0
    peak = sms * 4 * mhz * 1e6
    achieved = frames_per_s * RENDER_WARP_INST_PER_FRAME
    return {"bound": "issue", "kernel": "k_render", "achieved": round(achieved / 1e12, 4),
            "peak": round(peak / 1e12, 4), "unit": "T warp-instructions/s", "frac": round(achieved / peak, 4),
            "traffic": round(RENDER_DRAM_BYTES_PER_FRAME * frames_per_launch),
            "traffic_unit": f"bytes per launch of {frames_per_launch} frames (ncu, scaled from 16 frames)",
            "peak_source": f"{sms} SMs x 4 issue slots x {mhz:.0f} MHz (median SM clock under load)",
            "note": "no dense contraction and under 1% of HBM bandwidth: ray casting and shading are bound by "
                    "instruction issue"}


def run_render(args) -> dict | None:
    """Frames/s of the batched renderer: `value` device-resident (one launch
    renders every world's frame into HBM); `e2e` through the reference's
    arc_render_frame, one world per call into a host buffer."""
    import torch
    from arc_demo_b200.render import Renderer
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    n = args.render_worlds
    sim, markers, active = render_scene(n, 77 + rank)
    stream = torch.cuda.Stream()
    r = Renderer(RENDER_W, RENDER_H, visible=False)
    r.set_samples(RENDER_SAMPLES)
    d_markers = torch.from_numpy(markers).cuda()
    d_active = torch.from_numpy(active).cuda()
    out = torch.empty((n, RENDER_H, RENDER_W, 3), dtype=torch.uint8, device="cuda")
    h = stream.cuda_stream
    for _ in range(max(args.warmup, 3)):
        r.frames(sim, None, d_markers, d_active, out=out, stream=h)
    stream.synchronize()
    if dist:
        dist.barrier()
    K = args.steps
    with ClockSampler(local) as clocks:
        torch.cuda.synchronize()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record(stream)
        for _ in range(K):
            r.frames(sim, None, d_markers, d_active, out=out, stream=h)
        t1.record(stream)
        t1.synchronize()
        torch.cuda.synchronize()
    if dist:
        dist.barrier()
    ms_total = max_over_ranks(torch, dist, t0.elapsed_time(t1))
    clock = clocks.summary()
    # e2e: the reference's call, one world per call, frame copied to the host
    m = min(n, 64)
    img = np.empty((RENDER_H, RENDER_W, 3), dtype=np.uint8)
    one = Renderer(RENDER_W, RENDER_H, visible=False)
    for i in range(2):
        one.frame(sim, i, markers[i].astype(np.float64), int(active[i]), rgb=True)
    t = time.perf_counter()
    for i in range(m):
        one._lib.arc_render_frame(one._ptr, sim.ptr, i, markers[i].astype(np.float64).ctypes.data, 1,
                                  int(active[i]), img.ctypes.data)
    e2e_s = max_over_ranks(torch, dist, time.perf_counter() - t)
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return None
    value = world * n * K / (ms_total * 1e-3)
    rays = RENDER_W * RENDER_H * RENDER_SAMPLES
    res = {
        "metric": RENDER_METRIC, "value": round(value, 1), "unit": "frames/s", "n_gpus": world, "steps": K,
        "warmup": args.warmup, "ms_per_step": round(ms_total / K, 4), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": f"{n} worlds per GPU rendered per step at {RENDER_W}x{RENDER_H}, "
                               f"{RENDER_SAMPLES} rays per pixel, terrain difficulty uniform in {{0,...,1.0}}, "
                               "one checkpoint marker per world",
                   "frames_per_launch": n, "l2": f"output {n * rays // RENDER_SAMPLES * 3 / 1e6:.0f} MB per step, "
                                                  "larger than L2"},
        "primary_rays_per_s": round(value * rays, 1),
        "roofline": render_roofline(torch, value / world, clock, n),
        "gpu_launches": 2 * K,
        "clocks": clock,
        "e2e": {"value": round(m / e2e_s, 1), "unit": "frames/s", "h2d_bytes_per_step": 4 * 4 + 8,
                "d2h_bytes_per_step": RENDER_W * RENDER_H * 3,
                "path": "arc_render_frame (the reference's ABI), one world per call into a host buffer"},
    }
    if world == 1 and not args.no_cpu:
        res["cpu_baseline"] = render_cpu_baseline(sim, markers, active)
    return res


def main():
    args = parse()
    if args.workload == "render":
        if args.impl == "reference":
            if int(os.environ.get("RANK", "0")) == 0:
                print(json.dumps({"impl": "reference", "unavailable": "the reference renders with SDL2 and "
                                  "OpenGL 2.1 (csrc/arc_render.c); unavailable on this box"}), flush=True)
            return
        out = run_render(args)
        if out is not None:
            print(json.dumps(out), flush=True)
        return
    out = run_reference(args) if args.impl == "reference" else run_ours(args)
    if out is not None:
        print(json.dumps(out), flush=True)


if __name__ == "__main__":
    main()
