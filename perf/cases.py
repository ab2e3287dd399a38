"""What a user of this package has it do, as timed cases.

Each case is one pass through the public entry points: the batched control
step (device tensors, host buffers, the reference's own interfaces, FP32 and
FP64, worlds of one and of many terrain sizes), the reset of a batch, the
normalised training step, the serving engine and the renderer.

`exact` restates the control step - the XPBD solver and the task layer's
observations and rewards - in plain FP64 torch.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from arc_demo_b200.native import KERNEL_WARPS, Sim
from arc_demo_b200.render import Renderer
from arc_demo_b200.serve import Server
from arc_demo_b200.task import HEIGHT_OFFSETS, ArcTask, TaskConfig
from arc_demo_b200.torch_env import DeviceVecEnv
from arc_demo_b200.vec_env import DeviceVecEnvAdapter, DeviceVecNormalize

RING = 16    # control steps' actions a state holds; passes take them in turn
SETTLE = 4   # control steps from the reset's drop to standing on the ground
FLOPS = 415_600  # scalar operations of one world's control step of 20 substeps
STATE_BYTES = 4 * (13 * 13 + 21 * 6 + 12 * 4) + 4 * 21  # one world's FP32 record
OBS = 195


def listed() -> list[dict]:
    return [
        # one robot on rough ground through the task interface, as a viewer or
        # a controller in the loop steps it: latency only
        {"name": "play_1", "kind": "task", "n": 1, "difficulty": 0.5},
        # the small configuration: 64 worlds on flat ground through the
        # batched C ABI with host FP64 buffers, step then observe
        {"name": "sim_64", "kind": "sim", "n": 64, "difficulty": 0.0},
        # the medium configuration: 4,096 worlds of mixed difficulty, one
        # device-resident control step with auto-reset
        {"name": "env_4096", "kind": "env", "n": 4096, "fp64": False},
        # the large configuration, the benchmark's
        {"name": "env_65536", "kind": "env", "n": 65536, "fp64": False},
        # the reference's own precision
        {"name": "env64_16384", "kind": "env", "n": 16384, "fp64": True},
        # every world its own terrain size, 16..64 columns a side: the physics
        # step and the read-out, on the device
        {"name": "sized_16384", "kind": "sized", "n": 16384},
        # the large configuration for a policy on the host: actions from, and
        # observations to, pinned host memory
        {"name": "host_65536", "kind": "host", "n": 65536, "chunks": 3},
        # new episodes for a whole batch: terrain, stance, checkpoint, observation
        {"name": "reset_16384", "kind": "reset", "n": 16384},
        # a ragged batch (the last group of 32 worlds is partly filled)
        # through the training adapter with running normalisation
        {"name": "train_10007", "kind": "train", "n": 10007},
        # a client of the serving engine: 512 resident worlds, 8 control steps
        {"name": "serve_512", "kind": "serve", "n": 512, "steps": 8},
        # frames of every fourth of 1,024 worlds, as for a training video
        {"name": "render_256", "kind": "render", "n": 256, "width": 640, "height": 360},
        # one frame of one world into host memory (rgb_array)
        {"name": "frame_1", "kind": "frame", "n": 1, "width": 640, "height": 360},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["task", "sim", "env", "env", "env", "env64", "sized", "host", "reset", "train", "serve",
                       "render", "frame"])
    if kind == "task":
        return {"kind": kind, "n": _log_int(rng, 1, 256), "difficulty": round(rng.uniform(0.0, 1.0), 2)}
    if kind == "sim":
        return {"kind": kind, "n": _log_int(rng, 1, 8192), "difficulty": round(rng.choice([0.0, rng.random()]), 2)}
    if kind in ("env", "env64"):
        return {"kind": "env", "n": _log_int(rng, 1, 65536 if kind == "env" else 32768), "fp64": kind == "env64",
                "grid": rng.choice([64, 64, 48, 32])}
    if kind == "host":
        return {"kind": kind, "n": _log_int(rng, 256, 65536), "chunks": rng.randint(1, 4)}
    if kind == "serve":
        return {"kind": kind, "n": _log_int(rng, 1, 8192), "steps": rng.randint(1, 16)}
    if kind == "render":
        return {"kind": kind, "n": _log_int(rng, 1, 256), "width": 2 * rng.randint(100, 320),
                "height": 2 * rng.randint(80, 180)}
    if kind == "frame":
        return {"kind": kind, "n": 1, "width": 2 * rng.randint(100, 640), "height": 2 * rng.randint(80, 360)}
    return {"kind": kind, "n": _log_int(rng, 64, 16384)}


# ---------------------------------------------------------------------------
# states


def _seeds(rng, n):
    return rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)


def _actions(rng, n):
    """RING steps of an Ornstein-Uhlenbeck process (theta 0.15, sigma 0.3)
    clipped to [-1, 1], as exploring policies act; FP32, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(2**62)))
    ou = 0.5 * torch.randn((n, 12), device="cuda", generator=gen)
    out = torch.empty((RING, n, 12), device="cuda")
    for k in range(RING):
        ou += -0.15 * ou + 0.3 * torch.randn((n, 12), device="cuda", generator=gen)
        out[k] = ou.clamp(-1.0, 1.0)
    return out


def _env(case, rng, levels=True):
    n = case["n"]
    grid = case.get("grid", 64)
    env = DeviceVecEnv(n, TaskConfig(curriculum=False, grid=grid), seed=int(rng.integers(2**62)),
                       fp64=case.get("fp64", False), kernel=KERNEL_WARPS)
    env.sim.set_work_queue(True)
    if levels:
        env.set_levels(rng.uniform(0.0, 1.0, n))
    return env


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng([seed, case["n"]])
    kind, n = case["kind"], case["n"]
    st = {"kind": kind, "n": n, "k": 0}
    if kind == "task":
        st["task"] = task = ArcTask(n, TaskConfig(curriculum=False, difficulty=case["difficulty"]),
                                    seed=int(rng.integers(2**62)))
        st["actions"] = _actions(rng, n).cpu().numpy()
        task.reset(np.arange(n))
        for k in range(SETTLE):
            task.step(st["actions"][k])
        task.observe()
        st["k"] = SETTLE
    elif kind in ("sim", "sized"):
        grids = rng.integers(16, 65, n).astype(np.int32) if kind == "sized" else None
        st["sim"] = sim = Sim(n, grids=grids)
        sim.set_kernel(KERNEL_WARPS)
        sim.set_work_queue(True)
        diffs = rng.uniform(0.0, 1.0, n) if kind == "sized" else np.full(n, case["difficulty"])
        sim.reset(np.arange(n), _seeds(rng, n), diffs)
        st["actions"] = _actions(rng, n)
        st["targets"] = sim.default_angles + 0.6 * st["actions"].double().cpu().numpy()
        for k in range(SETTLE):
            sim.step(st["targets"][k])
        st["k"] = SETTLE
        if kind == "sized":
            del st["targets"]
            st["out"] = [torch.empty(s, dtype=t, device="cuda")
                         for s, t in (((n, 13), torch.float64), ((n, 9), torch.float64), ((n, 36), torch.float64),
                                      ((n, 6), torch.float64), ((n,), torch.int32))]
    elif kind in ("env", "host", "reset", "train", "render", "frame"):
        st["env"] = env = _env(case if kind not in ("render", "frame") else {**case, "n": 4 * n}, rng)
        if kind == "train":
            st["venv"] = DeviceVecNormalize(DeviceVecEnvAdapter(env))
            st["venv"].reset()
        else:
            env.reset()
        if kind != "reset":
            st["actions"] = _actions(rng, env.num_envs)
            for k in range(SETTLE):
                (st["venv"] if kind == "train" else env).step(st["actions"][k])
            st["k"] = SETTLE
        if kind == "host":
            st["actions"] = st["actions"].cpu().pin_memory()
            env.step_host(st["actions"][st["k"]], case["chunks"])  # allocates the host outputs
            st["k"] += 1
        if kind == "render":
            st["ids"] = torch.arange(0, 4 * n, 4, dtype=torch.int32, device="cuda")
            st["size"] = (case["width"], case["height"])
        if kind == "frame":
            st["renderer"] = Renderer(case["width"], case["height"], visible=False)
            task = env.gpu.get_state([0])[0]
            st["markers"] = np.array([[task[0], task[1], task[2], env.cfg.checkpoint_radius]])
        torch.cuda.synchronize()
    elif kind == "serve":
        st["server"] = server = Server(max(1024, 2 * n))
        st["session"] = server.open(rng.uniform(0.0, 1.0, n), key=int(rng.integers(2**62)))
        st["actions"] = np.tile(_actions(rng, n).cpu().numpy(), (1 + case["steps"] // RING, 1, 1))[: case["steps"]]
        server.wait(server.request(st["session"], SETTLE, ou_seed=int(rng.integers(2**62))))
    else:
        raise ValueError(kind)
    return st


_holder = {}  # the state run last: an env's outputs alias its device buffers, so it outlives them


def run(st: dict):
    kind, k = st["kind"], st["k"] % RING
    st["k"] += 1
    _holder["state"] = st
    if kind == "task":
        task = st["task"]
        reward, terminated, truncated, stats = task.step(st["actions"][k])
        root, joints = task.sim.root.copy(), task.sim.joints.copy()
        ended = np.flatnonzero(terminated | truncated)
        if len(ended):
            task.reset(ended)
        return {"obs": task.observe(), "reward": reward, "terminated": terminated, "truncated": truncated,
                "cause": stats["cause"], "root": root, "joints": joints}
    if kind == "sim":
        sim = st["sim"]
        sim.step(st["targets"][k])
        root, joints, contacts, flags = sim.observe()
        return {"root": root, "rot": sim.rot, "joints": joints, "contacts": contacts, "flags": flags}
    if kind == "sized":
        sim, out = st["sim"], st["out"]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or 1)
        sim._check(sim._lib.arc_sim_step_actions(sim.ptr, st["actions"][k].data_ptr(), stream))
        sim._check(sim._lib.arc_sim_observe_device(sim.ptr, *[o.data_ptr() for o in out], stream))
        return dict(zip(("root", "rot", "joints", "contacts", "flags"), out))
    if kind == "env":
        env = st["env"]
        obs, reward, terminated, truncated = env.step(st["actions"][k])
        return {"obs": obs, "reward": reward, "terminated": terminated, "truncated": truncated, "cause": env.cause}
    if kind == "host":
        obs, reward, terminated, truncated = st["env"].step_host(st["actions"][k])
        return {"obs": obs, "reward": reward, "terminated": terminated, "truncated": truncated}
    if kind == "reset":
        return st["env"].reset()
    if kind == "train":
        obs, reward, dones, infos = st["venv"].step(st["actions"][k])
        rms = st["venv"].obs_rms
        return {"obs": obs, "reward": reward, "dones": dones, "mean": rms.mean, "var": rms.var,
                "returns_var": st["venv"].ret_rms.var, "returns": st["venv"].returns}
    if kind == "serve":
        server = st["server"]
        (obs, reward, done), _ = server.wait(server.request(st["session"], len(st["actions"]), st["actions"]))
        return {"obs": obs, "reward": reward, "done": done}
    if kind == "render":
        return st["env"].render(st["ids"], *st["size"])
    return st["renderer"].frame(st["env"].sim, 0, st["markers"], 0, rgb=True)


def work(case: dict) -> dict:
    kind, n = case["kind"], case["n"]
    real = 2 if case.get("fp64") else 1
    step_bytes = 2 * real * STATE_BYTES
    if kind in ("sim", "sized"):
        return {"bytes": n * (step_bytes + (96 if kind == "sim" else 48) + 8 * 64 + 4), "flops": n * FLOPS}
    if kind in ("task", "env", "host", "train"):
        return {"bytes": n * (step_bytes + 48 + 4 * OBS + 4 + 2), "flops": n * FLOPS}
    if kind == "serve":
        return {"bytes": n * case["steps"] * (step_bytes + 48 + 5) + n * 4 * OBS, "flops": n * case["steps"] * FLOPS}
    if kind == "reset":
        # 4,096 columns a world: two interpolated noises, a jitter, a quantisation
        return {"bytes": n * (4 * 4096 + STATE_BYTES + 4 * OBS), "flops": n * 4096 * 40}
    # a frame: 4 primary rays a pixel against the grid and some of the 74 shapes, one surface shaded
    pixels = n * case["width"] * case["height"]
    return {"bytes": 3 * pixels, "flops": pixels * (4 * 150 + 300)}


# ---------------------------------------------------------------------------
# the same results in 64 bits


def exact(case: dict, seed: int):
    """The control step's outputs from the prepared inputs, in FP64 torch.
    None for: a reset (random draws), frames (8-bit pictures), the serving
    engine (its worlds cannot be read), batches too large to restate here.
    A world whose episode ends in the step keeps that step's observation
    here, where the framework returns the next episode's first."""
    if case["kind"] not in ("task", "sim", "sized", "env", "host", "train") or case["n"] > 20000:
        return None
    st = prepare(case, seed)
    k = st["k"] % RING
    env = st.get("env") or st.get("task")
    sim = st["sim"] if env is None else env.sim
    model = _Model(sim)
    w = _read_state(sim)
    targets = torch.as_tensor(st["targets"][k], device="cuda") if case["kind"] == "sim" else None
    if targets is None:
        act = torch.as_tensor(np.asarray(st["actions"][k].cpu() if torch.is_tensor(st["actions"]) else
                                         st["actions"][k]), device="cuda").double()
        targets = model.default + 0.6 * act
    before = None if env is None else torch.as_tensor(env.gpu.get_state(), device="cuda")
    rms = st["venv"].state_dict() if case["kind"] == "train" else None
    returns = st["venv"].returns.clone() if case["kind"] == "train" else None
    _control_step(model, w, torch.minimum(torch.maximum(targets, model.lo), model.hi), sim.dt, sim.substeps)
    root = torch.cat([w["x"][:, 0], w["q"][:, 0], w["v"][:, 0], w["w"][:, 0]], 1)
    joints = torch.cat([w["angle"], w["rate"], w["torque"]], 1)
    if case["kind"] in ("sim", "sized"):
        rot = _rotation(w["q"][:, 0])
        return {"root": root, "rot": rot if case["kind"] == "sim" else rot.reshape(-1, 9), "joints": joints,
                "contacts": w["contacts"], "flags": None}
    obs, reward = _observe(model, w, before, act, env.cfg, sim)
    out = {"obs": obs, "reward": reward, "terminated": None, "truncated": None, "cause": None}
    if case["kind"] == "task":
        out.update(root=root, joints=joints)
    if case["kind"] == "host":
        del out["cause"]
    if case["kind"] == "train":
        def merge(r, batch):  # Chan, Golub and LeVeque (1979)
            m, total = batch.shape[0], r["count"] + batch.shape[0]
            d = batch.mean(0) - r["mean"]
            m2 = r["var"] * r["count"] + batch.var(0, unbiased=False) * m + d * d * (r["count"] * m / total)
            return r["mean"] + d * (m / total), m2 / total
        mean, var = merge(rms["obs_rms"], obs)
        returns = returns * 0.99 + reward
        _, ret_var = merge(rms["ret_rms"], returns)
        out = {"obs": ((obs - mean) / torch.sqrt(var + 1e-8)).clamp(-10.0, 10.0),
               "reward": (reward / torch.sqrt(ret_var + 1e-8)).clamp(-10.0, 10.0), "dones": None, "mean": mean,
               "var": var, "returns_var": ret_var, "returns": None}
    return out


class _Model:
    """The robot's constants, from world 0's arc_world record (include/arc_world.h)."""

    def __init__(self, sim):
        p = sim._lib.arc_sim_world(sim.ptr, 0)
        head = np.frombuffer(ctypes.string_at(p, 72), dtype=np.float64)
        self.g, self.mu_s, self.mu_d = head[:3].copy(), head[3], head[4]
        bodies = np.frombuffer(ctypes.string_at(p + 72, 16 * 368), dtype=np.float64).reshape(16, 46)[:13]
        joints = np.frombuffer(ctypes.string_at(p + 72 + 16 * 368, 16 * 296), dtype=np.float64).reshape(16, 37)[:12]
        raw = ctypes.string_at(p + 72 + 16 * 368 + 16 * 296, 48 * 96)
        spheres = np.frombuffer(raw, dtype=np.float64).reshape(48, 12)[:21]

        def dev(a):
            return torch.as_tensor(np.ascontiguousarray(a), device="cuda")
        self.inv_mass = dev(bodies[:, 21])
        self.inertia, self.inv_inertia = dev(bodies[:, 22:25]), dev(bodies[:, 25:28])
        self.r1, self.r2, self.a1, self.a2, self.b1, self.b2 = (dev(joints[:, 1 + 3 * i:4 + 3 * i]) for i in range(6))
        self.jlo, self.jhi, self.kp, self.kd, self.max_torque = (dev(joints[:, 23 + i]) for i in range(5))
        self.pos, self.radius = dev(spheres[:, 1:4]), spheres[:, 4].copy()
        self.default, self.lo, self.hi = dev(sim.default_angles), dev(sim.lo), dev(sim.hi)
        self.stand_height = sim.stand_height


def _read_state(sim) -> dict:
    n = sim.num_worlds
    s = torch.as_tensor(sim.get_state(), device="cuda")
    body = s[:, :169].reshape(n, 13, 13)
    ball = s[:, 169:337].reshape(n, 21, 8)
    h = np.full((n, sim.grid * sim.grid), -100.0)
    geom = np.zeros((n, 5))
    for i in range(n):
        t, g = sim.get_terrain(i)
        h[i, :t.size] = t.ravel()
        geom[i] = (t.shape[1], *g)
    return {"x": body[..., 0:3].clone(), "q": body[..., 3:7].clone(), "v": body[..., 7:10].clone(),
            "w": body[..., 10:13].clone(), "anchored": ball[..., 0] != 0, "anchor": ball[..., 1:4].clone(),
            "anchor_n": ball[..., 4:7].clone(), "h": torch.as_tensor(h, device="cuda"),
            "geom": torch.as_tensor(geom, device="cuda")}


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _cross(a, b):
    return torch.linalg.cross(*torch.broadcast_tensors(a, b))


def _mv(m, v):
    return (m @ v.expand(m.shape[:-1]).unsqueeze(-1)).squeeze(-1)


def _rotation(q):
    w, x, y, z = (q / q.norm(dim=-1, keepdim=True)).unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1
                       ).reshape(*q.shape[:-1], 3, 3)


def _turn(q, w):
    """q + 0.5 [w, 0] q"""
    return q + 0.5 * torch.cat([-_dot(w, q[..., 1:]), q[..., :1] * w + _cross(w, q[..., 1:])], -1)


def _skew(v):
    x, y, z = v.unbind(-1)
    o = torch.zeros_like(x)
    return torch.stack([o, -z, y, z, o, -x, -y, x, o], -1).reshape(*v.shape[:-1], 3, 3)


def _solve(K, r):
    return torch.linalg.solve(K, r.unsqueeze(-1)).squeeze(-1)


class _Bodies:
    """Bodies idx (one, or one per leg) of every world, with the rotation and
    world inverse inertia of their current q."""

    def __init__(self, m, w, idx):
        self.w, self.idx, self.im = w, idx, m.inv_mass[idx].unsqueeze(-1)
        self.ii = m.inv_inertia[idx]
        self.x, self.q = w["x"][:, idx], w["q"][:, idx]
        self.sync()

    def sync(self):
        self.rot = _rotation(self.q)
        self.iiw = (self.rot * self.ii.unsqueeze(-2)) @ self.rot.transpose(-1, -2)

    def push(self, r, p):
        self.x = self.x + self.im * p
        self.q = _turn(self.q, _mv(self.iiw, _cross(r, p)))
        self.sync()

    def twist(self, p):
        self.q = _turn(self.q, _mv(self.iiw, p))
        self.sync()

    def mass_at(self, r, n):
        rn = _cross(r, n)
        return self.im + _dot(rn, _mv(self.iiw, rn))

    def store(self):
        self.w["x"][:, self.idx], self.w["q"][:, self.idx] = self.x, self.q


def _joint(m, w, p, c, j, target, acc, hh):
    """One joint (or one per leg) between bodies p and c: drive, limit, axis, attachment."""
    A, B = _Bodies(m, w, p), _Bodies(m, w, c)

    def col(v):
        return v[j].unsqueeze(-1)

    def axis_angle():
        a1, b1, b2 = _mv(A.rot, m.a1[j]), _mv(A.rot, m.b1[j]), _mv(B.rot, m.b2[j])
        return a1, torch.atan2(_dot(_cross(b1, b2), a1), _dot(b1, b2))

    def block(rhs):
        ok = _dot(rhs, rhs) >= 1e-24
        p_ = torch.where(ok, _solve(A.iiw + B.iiw, rhs), torch.zeros_like(rhs))
        A.twist(p_)
        B.twist(-p_)

    a1, phi = axis_angle()
    err = phi - target[:, j].unsqueeze(-1)
    n = a1 * torch.sign(err)
    denom = _dot(n, _mv(A.iiw, n)) + _dot(n, _mv(B.iiw, n)) + 1.0 / (col(m.kp) * hh)
    dl = torch.minimum(err.abs() / denom, col(m.max_torque) * hh)
    acc[:, j] -= (_dot(n, a1) * dl / hh).squeeze(-1)
    A.twist(n * dl)
    B.twist(-n * dl)
    a1, phi = axis_angle()
    block(a1 * (phi - torch.minimum(torch.maximum(phi, col(m.jlo)), col(m.jhi))))
    block(_cross(_mv(A.rot, m.a1[j]), _mv(B.rot, m.a2[j])))
    r1, r2 = _mv(A.rot, m.r1[j]), _mv(B.rot, m.r2[j])
    d = (B.x + r2) - (A.x + r1)
    K = torch.eye(3, dtype=d.dtype, device=d.device) * (A.im + B.im).unsqueeze(-1)
    K = K - _skew(r1) @ A.iiw @ _skew(r1) - _skew(r2) @ B.iiw @ _skew(r2)
    imp = torch.where(_dot(d, d) >= 1e-24, _solve(K, d), torch.zeros_like(d))
    A.push(r1, imp)
    B.push(r2, -imp)
    A.store()
    B.store()


def _height(w, ix, iy):
    """Column heights, ix and iy (N, ...)."""
    n = w["geom"][:, 0].reshape(-1, *[1] * (ix.dim() - 1))
    inside = (ix >= 0) & (iy >= 0) & (ix < n) & (iy < n)
    at = torch.where(inside, ix + iy * n, torch.zeros_like(ix)).long()
    h = torch.gather(w["h"], 1, at.reshape(at.shape[0], -1)).reshape(at.shape)
    return torch.where(inside, h, w["geom"][:, 4].reshape(n.shape).expand_as(h))


def _collide(m, w, B, s, xp, qp, touched_out, contacts):
    """Sphere s (one, or one per leg) of bodies B against the columns, then its friction."""
    rad, pos = m.radius[s if isinstance(s, int) else s[0]], m.pos[s]
    c = B.x + _mv(B.rot, pos)
    cell, ox, oy = (w["geom"][:, i].reshape(-1, *[1] * (c.dim() - 2)) for i in (1, 2, 3))
    first = [torch.floor((c[..., i] - rad - o) / cell) for i, o in ((0, ox), (1, oy))]
    last = [torch.floor((c[..., i] + rad - o) / cell) for i, o in ((0, ox), (1, oy))]
    ln = torch.zeros_like(c[..., :1])
    deepest, n_max = ln.clone(), torch.zeros_like(c)
    n_max[..., 2] = 1.0
    touched = torch.zeros_like(ln, dtype=torch.bool)
    span = int(2 * rad / float(w["geom"][:, 1].min())) + 2
    for dy in range(span):
        for dx in range(span):
            ix, iy = first[0] + dx, first[1] + dy
            top = _height(w, ix, iy)
            hit = (ix <= last[0]) & (iy <= last[1]) & (c[..., 2] - rad < top)
            x0, y0 = ox + ix * cell, oy + iy * cell
            sx = (c[..., 0] > x0 + cell).double() - (c[..., 0] < x0).double()
            sy = (c[..., 1] > y0 + cell).double() - (c[..., 1] < y0).double()
            hit &= ~((sx != 0) & (_height(w, ix + sx, iy) >= top))
            hit &= ~((sy != 0) & (_height(w, ix, iy + sy) >= top))
            hit &= ~((sx != 0) & (sy != 0) & (_height(w, ix + sx, iy + sy) >= top))
            near = torch.stack([torch.minimum(torch.maximum(c[..., 0], x0), x0 + cell),
                                torch.minimum(torch.maximum(c[..., 1], y0), y0 + cell),
                                torch.minimum(c[..., 2], top)], -1)
            diff = c - near
            dist = diff.norm(dim=-1, keepdim=True)
            out = dist > 1e-9
            hit = hit.unsqueeze(-1) & ~(out & (dist >= rad))
            up = torch.zeros_like(c)
            up[..., 2] = 1.0
            n = torch.where(out, diff / torch.where(out, dist, torch.ones_like(dist)), up)
            depth = torch.where(out, rad - dist, top.unsqueeze(-1) - c[..., 2:] + rad)
            depth = torch.where(hit, depth, torch.zeros_like(depth))
            r = c - n * rad - B.x
            dl = depth / B.mass_at(r, n)
            B.push(r, n * dl)
            contacts.append((hit, _mv(B.rot.transpose(-1, -2), r), n))
            ln = ln + dl
            n_max = torch.where(hit & (depth > deepest), n, n_max)
            deepest = torch.maximum(deepest, depth)
            touched |= hit
            c = B.x + _mv(B.rot, pos)
    anchored, anchor, anchor_n = w["anchored"][:, s].unsqueeze(-1), w["anchor"][:, s], w["anchor_n"][:, s]
    fresh = touched & (~anchored | (_dot(n_max, anchor_n) < 0.9))
    anchor = torch.where(fresh, xp + _mv(_rotation(qp), pos) - n_max * rad, anchor)
    anchor_n = torch.where(fresh, n_max, anchor_n)
    e = c - n_max * rad - anchor
    e = e - n_max * _dot(e, n_max)
    length = e.norm(dim=-1, keepdim=True)
    slips = touched & (length >= 1e-12)
    r = c - n_max * rad - B.x
    dl = length / B.mass_at(r, e / torch.where(slips, length, torch.ones_like(length)))
    frac = torch.where(dl > m.mu_s * ln, torch.clamp(m.mu_d * ln / torch.where(slips, dl, torch.ones_like(dl)), max=1.0),
                       torch.ones_like(dl))
    frac = torch.where(slips, frac, torch.zeros_like(frac))
    w["anchor"][:, s] = torch.where(slips, anchor + e * (1.0 - frac), anchor)
    w["anchor_n"][:, s] = anchor_n
    w["anchored"][:, s] = touched.squeeze(-1)
    B.push(r, -e * (frac * dl / torch.where(slips, length, torch.ones_like(length))))
    touched_out[:, s] += touched.squeeze(-1)


def _control_step(m, w, target, dt, substeps):
    h = dt / substeps
    g = torch.as_tensor(m.g, device="cuda")
    coxa, femur, tibia = ([1 + 3 * l + i for l in range(4)] for i in range(3))
    n = target.shape[0]
    acc = torch.zeros_like(target)
    touch = torch.zeros((n, 21), dtype=torch.float64, device="cuda")
    rot = _rotation(w["q"])
    for _ in range(substeps):
        xp, qp = w["x"].clone(), w["q"].clone()
        w["v"] = w["v"] + g * h
        w["x"] = w["x"] + w["v"] * h
        # gyroscopic term, implicit, in the body frame
        wb = _mv(rot.transpose(-1, -2), w["w"])
        iw = wb * m.inertia
        J = torch.diag_embed(m.inertia) + h * (_skew(wb) * m.inertia.unsqueeze(-2) - _skew(iw))
        w["w"] = _mv(rot, wb - _solve(J, h * _cross(wb, iw)))
        w["q"] = _turn(w["q"], w["w"] * h)
        for l in range(4):
            _joint(m, w, 0, coxa[l], 3 * l, target, acc, h * h)
        legs = [3 * l for l in range(4)]
        _joint(m, w, coxa, femur, [j + 1 for j in legs], target, acc, h * h)
        _joint(m, w, femur, tibia, [j + 2 for j in legs], target, acc, h * h)
        found = []
        for body, balls in ((0, [0]), (femur, [[1 + 5 * l for l in range(4)]]),
                            (tibia, [[i + 5 * l for l in range(4)] for i in (2, 3, 4, 5)])):
            B, contacts = _Bodies(m, w, body), []
            for s in balls:
                _collide(m, w, B, s, xp[:, body], qp[:, body], touch, contacts)
            B.store()
            found.append((body, contacts))
        rot = _rotation(w["q"])
        iiw = (rot * m.inv_inertia.unsqueeze(-2)) @ rot.transpose(-1, -2)
        w["q"] = w["q"] / w["q"].norm(dim=-1, keepdim=True)
        qw, qv = w["q"][..., :1], w["q"][..., 1:]
        pw, pv = qp[..., :1], -qp[..., 1:]
        w["v"] = (w["x"] - xp) / h
        spin = qw * pv + pw * qv + _cross(qv, pv)
        w["w"] = torch.where(qw * pw - _dot(qv, pv) < 0, -spin, spin) * (2.0 / h)

        def damp(p, c, j):
            a = _mv(rot[:, p], m.a1[j])
            rel = _dot(w["w"][:, c] - w["w"][:, p], a)
            cap = torch.minimum(rel.abs() / (_dot(a, _mv(iiw[:, p], a)) + _dot(a, _mv(iiw[:, c], a))),
                                m.max_torque[j].unsqueeze(-1) * h)
            imp = torch.minimum(torch.maximum(-m.kd[j].unsqueeze(-1) * rel * h, -cap), cap)
            w["w"][:, p] -= _mv(iiw[:, p], a * imp)
            w["w"][:, c] += _mv(iiw[:, c], a * imp)
            acc[:, j] += imp.squeeze(-1) / h
        for l in range(4):
            damp(0, coxa[l], 3 * l)
        damp(coxa, femur, [j + 1 for j in legs])
        damp(femur, tibia, [j + 2 for j in legs])
        for body, contacts in found:
            for hit, local, nrm in contacts:
                r = _mv(rot[:, body], local)
                im = m.inv_mass[body].unsqueeze(-1)
                rn = _cross(r, nrm)
                vn = _dot(nrm, w["v"][:, body] + _cross(w["w"][:, body], r))
                p = nrm * (-vn / (im + _dot(rn, _mv(iiw[:, body], rn))))
                p = torch.where(hit, p, torch.zeros_like(p))
                w["v"][:, body] = w["v"][:, body] + p * im
                w["w"][:, body] = w["w"][:, body] + _mv(iiw[:, body], _cross(r, p))
    rot = _rotation(w["q"])
    par = [0 if j % 3 == 0 else j for j in range(12)]
    chi = list(range(1, 13))
    a, b1, b2 = _mv(rot[:, par], m.a1), _mv(rot[:, par], m.b1), _mv(rot[:, chi], m.b2)
    w["angle"] = torch.atan2(_dot(_cross(b1, b2), a), _dot(b1, b2)).squeeze(-1)
    w["rate"] = _dot(w["w"][:, chi] - w["w"][:, par], a).squeeze(-1)
    w["torque"] = acc / substeps
    share = touch / substeps
    leg = share[:, 1:].reshape(n, 4, 5)
    w["contacts"] = torch.cat([leg[:, :, 4], share[:, :1], leg[:, :, :4].reshape(n, -1).amax(1, keepdim=True)], 1)


def _observe(m, w, task, act, cfg, sim):
    """ArcTask's reward and observation after the step; task: the state before it."""
    x, v, om = w["x"][:, 0], w["v"][:, 0], w["w"][:, 0]
    rot = _rotation(w["q"][:, 0])
    lin, ang = _mv(rot.transpose(1, 2), v), _mv(rot.transpose(1, 2), om)
    head = torch.atan2(rot[:, 1, 0], rot[:, 0, 0])
    d = task[:, 0:2] - x[:, :2]
    dist = d.norm(dim=1)
    fwd, left = head.cos() * d[:, 0] + head.sin() * d[:, 1], head.cos() * d[:, 1] - head.sin() * d[:, 0]
    off = torch.as_tensor(HEIGHT_OFFSETS, device="cuda")
    px = x[:, :1] + head.cos()[:, None] * off[:, 0] - head.sin()[:, None] * off[:, 1]
    py = x[:, 1:2] + head.sin()[:, None] * off[:, 0] + head.cos()[:, None] * off[:, 1]
    cell, ox, oy = (w["geom"][:, i:i + 1] for i in (1, 2, 3))
    top = _height(w, torch.floor((px - ox) / cell), torch.floor((py - oy) / cell))
    obs = torch.cat([-rot[:, 2], lin, 0.25 * ang, w["angle"] - m.default, 0.1 * w["rate"], act.clamp(-1, 1),
                     torch.stack([fwd / dist.clamp(min=1e-6), left / dist.clamp(min=1e-6),
                                  dist.clamp(1e-6, 6.0) / 6.0], 1),
                     (x[:, 2:] - m.stand_height - top).clamp(-1.0, 1.0), w["contacts"][:, :4]], 1)
    gaze = torch.atan2(rot[:, 0, 0] * d[:, 1] - rot[:, 1, 0] * d[:, 0],
                       rot[:, 0, 0] * d[:, 0] + rot[:, 1, 0] * d[:, 1]).abs()
    cos_fov = math.cos(math.radians(cfg.fov))
    view = ((gaze.cos() - cos_fov) / (1.0 - cos_fov)).clamp(0.0, 1.0)
    progress = (task[:, 3] - dist).clamp(max=cfg.max_speed * cfg.dt)
    progress = torch.where(progress > 0, progress * view, progress)
    reached = (dist < cfg.checkpoint_radius) & (gaze < math.radians(cfg.fov))
    torso = w["contacts"][:, 4] > 0
    half = 0.5 * sim.grid * sim.cell
    fell = ((rot[:, 2, 2] < cfg.flip_up_z) | (torch.where(torso, task[:, 17] + 1, 0 * dist) > cfg.beached_steps)
            | (x[:, 0].abs() > half) | (x[:, 1].abs() > half) | (x[:, 2] < cfg.void_z))
    reward = (cfg.w_progress * progress + cfg.w_turn * (task[:, 4] - gaze) + cfg.w_checkpoint * reached.double()
              - cfg.w_time - cfg.w_energy * cfg.dt * (w["rate"] * w["torque"]).abs().sum(1)
              - cfg.w_action_rate * (act.clamp(-1, 1) - task[:, 5:17]).square().sum(1)
              - cfg.w_body_contact * (w["contacts"][:, 5] > 0).double() - cfg.w_torso_contact * torso.double()
              - cfg.w_body_rate * ang[:, :2].square().sum(1) - cfg.w_bounce * v[:, 2].square()
              - cfg.w_fall * fell.double())
    return obs, reward
