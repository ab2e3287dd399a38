"""A vectorised-env adapter and observation/reward normalisation on the device.

The reference trains through Stable-Baselines3: `ArcVecEnv` (an SB3 `VecEnv`
with auto-reset and terminal observations, arc/env.py:74-141) wrapped in SB3's
`VecNormalize` (scripts/train.py:116-142). Both keep their data in host numpy
arrays. This module gives the same interface on device tensors, over
`DeviceVecEnv` (or any env with `reset()` and `step(actions)` returning torch
tensors):

- `DeviceVecEnvAdapter`: `num_envs`, `reset()`, `step_async(actions)` /
  `step_wait()` returning (obs, rewards, dones, infos) as device tensors;
  `infos` is one dict of tensors ("terminal_observation", "truncated") rather
  than one dict per world, which would bring every step back to the host.
- `DeviceVecNormalize`: running mean/variance of the observations and of the
  discounted returns, observations normalised and clipped to +-clip_obs,
  rewards scaled by the returns' standard deviation and clipped to
  +-clip_reward, the statistics frozen when `training` is False - the
  behaviour of SB3's VecNormalize with its defaults (clip 10, gamma 0.99,
  epsilon 1e-8). The statistics are FP64, as SB3's numpy ones are.
"""

from __future__ import annotations

import ctypes
import functools

import torch

_vp, _dbl, _int = ctypes.c_void_p, ctypes.c_double, ctypes.c_int


class _NormArgs(ctypes.Structure):
    """arc_norm_step_args of include/arc_sim.h."""
    _fields_ = ([("rows", ctypes.c_longlong)] + [(k, _int) for k in ("cols", "training", "norm_obs", "norm_reward")]
                + [(k, _vp) for k in ("obs", "terminal_obs", "rewards", "dones", "returns", "obs_mean", "obs_var",
                                      "ret_mean", "ret_var")]
                + [(k, _dbl) for k in ("obs_count", "ret_count", "gamma", "epsilon", "clip_obs", "clip_reward")]
                + [(k, _vp) for k in ("obs_out", "terminal_out", "rewards_out", "returns_out", "obs_mean_out",
                                      "obs_var_out", "ret_mean_out", "ret_var_out", "work")])


@functools.cache
def _norm_lib():
    from .native import sim_lib
    lib = sim_lib()
    lib.arc_norm_work_size.restype, lib.arc_norm_work_size.argtypes = ctypes.c_longlong, [ctypes.c_longlong, _int]
    lib.arc_norm_step.restype, lib.arc_norm_step.argtypes = _int, [ctypes.POINTER(_NormArgs), _vp]
    return lib


def _plain(x, dtype, shape, device) -> bool:
    """Whether the kernels can read x: a contiguous CUDA tensor of that type,
    shape and device, with nothing recorded or transformed about it."""
    # forward-mode derivatives ride on plain tensors, but only inside a level
    if torch.autograd.forward_ad._current_level >= 0:
        return False
    return (type(x) is torch.Tensor and x.dtype == dtype and tuple(x.shape) == shape and x.device == device
            and x.is_contiguous() and not x.requires_grad and not x.is_neg() and not x.is_inference()
            and torch._C._functorch.maybe_get_level(x) == -1 and not torch.compiler.is_compiling())


class DeviceRunningMeanStd:
    """Running mean and (population) variance over batches, merged with the
    parallel-variance formula of Chan, Golub and LeVeque (1979), starting
    from mean 0, variance 1 and a count of `epsilon`."""

    def __init__(self, shape=(), epsilon: float = 1e-4, device=None):
        self.mean = torch.zeros(shape, dtype=torch.float64, device=device)
        self.var = torch.ones(shape, dtype=torch.float64, device=device)
        self.count = epsilon

    def update(self, x: torch.Tensor) -> None:
        x = x.to(torch.float64)
        batch_mean = x.mean(dim=0)
        batch_var = x.var(dim=0, unbiased=False)
        self.update_from_moments(batch_mean, batch_var, x.shape[0])

    def update_from_moments(self, batch_mean, batch_var, batch_count: int) -> None:
        delta = batch_mean - self.mean
        total = self.count + batch_count
        new_mean = self.mean + delta * (batch_count / total)
        m2 = self.var * self.count + batch_var * batch_count + delta.square() * (self.count * batch_count / total)
        self.mean, self.var, self.count = new_mean, m2 / total, total

    def state_dict(self) -> dict:
        return {"mean": self.mean.clone(), "var": self.var.clone(), "count": self.count}

    def load_state_dict(self, d: dict) -> None:
        self.mean = d["mean"].to(self.mean.device, torch.float64).clone()
        self.var = d["var"].to(self.var.device, torch.float64).clone()
        self.count = float(d["count"])


class DeviceVecEnvAdapter:
    """SB3's VecEnv calling convention over a device env: step_async stores
    the actions, step_wait steps and returns device tensors."""

    def __init__(self, env):
        self.env = env
        self.num_envs = env.num_envs
        self._actions = None

    def reset(self) -> torch.Tensor:
        return self.env.reset()

    def step_async(self, actions: torch.Tensor) -> None:
        self._actions = actions

    def step_wait(self):
        obs, reward, terminated, truncated = self.env.step(self._actions)
        term, trunc = terminated.bool(), truncated.bool()
        infos = {"terminal_observation": self.env.terminal_obs, "truncated": trunc & ~term}
        return obs, reward, term | trunc, infos

    def step(self, actions: torch.Tensor):
        self.step_async(actions)
        return self.step_wait()


class DeviceVecNormalize:
    """SB3's VecNormalize on device tensors over a `DeviceVecEnvAdapter`-like
    env (reset, step_async/step_wait returning (obs, rewards, dones, infos))."""

    def __init__(self, venv, training: bool = True, norm_obs: bool = True, norm_reward: bool = True,
                 clip_obs: float = 10.0, clip_reward: float = 10.0, gamma: float = 0.99, epsilon: float = 1e-8):
        self.venv = venv
        self.num_envs = venv.num_envs
        self.training, self.norm_obs, self.norm_reward = training, norm_obs, norm_reward
        self.clip_obs, self.clip_reward, self.gamma, self.epsilon = clip_obs, clip_reward, gamma, epsilon
        self.obs_rms = None
        self.ret_rms = None
        self.returns = None
        self.old_obs = self.old_reward = None

    def _init_stats(self, obs: torch.Tensor) -> None:
        if self.obs_rms is None:
            self.obs_rms = DeviceRunningMeanStd(shape=obs.shape[1:], device=obs.device)
            self.ret_rms = DeviceRunningMeanStd(shape=(), device=obs.device)
            self.returns = torch.zeros(self.num_envs, dtype=torch.float64, device=obs.device)

    def normalize_obs(self, obs: torch.Tensor) -> torch.Tensor:
        if not self.norm_obs:
            return obs
        z = (obs.to(torch.float64) - self.obs_rms.mean) / torch.sqrt(self.obs_rms.var + self.epsilon)
        return z.clamp(-self.clip_obs, self.clip_obs).to(obs.dtype)

    def normalize_reward(self, reward: torch.Tensor) -> torch.Tensor:
        if not self.norm_reward:
            return reward
        r = reward.to(torch.float64) / torch.sqrt(self.ret_rms.var + self.epsilon)
        return r.clamp(-self.clip_reward, self.clip_reward).to(reward.dtype)

    def reset(self) -> torch.Tensor:
        obs = self.venv.reset()
        self._init_stats(obs)
        self.old_obs = obs
        self.returns.zero_()
        if self.training and self.norm_obs:
            self.obs_rms.update(obs)
        return self.normalize_obs(obs)

    def step_async(self, actions: torch.Tensor) -> None:
        self.venv.step_async(actions)

    def step_wait(self):
        obs, rewards, dones, infos = self.venv.step_wait()
        self._init_stats(obs)
        self.old_obs, self.old_reward = obs, rewards
        done = self._step_kernels(obs, rewards, dones, infos)
        if done is not None:
            return done
        if self.training and self.norm_obs:
            self.obs_rms.update(obs)
        norm_obs = self.normalize_obs(obs)
        if self.training:
            self.returns = self.returns * self.gamma + rewards.to(torch.float64)
            self.ret_rms.update(self.returns)
        norm_rewards = self.normalize_reward(rewards)
        infos = dict(infos)
        if "terminal_observation" in infos:
            infos["terminal_observation"] = self.normalize_obs(infos["terminal_observation"])
        self.returns = torch.where(dones.bool(), torch.zeros_like(self.returns), self.returns)
        return norm_obs, norm_rewards, dones, infos

    def _step_kernels(self, obs, rewards, dones, infos):
        """step_wait's statistics and normalisation by the library's kernels
        (arc_norm_step): what it returns, or None where the tensors are not
        ones they take (not on a CUDA device, other types, empty, recorded by
        autograd, ...), which the tensor operations below handle. Like them it
        leaves every tensor it was given or handed out before as it was."""
        if type(obs) is not torch.Tensor or obs.device.type != "cuda" or obs.dim() != 2 or not obs.numel():
            return None
        n, cols = obs.shape
        dev, f32, f64 = obs.device, torch.float32, torch.float64
        term = infos.get("terminal_observation") if type(infos) is dict else None
        rms, ret = self.obs_rms, self.ret_rms
        if (_replaced(self, _NORMALIZE) or any(type(r) is not DeviceRunningMeanStd or _replaced(r, _UPDATE)
                                               for r in (rms, ret))
                or torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack()
                or torch.jit.is_tracing()
                or not all(isinstance(v, (int, float)) for v in (rms.count, ret.count, self.gamma, self.epsilon,
                                                                 self.clip_obs, self.clip_reward))
                or not (self.clip_obs >= 0.0 and self.clip_reward >= 0.0)):
            return None  # normalisation of the caller's own, something that traces the operations, odd settings
        if (cols > 2048 or n != self.num_envs or type(infos) is not dict
                or not _plain(obs, f32, (n, cols), dev) or not _plain(rewards, f32, (n,), dev)
                or not _plain(dones, torch.bool, (n,), dev) or not _plain(self.returns, f64, (n,), dev)
                or not all(_plain(t, f64, (cols,), dev) for t in (rms.mean, rms.var))
                or not all(_plain(t, f64, (), dev) for t in (ret.mean, ret.var))
                or ("terminal_observation" in infos and not _plain(term, f32, (n, cols), dev))):
            return None
        lib = _norm_lib()
        with torch.cuda.device(dev):
            work = torch.empty(lib.arc_norm_work_size(n, cols) if self.training else 1, dtype=f64, device=dev)
            returns, mean, var, ret_mean, ret_var = (torch.empty(s, dtype=f64, device=dev)
                                                     for s in (n, cols, cols, (), ()))
            norm_obs = torch.empty_like(obs) if self.norm_obs else obs
            norm_term = torch.empty_like(term) if self.norm_obs and term is not None else term
            norm_rewards = torch.empty_like(rewards) if self.norm_reward else rewards
            args = _NormArgs(
                n, cols, bool(self.training), bool(self.norm_obs), bool(self.norm_reward), obs.data_ptr(),
                None if term is None else term.data_ptr(), rewards.data_ptr(), dones.data_ptr(),
                self.returns.data_ptr(), rms.mean.data_ptr(), rms.var.data_ptr(), ret.mean.data_ptr(),
                ret.var.data_ptr(), rms.count, ret.count, self.gamma, self.epsilon, self.clip_obs, self.clip_reward,
                norm_obs.data_ptr() if self.norm_obs else None,
                norm_term.data_ptr() if self.norm_obs and term is not None else None, norm_rewards.data_ptr(),
                returns.data_ptr(), mean.data_ptr(), var.data_ptr(), ret_mean.data_ptr(), ret_var.data_ptr(),
                work.data_ptr())
            stream = torch.cuda.current_stream(dev).cuda_stream
            if lib.arc_norm_step(ctypes.byref(args), stream or 1):  # 1: the legacy default stream
                raise RuntimeError("arc_norm_step failed")
        if self.training:
            if self.norm_obs:
                rms.mean, rms.var, rms.count = mean, var, rms.count + n
            ret.mean, ret.var, ret.count = ret_mean, ret_var, ret.count + n
        self.returns = returns
        infos = dict(infos)
        if term is not None:
            infos["terminal_observation"] = norm_term
        return norm_obs, norm_rewards, dones, infos

    def step(self, actions: torch.Tensor):
        self.step_async(actions)
        return self.step_wait()

    def state_dict(self) -> dict:
        return {"obs_rms": self.obs_rms.state_dict(), "ret_rms": self.ret_rms.state_dict()}

    def load_state_dict(self, d: dict) -> None:
        if self.obs_rms is None:
            dev = d["obs_rms"]["mean"].device
            self.obs_rms = DeviceRunningMeanStd(shape=d["obs_rms"]["mean"].shape, device=dev)
            self.ret_rms = DeviceRunningMeanStd(shape=(), device=dev)
            self.returns = torch.zeros(self.num_envs, dtype=torch.float64, device=dev)
        self.obs_rms.load_state_dict(d["obs_rms"])
        self.ret_rms.load_state_dict(d["ret_rms"])


# the methods that the kernels stand in for, unless a subclass, an instance or
# a patched class has others
_UPDATE = {n: getattr(DeviceRunningMeanStd, n) for n in ("update", "update_from_moments")}
_NORMALIZE = {n: getattr(DeviceVecNormalize, n) for n in ("normalize_obs", "normalize_reward")}


def _replaced(obj, methods) -> bool:
    return any(n in vars(obj) or getattr(type(obj), n) is not f for n, f in methods.items())
