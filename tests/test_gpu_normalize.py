"""DeviceVecNormalize's kernels (arc_norm_step) against its tensor operations
on the same batches: one column, ragged tiles of 256 columns and blocks of 32
rows, every combination of its switches, values that are not finite."""

import itertools

import pytest
import torch

from arc_demo_b200.vec_env import DeviceRunningMeanStd, DeviceVecNormalize

pytestmark = pytest.mark.gpu


class Env:
    """Random batches (column 0 constant), the same for the same seed."""

    def __init__(self, n, cols, bad=False):
        self.num_envs, self.cols, self.bad = n, cols, bad
        self.g = torch.Generator(device="cuda").manual_seed(1000 * n + cols)

    def _obs(self):
        x = torch.randn((self.num_envs, self.cols), device="cuda", generator=self.g)
        x = x * torch.logspace(-3, 3, self.cols, device="cuda") + torch.linspace(-50, 50, self.cols, device="cuda")
        x[:, 0] = 7.25
        if self.bad:
            x[0, 1], x[1, 2], x[2, 3] = float("inf"), float("nan"), float("-inf")
        return x

    def reset(self):
        return self._obs()

    def step_async(self, actions):
        pass

    def step_wait(self):
        r = torch.randn(self.num_envs, device="cuda", generator=self.g) * 3 + 1
        d = torch.rand(self.num_envs, device="cuda", generator=self.g) < 0.2
        return self._obs(), r, d, {"terminal_observation": self._obs(), "truncated": d}


class Tensors(DeviceVecNormalize):
    def _step_kernels(self, *a):
        return None


def _close(a, b, rel):
    assert a.dtype == b.dtype and a.shape == b.shape
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.allclose(a, b, rtol=rel, atol=rel, equal_nan=True), (a - b).abs().max()


@pytest.mark.parametrize("n,cols", [(1, 1), (2, 195), (33, 5), (1000, 195), (8195, 256), (300, 300), (40, 2048)])
@pytest.mark.parametrize("training,norm_obs,norm_reward", list(itertools.product([True, False], repeat=3)))
def test_kernels_equal_tensor_operations(n, cols, training, norm_obs, norm_reward):
    kw = dict(training=training, norm_obs=norm_obs, norm_reward=norm_reward)
    a, b = DeviceVecNormalize(Env(n, cols), **kw), Tensors(Env(n, cols), **kw)
    a.reset(), b.reset()
    assert a._step_kernels(a.old_obs, torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda").bool(), {})
    a = DeviceVecNormalize(Env(n, cols), **kw)  # that call was a step
    a.reset()
    kept = a.obs_rms.mean, a.obs_rms.mean.clone()
    for _ in range(4):
        x, y = a.step(None), b.step(None)
        # FP32 results of FP64 arithmetic: within an ulp (6e-8) and what the
        # 1e-11 of the statistics makes of values of up to 1e3 deviations
        for u, v in zip((x[0], x[1], x[3]["terminal_observation"]), (y[0], y[1], y[3]["terminal_observation"])):
            _close(u, v, 2e-7)
        assert torch.equal(x[2], y[2])
    # sums of up to 8,195 FP64 terms, 4 times: 8,195 x 1.1e-16 x a mean of up
    # to 50 deviations squared at most
    for u, v in ((a.obs_rms.mean, b.obs_rms.mean), (a.obs_rms.var, b.obs_rms.var), (a.ret_rms.mean, b.ret_rms.mean),
                 (a.ret_rms.var, b.ret_rms.var), (a.returns, b.returns)):
        _close(u, v, 1e-9)
    assert a.obs_rms.count == b.obs_rms.count and a.ret_rms.count == b.ret_rms.count
    assert torch.equal(*kept)  # statistics handed out before stay as they were


def test_values_that_are_not_finite():
    a, b = DeviceVecNormalize(Env(64, 8, bad=True)), Tensors(Env(64, 8, bad=True))
    a.reset(), b.reset()
    for _ in range(2):
        x, y = a.step(None), b.step(None)
        _close(x[0], y[0], 2e-7)
    _close(a.obs_rms.mean, b.obs_rms.mean, 1e-9)
    _close(a.obs_rms.var, b.obs_rms.var, 1e-9)


def test_other_tensors_take_the_tensor_operations():
    a = DeviceVecNormalize(Env(16, 6))
    a.reset()
    r, d = torch.zeros(16, device="cuda"), torch.zeros(16, device="cuda").bool()
    x = a.old_obs
    assert a._step_kernels(x, r, d, {}) is not None
    for obs, rew, done in ((x.t().contiguous().t(), r, d), (x.double(), r, d), (x, r.double(), d),
                           (x, r, d.to(torch.uint8)), (x.clone().requires_grad_(), r, d), (x[:8], r[:8], d[:8]),
                           (x.cpu(), r, d)):
        assert a._step_kernels(obs, rew, done, {}) is None


def test_overridden_normalisation_is_used():
    """A subclass's normalize_obs (or statistics of another class) decides, as
    in the tensor operations; statistics keep storages of their own."""
    class Half(DeviceVecNormalize):
        def normalize_obs(self, obs):
            return 0.5 * obs

    class Rms(DeviceRunningMeanStd):
        pass

    a = Half(Env(16, 6))
    a.reset()
    obs = a.step(None)[0]
    assert torch.equal(obs, 0.5 * a.old_obs)
    b = DeviceVecNormalize(Env(16, 6))
    b.reset()
    b.step(None)
    assert b.obs_rms.mean.untyped_storage().nbytes() == 6 * 8
    r, d = torch.zeros(16, device="cuda"), torch.zeros(16, device="cuda").bool()
    b.obs_rms = Rms(shape=(6,), device="cuda")
    assert b._step_kernels(b.old_obs, r, d, {}) is None
    b.obs_rms = DeviceRunningMeanStd(shape=(6,), device="cuda")
    with torch.autograd.forward_ad.dual_level():
        assert b._step_kernels(b.old_obs, r, d, {}) is None
    assert b._step_kernels(b.old_obs, r, d, {}) is not None


@pytest.mark.parametrize("n", [7, 4000, 8195])
def test_moments_do_not_lean_on_one_row(n):
    """A first (or any) row far out costs the other rows' moments nothing:
    the batch's mean and variance against 80-bit arithmetic. Per variance at
    most 33 rows in turn, 13 sums of lanes and blocks and 8 roundings beside
    them, each 2^-53 of the sum; per mean a quarter of that, of the largest
    summand's share."""
    import numpy as np

    g = np.random.default_rng(n)
    x = (g.normal(size=(n, 9)) * np.logspace(-3, 3, 9) + np.linspace(-50, 50, 9)).astype(np.float32)
    x[0] += np.array([0, 1, 10, 1e2, 1e3, 1e4, 1e5, 0, 0]) * x.std(0)
    x[n // 2, 7] += 1e5 * x[:, 7].std()
    x[:, 8] = 0.1
    a = DeviceVecNormalize(Env(n, 9))
    a.reset()
    a.obs_rms.count = a.ret_rms.count = 0.0  # the merged statistics are then the batch's
    a.returns = torch.as_tensor(np.concatenate([[1e5], g.normal(size=n - 1)]), device="cuda")
    r, d = torch.as_tensor(g.normal(size=n).astype(np.float32), device="cuda"), torch.zeros(n, device="cuda").bool()
    returns = a.returns.cpu().numpy() * a.gamma + r.cpu().numpy().astype(np.float64)
    assert a._step_kernels(torch.as_tensor(x, device="cuda"), r, d, {}) is not None
    for got, data in ((a.obs_rms, x), (a.ret_rms, returns[:, None])):
        data = data.astype(np.longdouble)
        mean = data.mean(0)
        var = ((data - mean) ** 2).mean(0)
        assert (np.abs(got.var.cpu().numpy() - var) <= 54 * 2.0**-53 * var).all()
        assert (np.abs(got.mean.cpu().numpy() - mean) <= 14 * 2.0**-53 * np.abs(data).mean(0)).all()
    assert a.obs_rms.var[8] == 0.0


def test_quotients_are_divisions():
    """(obs - mean) / deviation rounds once, as a division does: quotients
    halfway between two FP32 values (exact in FP64) round to the even one,
    which a product with the reciprocal misses by the last bit; infinities,
    NaN and deviations of zero as a division gives them."""
    bad = float("inf"), float("-inf"), float("nan"), 0.0, 1.0
    a = DeviceVecNormalize(Env(5, 900), training=False, norm_reward=False, clip_obs=float("inf"), epsilon=0.0)
    a.reset()
    dev = torch.arange(3, 1803, 2, dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    half = torch.randint(2**23, 2**24, (900,), device="cuda", generator=g).double() + 0.5
    a.obs_rms.mean, a.obs_rms.var = -half * dev, dev.square()
    a.obs_rms.mean[:10] = 0.0
    a.obs_rms.var[5:10] = 0.0
    x = torch.zeros((5, 900), device="cuda")
    x[:, :10] = torch.tensor(bad, device="cuda")[:, None]
    r, d = torch.zeros(5, device="cuda"), torch.zeros(5, device="cuda").bool()
    got = a._step_kernels(x, r, d, {})[0]
    assert torch.equal(got[:, 10:], half[10:].float().expand(5, -1))
    assert torch.equal(got.nan_to_num(7.0), a.normalize_obs(x).nan_to_num(7.0))


def test_replaced_methods_are_used(monkeypatch):
    """Functions set on the normaliser or its statistics, or patched into
    their classes, decide as they do for the tensor operations."""
    def fresh():
        a = DeviceVecNormalize(Env(16, 6))
        a.reset()
        return a

    a = fresh()
    a.normalize_obs = lambda obs: 0.5 * obs
    obs = a.step(None)[0]
    assert torch.equal(obs, 0.5 * a.old_obs)
    a = fresh()
    a.normalize_reward = lambda r: r + 1
    assert torch.equal(a.step(None)[1], a.old_reward + 1)
    for name in ("update", "update_from_moments"):
        for rms in ("obs_rms", "ret_rms"):
            a, calls = fresh(), []
            setattr(getattr(a, rms), name, lambda *x: calls.append(x))
            a.step(None)
            assert len(calls) == 1
    a, calls = fresh(), []
    monkeypatch.setattr(DeviceRunningMeanStd, "update", lambda self, x: calls.append(x))
    a.step(None)
    assert len(calls) == 2


@pytest.mark.parametrize("limit", [-1.0, float("nan")])
def test_limits_that_are_no_limits(limit):
    """Limits below zero, or NaN: what clamp makes of them."""
    kw = dict(clip_obs=limit, clip_reward=limit)
    a, b = DeviceVecNormalize(Env(33, 6), **kw), Tensors(Env(33, 6), **kw)
    a.reset(), b.reset()
    x, y = a.step(None), b.step(None)
    for u, v in zip(x[:3], y[:3]):
        assert torch.equal(u.nan_to_num(7.0), v.nan_to_num(7.0))


def test_traced_steps_take_the_tensor_operations():
    a, seen = DeviceVecNormalize(Env(16, 6)), []
    a.reset()
    r, d = torch.zeros(16, device="cuda"), torch.zeros(16, device="cuda").bool()
    torch.jit.trace(lambda x: x + 0 * len(seen.append(a._step_kernels(x, r, d, {})) or seen), a.old_obs,
                    check_trace=False)
    assert seen == [None]
