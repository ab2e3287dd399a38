"""The library's host code on a runtime without a GPU (fake_cudart.cpp, linked
with the library's own objects): read-outs of one sim by several threads, and
arguments that must not reach a kernel."""

import ctypes
import subprocess
import threading
from pathlib import Path

import numpy as np
import pytest

from arc_demo_b200.build import BUILD, build, nvcc, sources
from arc_demo_b200.task import ENDED_DIFFICULTY, REWARD, TASK_STATE_SIZE
from arc_demo_b200.vec_env import _NormArgs

_vp, _int = ctypes.c_void_p, ctypes.c_int


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    objs = [BUILD / (s.stem + ".o") for s in sources()]
    if not all(o.exists() for o in objs):
        build()
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    include = Path(nvcc()).resolve().parent.parent / "include"
    # -Bsymbolic: not another CUDA runtime of this process
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{include}", "-o", str(out),
                    str(Path(__file__).parent / "fake_cudart.cpp"), *map(str, objs), "-lpthread", "-ldl", "-lrt"],
                   check=True, capture_output=True)
    lib = ctypes.CDLL(str(out))
    lib.arc_sim_create.restype = _vp
    lib.arc_sim_create.argtypes = [_int, ctypes.c_double, _int, _int, ctypes.c_double]
    lib.arc_sim_destroy.argtypes = [_vp]
    lib.arc_env_init.argtypes = [_vp, _vp, ctypes.c_ulonglong]
    lib.arc_env_upload.argtypes = lib.arc_env_download.argtypes = [_vp, _int, _vp]
    lib.arc_env_get_task_state.argtypes = [_vp, _vp, _int, _vp]
    return lib


@pytest.fixture
def sim(lib):
    s = lib.arc_sim_create(64, 1.0 / 30.0, 20, 64, 0.4)
    assert s and lib.arc_env_init(s, None, 1) == 0
    yield s
    lib.fake_delay_us(0)
    lib.arc_sim_destroy(s)


def _at_once(*calls):
    start = threading.Barrier(len(calls))

    def go(call):
        start.wait()
        call()
    threads = [threading.Thread(target=go, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()


def test_two_threads_read_their_own_arrays(lib, sim):
    want = {REWARD: np.full(64, 1.0, np.float32), ENDED_DIFFICULTY: np.full(64, 2.0)}
    for which, a in want.items():
        assert lib.arc_env_upload(sim, which, a.ctypes.data) == 0
    wrong = []

    def read(which):
        for _ in range(20):
            got = np.zeros_like(want[which])
            if lib.arc_env_download(sim, which, got.ctypes.data) or not np.array_equal(got, want[which]):
                wrong.append(which)
    lib.fake_delay_us(500)
    _at_once(lambda: read(REWARD), lambda: read(ENDED_DIFFICULTY))
    assert not wrong


def test_two_threads_read_task_rows(lib, sim):
    """No thread's rows or ids lie in memory that another thread's larger
    request has given back."""
    def read(n):
        ids, out = np.arange(n, dtype=np.int32), np.zeros((n, TASK_STATE_SIZE))
        assert lib.arc_env_get_task_state(sim, ids.ctypes.data, n, out.ctypes.data) == 0
    before = lib.fake_launches()
    lib.fake_delay_us(500)
    _at_once(lambda: [read(n) for n in range(1, 64, 2)], lambda: [read(n) for n in range(2, 65, 2)])
    assert lib.fake_launches() == before + 64 and lib.fake_with_freed_memory() == 0


def test_rows_are_gathered_on_the_sims_device(lib, sim):
    """A thread whose current device is another one reads what it did with
    plain copies, and keeps its device."""
    out, device = np.zeros((64, TASK_STATE_SIZE)), _int()
    ids = np.arange(64, dtype=np.int32)
    lib.cudaSetDevice(1)
    try:
        before = lib.fake_launches(), lib.fake_on_other_device()
        assert lib.arc_env_get_task_state(sim, ids.ctypes.data, 64, out.ctypes.data) == 0
        lib.cudaGetDevice(ctypes.byref(device))
    finally:
        lib.cudaSetDevice(0)
    assert (lib.fake_launches(), lib.fake_on_other_device()) == (before[0] + 1, before[1])
    assert device.value == 1


@pytest.mark.parametrize("training,norm_obs,norm_reward,needs", [
    (1, 1, 1, "obs_mean obs_var ret_mean ret_var obs_mean_out obs_var_out ret_mean_out ret_var_out rewards_out"),
    (1, 0, 0, "ret_mean ret_var ret_mean_out ret_var_out"),
    (0, 1, 1, "obs_mean obs_var ret_var rewards_out"),
    (0, 0, 0, "")])
def test_normalisation_refuses_missing_statistics(lib, training, norm_obs, norm_reward, needs):
    """arc_norm_step without a pointer that its kernels would follow."""
    always = ("obs", "rewards", "dones", "returns", "returns_out", "work")
    a = _NormArgs(rows=4, cols=3, training=training, norm_obs=norm_obs, norm_reward=norm_reward)
    for name in (*always, *needs.split()) + (("obs_out", "terminal_obs", "terminal_out") if norm_obs else ()):
        setattr(a, name, 4096)
    assert lib.arc_norm_step(ctypes.byref(a), None) == 0
    for name in (*always, *needs.split()):
        b = _NormArgs.from_buffer_copy(a)
        setattr(b, name, None)
        assert lib.arc_norm_step(ctypes.byref(b), None) != 0, name
