"""The engine's host code (csrc/dms_capi.cu, dms_driver.cpp) without a GPU: linked with stand-ins for the CUDA
runtime and for the kernels (tests/fake), which write down what is launched and in what order."""
import os
import subprocess
import sys

import pytest

from dms_ctypes import PACKAGE_DIR, REPO

TESTS = os.path.dirname(os.path.abspath(__file__))
FAKE = os.path.join(TESTS, "fake")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PRELUDE = r"""
import ctypes, sys
sys.path.insert(0, %(pkg)r)
import numpy as np
import dms_b200
class Launch(ctypes.Structure):
    _fields_ = [("total", ctypes.c_uint64), ("done", ctypes.c_uint64), ("parked_room", ctypes.c_uint64)] + [
        (n, ctypes.c_int32) for n in ("blocks", "threads", "mixed", "resume", "lanes_per_block", "lockstep_min")] + [
        ("queue_chunk", ctypes.c_uint32), ("parked_capacity", ctypes.c_uint32), ("options", ctypes.c_int32 * 6)]
lib = dms_b200.library()
def launches():
    a = (Launch * 4096)()
    return list(a[:lib.fake_take_launches(a, 4096)])
def violations():
    text = ctypes.create_string_buffer(4096)
    return lib.fake_violations(text, 4096), text.value.decode()
rate = ctypes.c_double.in_dll(lib, "fake_rate")
def point(e, **kw):
    return e.add_point(dms_b200.point_params(0.3, 1e-36, **dict(dict(interpolation_points=20), **kw)))
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """Runs a script on the engine linked with the stand-ins."""
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    d = tmp_path_factory.mktemp("host")
    objects = [os.path.join(PACKAGE_DIR, "_build", n) for n in ("dms_capi.o", "dms_host_model.o", "dms_driver.o")]
    subprocess.run(["make", "-C", PACKAGE_DIR] + objects, check=True, stdout=subprocess.DEVNULL)
    include = ["-I", os.path.join(REPO, "include"), "-I", os.path.join(PACKAGE_DIR, "csrc"), "-I", "/usr/local/cuda/include"]
    kernels, runtime, library = (str(d / n) for n in ("kernels.o", "runtime.o", "libhost.so"))
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-Xcompiler", "-fPIC", "-w"] + include +
                   ["-c", "-o", kernels, os.path.join(FAKE, "kernels.cu")], check=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC"] + include + ["-c", "-o", runtime, os.path.join(FAKE, "cuda_runtime.cpp")], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", library, kernels, runtime] + objects + ["-ldl", "-lpthread"], check=True)

    def run(code):
        p = subprocess.run([sys.executable, "-c", PRELUDE % {"pkg": PACKAGE_DIR} + code], env=dict(os.environ, DMS_LIBRARY=library),
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-4000:]
        return p.stdout
    return run


def test_no_launch_overtakes_a_write_of_the_legacy_stream(host):
    """The engine's stream is a non-blocking one: what the host code writes on the legacy stream has to be waited for."""
    host(r"""
e = dms_b200.Engine(0)
def ordered(what):
    n, text = violations()
    assert n == 0, (what, text)
small = dms_b200.run_opts(seed=1, capture_mode=True, max_scatterings=10)
pid = point(e)
e.run([(pid, 0, 64)], small)
ordered("first run")
for k in range(9):  # past the first allocation of points
    pid = point(e, interpolation_points=0 if k == 4 else 20)
    e.run([(pid, 0, 64)], small)
    ordered("run after add_point")
e.rate(pid, np.array([1e5, 2e5]), np.array([300.0, 400.0]))
ordered("rate query")
e.set_rate_grid(pid, np.zeros((20, 20)))
e.run([(pid, 0, 64)], dms_b200.run_opts(seed=1, precision=dms_b200.PRECISION_MIXED))
ordered("run after set_rate_grid")
e.run_records(pid, 0, 3, small)
ordered("records")
e.reset_results(pid)
e.run([(pid, 0, 40000)], small)
ordered("large run after reset_results")
e.autotune([(pid, 0, 100)], small, trial_seconds=0.001)
ordered("autotune")
buffer = (ctypes.c_char * (ctypes.sizeof(dms_b200.TrajRecord) * 4))()
pid = point(e)
e.run_records_noalloc(pid, 0, 4, small, ctypes.addressof(buffer))
ordered("no-alloc records after add_point")
e.close()
""")


def test_parked_states_have_room(host):
    """A large launch hands at most lockstep_min lanes of each block to the launch behind it."""
    host(r"""
e = dms_b200.Engine(0)
pid = point(e)
for precision in (dms_b200.PRECISION_FP64, dms_b200.PRECISION_MIXED):
    for count in (128 * 148 + 1, 512 * 148, 2 * 640 * 148):
        e.run([(pid, 0, count)], dms_b200.run_opts(seed=1, precision=precision))
        first, second = launches()
        assert (first.resume, second.resume) == (0, 1) and second.threads == 128
        for l in (first, second):
            assert l.parked_capacity * 1024 <= l.parked_room
            assert l.parked_capacity >= first.blocks * first.lockstep_min
        assert second.blocks * second.threads >= second.parked_capacity
e.run([(pid, 0, 128 * 148)], dms_b200.run_opts(seed=1))
only, = launches()
assert only.threads == 128 and not only.resume
e.close()
""")


@pytest.mark.parametrize("per_second, seconds", [(2 ** 17 / 0.1, 0.1), (2 ** 21 / 0.1, 0.1), (2 ** 24 / 0.1, 0.1), (2 ** 26 / 0.4, 0.8)])
def test_autotuner_times_the_steady_state_of_different_launches(host, per_second, seconds):
    """No setting is timed on a launch whose queue has run dry, and none that is the launch of the best one so far."""
    host("per_second, seconds = %r, %r" % (per_second, seconds) + r"""
rate.value = per_second
e = dms_b200.Engine(0)
pid = point(e)
tuned, trials = e.autotune([(pid, 0, 100)], dms_b200.run_opts(seed=1), trial_seconds=seconds)
trial = [l for l in launches() if not l.resume]
assert len(trial) == trials
form = lambda l: (l.threads, l.queue_chunk) + tuple(l.options)
base = form(trial[0])
sized = [l for l in trial if form(l) == base]
others = trial[len(sized):]
# every setting runs at the same speed here: the base stays the best, and nothing but it is launched twice in a pass
assert all(form(l) != base for l in others)
assert len(others) >= 8 and len(set(map(form, others))) == len(others)
assert dms_b200.lane_options(tuned) == dms_b200.lane_options(dms_b200.run_opts(seed=1))
assert len(set(l.total for l in others)) == 1 and others[0].total <= 2 ** 25
assert sized[-1].done <= others[0].total // 2
assert all(l.done < l.total for l in others)
e.close()
""")


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_a_batch_that_is_set_is_the_same_share_of_a_warp_and_of_a_block(host, precision):
    host("precision = dms_b200.PRECISION_%s" % precision + r"""
e = dms_b200.Engine(0)
pid = point(e)
for count in (100, 100000):
    for scatter, final in ((1, 1), (32, 32), (8, 3)):
        e.run([(pid, 0, count)], dms_b200.run_opts(seed=1, precision=precision, scatter_batch=scatter, final_batch=final,
                                                   scatter_wait=5, final_wait=1024))
        for l in launches():
            assert tuple(l.options) == (scatter, 5, final, 1024, 2 * scatter, 2 * final)  # of 32 lanes, of 64
e.close()
""")


def test_a_large_mixed_launch_takes_the_rows_that_there_is_memory_for(host):
    """640 lanes per SM need 3.0 GB of histogram rows; where only the 2.4 GB of 512 are there, 512 run."""
    host(r"""
limit = ctypes.c_size_t.in_dll(lib, "fake_malloc_limit")
row, wide = 2000 * 16, [(0, 0, 2 * 640 * 148)]
mixed = dms_b200.run_opts(seed=1, precision=dms_b200.PRECISION_MIXED)
e = dms_b200.Engine(0)
point(e)
for lanes in (512, 640):
    limit.value = lanes * 148 * row
    e.run(wide, mixed)
    first, second = launches()
    assert (first.threads, first.lanes_per_block) == (lanes, lanes)
limit.value = 128 * 148 * row
e = dms_b200.Engine(0)
point(e)
try:
    e.run(wide, mixed)
except dms_b200.EngineError as error:
    assert "CUDA error" in str(error)
else:
    raise AssertionError("ran without rows")
assert not launches()
""")
