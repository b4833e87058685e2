"""The forms that a trajectory can go through are taken where the other tests mean them to be (B200 required).

The checked build counts them: teams of a lone lane and their steps, warps that stopped waiting for a team, and
trajectories handed from a large launch to the one behind it.  It waits for a team for some 50 ms only, not
20 s.  The library is loaded in a child process, since one process holds one engine library."""
import os
import subprocess
import sys

import pytest

from dms_ctypes import PACKAGE_DIR

pytestmark = pytest.mark.gpu

CHECKED = os.path.join(PACKAGE_DIR, "libdms_cuda_checked.so")
TESTS = os.path.dirname(os.path.abspath(__file__))

PRELUDE = r"""
import ctypes, sys
sys.path.insert(0, %(tests)r)
sys.path.insert(0, %(pkg)r)
import dms_b200
from engine_fixtures import REPLAY_POINT
SMS = 148
precision = dms_b200.PRECISION_%(precision)s
e = dms_b200.Engine(0)
pid = e.add_point(dms_b200.point_params(**REPLAY_POINT))
def opts(**kw):
    return dms_b200.run_opts(seed=11, precision=precision, **kw)
def forms():
    a = (ctypes.c_ulonglong * 5)()
    assert e.lib.dms_checked_form_counts(e.h, precision, a) == 0
    return dict(zip(("teams", "team_steps", "gave_up", "parked", "resumed"), a))
forms()
"""


def run(precision, code):
    if not os.path.exists(CHECKED):
        pytest.skip("checked library not built (make checked)")
    p = subprocess.run([sys.executable, "-c", PRELUDE % {"tests": TESTS, "pkg": PACKAGE_DIR, "precision": precision} + code],
                       env=dict(os.environ, DMS_LIBRARY=CHECKED), capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-4000:]


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_a_lone_lane_gets_a_team(precision):
    run(precision, r"""
o = opts(max_scatterings=200)
steps = 0
for first in range(3000, 3012):
    e.reset_results(pid)
    e.run([(pid, first, 1)], o)
    steps += e.results(pid)["counters"]["rk_steps"]
f = forms()
print(f, steps)
assert f["teams"] == 12 and f["parked"] == 0 and f["gave_up"] == 0
assert 0.5 * steps < f["team_steps"] <= steps
o.max_trajectory_wall_time_s = 1e6
e.run([(pid, 3000, 12)], o)
assert forms()["teams"] == 0
""")


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_a_large_launch_parks_its_last_trajectories(precision):
    run(precision, r"""
for capture in (True, False):
    for count, chunk in ((128 * SMS + 1, 0), (1024 * SMS, 0), (128 * SMS + 1, 7), (2 * 640 * SMS, 0)):
        e.run([(pid, 10 ** 6, count)], opts(capture_mode=capture, max_scatterings=20, queue_chunk=chunk))
        f = forms()
        print(capture, count, chunk, f)
        assert f["parked"] == f["resumed"] and 0 < f["parked"] <= 64 * SMS
e.run([(pid, 10 ** 6, 128 * SMS)], opts(capture_mode=True, max_scatterings=20))
assert forms()["parked"] == 0
""")


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_helpers_wait_while_their_block_makes_steps(precision):
    """Two lanes in each block, for longer than a warp without work waits for a block that shows no life."""
    run(precision, r"""
heavy = e.add_point(dms_b200.point_params(1.0, 1e-35, interpolation_points=200))
e.run([(heavy, 0, 2 * SMS)], opts(max_scatterings=2000))
f = forms()
print(f, e.last_kernel_ms())
assert e.last_kernel_ms() > 200.0  # four times as long as the wait
assert f["teams"] > 0 and f["gave_up"] == 0
""")
