"""Histograms, batches of claimed ids and stops in the forms that a launch takes (B200 required).

A trajectory's radial histogram passes through whatever makes its steps: a lane of a large launch, the launch that
resumes it when it was parked, a team's committing warp.  Its bins have to be the same bits in all of them.  And a
run that is stopped in any of them has to account for every trajectory and leave clean rows behind."""
import ctypes

import numpy as np
import pytest

from engine_fixtures import REPLAY_POINT, dms_b200

pytestmark = pytest.mark.gpu

SMS = 148
BOTH = pytest.mark.parametrize("precision", [dms_b200.PRECISION_FP64, dms_b200.PRECISION_MIXED], ids=["fp64", "mixed"])


@pytest.fixture(scope="module")
def engine():
    e = dms_b200.Engine(0)
    pid = e.add_point(dms_b200.point_params(**REPLAY_POINT))
    yield e, pid
    e.close()


def _opts(precision, **more):
    return dms_b200.run_opts(seed=11, precision=precision, **more)


def _all(e, pid, first, count, o):
    r = e.run_records(pid, first, count, o, histograms=True)
    size = ctypes.sizeof(dms_b200.TrajRecord)
    return np.frombuffer(r["records"], dtype=np.uint8).reshape(-1, size), r["hist_dt"], r["hist_v2dt"]


def _assert_same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@BOTH
@pytest.mark.parametrize("chunk", [0, 7])
def test_histograms_of_parked_trajectories(engine, precision, chunk):
    """Launches of 12 per SM (no second launch), against one that parks its last lanes; chunk 7: with claimed ids."""
    e, pid = engine
    first, count, part = 9_000_000, 128 * SMS + 301, 12 * SMS
    whole = _all(e, pid, first, count, _opts(precision, max_scatterings=30, queue_chunk=chunk))
    for at in range(0, count, part):
        n = min(part, count - at)
        _assert_same([x[at:at + n] for x in whole], _all(e, pid, first + at, n, _opts(precision, max_scatterings=30)))


@BOTH
@pytest.mark.parametrize("more", [dict(), dict(max_scatterings=3), dict(boundary_rsun=1.0), dict(boundary_rsun=30.0)])
def test_histograms_of_a_team(engine, precision, more):
    """A wall-time limit, here one that is never reached, keeps a lone lane to itself."""
    e, pid = engine
    base = dict(dict(max_scatterings=200), **more)
    alone = _opts(precision, **base)
    alone.max_trajectory_wall_time_s = 1e6
    for first in range(3_000, 3_012):
        _assert_same(_all(e, pid, first, 1, _opts(precision, **base)), _all(e, pid, first, 1, alone))


def _accounted(c):
    return c["trajectories"] + c["unfinished_trajectories"]


@BOTH
@pytest.mark.parametrize("count", [1, 3 * SMS, 128 * SMS + 301])
@pytest.mark.parametrize("stop", [dict(iteration_budget=2500), dict(time_limit_s=0.02)], ids=["budget", "time"])
def test_a_stopped_run_accounts_for_every_trajectory(engine, precision, count, stop):
    """Stopped in a lane loop, in a team's steps, or in the launch that resumes parked trajectories."""
    e, _ = engine
    heavy = e.add_point(dms_b200.point_params(1.0, 1e-35, interpolation_points=100))
    first = 0
    clean = _all(e, heavy, 500, 64, _opts(precision, max_scatterings=30))
    stopped = _opts(precision, max_scatterings=10 ** 5, **stop)
    if count == 1:  # a captured trajectory, which makes 10^6 steps
        first = next(k for k in range(100) if e.run_records(heavy, k, 1, _opts(precision, capture_mode=True, max_scatterings=10 ** 5))["records"][0].flags & 2)
    e.reset_results(heavy)
    with pytest.raises(dms_b200.EngineError, match="budget" if "iteration_budget" in stop else "cancelled"):
        e.run([(heavy, first, count)], stopped)
    c = e.results(heavy)["counters"]
    assert c["unfinished_trajectories"] > 0
    assert _accounted(c) == count
    assert c["unfinished_rk_steps"] > 0
    # the rows that the stopped lanes were filling are clean
    _assert_same(clean, _all(e, heavy, 500, 64, _opts(precision, max_scatterings=30)))
