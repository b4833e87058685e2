"""The forms a launch takes by its size, against one another (B200 required).

Which kernel runs a trajectory, with how many others in its warp, whether its last steps are made in a second launch
or by three warps together: none of it may change a bit of its record.  Each test runs the same ids in
two forms and compares the records byte for byte; the small form is the one that the replay tests hold
against the CPU oracle."""
import ctypes

import numpy as np
import pytest

from dms_ctypes import Oracle, point_params as oracle_point_params
from engine_fixtures import REPLAY_POINT, dms_b200, outcome, state

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.fixture(scope="module")
def engine():
    e = dms_b200.Engine(0)
    p = REPLAY_POINT
    pid = e.add_point(dms_b200.point_params(p["mass_gev"], p["sigma_p_cm2"], interpolation_points=p["interpolation_points"]))
    yield e, pid
    e.close()


def _bytes(records):
    size = ctypes.sizeof(dms_b200.TrajRecord)
    return np.frombuffer(records, dtype=np.uint8).reshape(-1, size)


def _opts(precision, **more):
    return dms_b200.run_opts(seed=11, precision=precision, **more)


@pytest.mark.parametrize("precision", [dms_b200.PRECISION_FP64, dms_b200.PRECISION_MIXED])
@pytest.mark.parametrize("capture", [True, False])
@pytest.mark.parametrize("count", [1, SMS - 1, SMS + 1, 128 * SMS, 128 * SMS + 1, 512 * SMS + 1])
def test_a_record_does_not_depend_on_the_size_of_its_launch(engine, precision, capture, count):
    e, pid = engine
    first = 5_000_000
    o = _opts(precision, capture_mode=capture, max_scatterings=100000 if capture else 20)
    whole = _bytes(e.run_records(pid, first, count, o)["records"])
    # the ends and a stretch in the middle, a few at a time: one lane per block, then three per block
    for at, n in ((0, min(count, 7)), (count // 2, min(count - count // 2, 3 * SMS)), (count - 1, 1)):
        part = _bytes(e.run_records(pid, first + at, n, o)["records"])
        assert np.array_equal(whole[at:at + n], part)


def test_the_wide_mixed_form_gives_the_same_records(engine):
    """From two trajectories per lane on, a mixed launch runs 640 threads per SM."""
    e, pid = engine
    o = _opts(dms_b200.PRECISION_MIXED, capture_mode=True, max_scatterings=100000)
    edge = 2 * 640 * SMS
    wide = _bytes(e.run_records(pid, 0, edge, o)["records"])
    assert np.array_equal(wide[:edge - 1], _bytes(e.run_records(pid, 0, edge - 1, o)["records"]))


@pytest.mark.parametrize("precision", [dms_b200.PRECISION_FP64, dms_b200.PRECISION_MIXED])
@pytest.mark.parametrize("more", [dict(), dict(max_scatterings=3), dict(max_free_steps=7), dict(boundary_rsun=1.0), dict(boundary_rsun=30.0)])
def test_a_team_makes_the_steps_of_a_lone_lane(engine, precision, more):
    """A wall-time limit, here one that is never reached, keeps the lane to itself."""
    e, pid = engine
    base = dict(max_scatterings=200)
    base.update(more)
    for first in range(3_000, 3_012):
        team = _bytes(e.run_records(pid, first, 1, _opts(precision, **base), histograms=False)["records"])
        o = _opts(precision, **base)
        o.max_trajectory_wall_time_s = 1e6
        assert np.array_equal(team, _bytes(e.run_records(pid, first, 1, o)["records"]))


@pytest.mark.parametrize("counts", [(1, 1, 1), (592, 1, 31), (593, 18944, 7)])
def test_initial_states_of_several_ranges(engine, counts):
    """One launch over ragged ranges, against a launch per range: the same trajectories, counted the same."""
    e, pid = engine
    o = _opts(dms_b200.PRECISION_FP64, capture_mode=True, max_scatterings=100000)
    ranges = [(pid, 1_000_000 * (k + 1), n) for k, n in enumerate(counts)]
    e.reset_results(pid)
    e.run(ranges, o)
    together = dict(e.results(pid)["counters"])
    e.reset_results(pid)
    for r in ranges:
        e.run([r], o)
    assert together == dict(e.results(pid)["counters"])


@pytest.mark.parametrize("rows", [1, 4])
def test_solar_table_with_several_knots_in_a_bucket(tmp_path, rows):
    """Rows put between two of the model's, 10^-5 R_sun apart, leave a bucket of the knot search with more than one
    knot: the interval is then searched for.  FP64 replays the oracle on that model (states to 1e-10); the mixed form
    keeps the capture fraction of FP64 within one binomial standard error, its gate on the unchanged model."""
    lines = open(dms_b200.SOLAR_MODEL).read().split("\n")
    at = next(i for i, l in enumerate(lines) if len(l.split()) > 30 and l.split()[0][0].isdigit() and float(l.split()[1]) >= 0.3)
    a, b = (np.array([float(x) for x in lines[i].split()]) for i in (at, at + 1))
    new = []
    for k in range(rows):
        row = a + (k + 1) * 1e-5 / (b[1] - a[1]) * (b - a)
        new.append(" ".join("%.7f" % x if c < 2 else "%.6e" % x for c, x in enumerate(row)))
    path = tmp_path / "dense.dat"
    path.write_text("\n".join(lines[:at + 1] + new + lines[at + 1:]))
    oracle = Oracle(str(path))
    oracle.set_point(oracle_point_params(1.0, 1e-35, interpolation_points=100))
    with dms_b200.Engine(0, solar_model=str(path)) as e:
        assert len(e.solar_table(0)) == len(oracle.tables()["r"])
        pid = e.add_point(dms_b200.point_params(1.0, 1e-35, interpolation_points=100))
        e.set_rate_grid(pid, oracle.rate_grid())
        x = e.run_records(pid, 0, 64, _opts(dms_b200.PRECISION_FP64, capture_mode=True, max_scatterings=1000))["records"]
        y = oracle.run_records(11, pid, 0, 64, capture_mode=True, max_scatterings=1000)["records"]
        for p, q in zip(x, y):
            assert outcome(p) == outcome(q)
            assert np.allclose(state(p), state(q), rtol=1e-10, atol=0.0)
        n, fraction = 8192, []
        for precision in (dms_b200.PRECISION_FP64, dms_b200.PRECISION_MIXED):
            e.reset_results(pid)
            e.run([(pid, 0, n)], _opts(precision, capture_mode=True, max_scatterings=1000))
            fraction.append(e.results(pid)["counters"]["captured"] / n)
        assert abs(fraction[0] - fraction[1]) <= np.sqrt(fraction[0] * (1 - fraction[0]) / n)
