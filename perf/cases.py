"""Performance cases of the trajectory engine: what a program has it do, through the Python binding.

Every case is one whole call chain of the binding (reset, launch, results back on the host) on an
engine, a solar model and parameter points that the program already holds.  The seed picks the
draw-stream key and the trajectory ids, so another seed means other trajectories.

Four kinds of call:
  run        Engine.run over one or several points, then the accumulated results of each point
  generate   Engine.generate, the run driver behind the command line: rounds until sample_size
             captures
  records    Engine.run_records, one record per trajectory on the host
  noalloc    Engine.run_records_noalloc, records and histograms into buffers on the GPU

The trajectories are a Monte Carlo whose decisions amplify every rounding (see `exact`), so an
implementation in plain torch or numpy does not give the same values.
"""
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "damascus-earth-evap_b200"))
import dms_b200  # noqa: E402

# Parameter points with the mean work of one trajectory: (mass [GeV], sigma [cm^2]) ->
# accepted free steps and scatterings per trajectory in Capture mode.
CAPTURE_WORK = {(0.1, 1e-39): (61, 0.001), (0.1, 1e-33): (75, 3.2), (0.3, 1e-36): (56, 0.39), (1.0, 1e-35): (47, 0.79),
                (3.0, 1e-38): (60, 0.025)}
# The same for whole evaporation histories (Parameter-point mode).
POINT_WORK = {(0.1, 1e-36): (115, 1.3), (0.1, 1e-35): (355, 11.7), (0.3, 1e-36): (232, 4.8)}
# Heavier particles stay bound for 10^5 scatterings and more: their runs are cut off by
# max_scatterings, and about half of the trajectories reach it at some 25 steps per scattering.
CAPPED_POINTS = ((1.0, 1e-35), (3.0, 1e-35))
# The 20-point grid of the benchmark: masses [GeV] x cross sections [cm^2].
GRID = [(m, s) for m in (0.1, 0.3, 1.0, 3.0) for s in (1e-39, 1e-38, 1e-37, 1e-36, 1e-35)]
# Counted FP64 operations per RK45 attempt (1.4 per step), free step, scattering and trajectory.
FLOP_STEP, FLOP_SCATTER, FLOP_TRAJECTORY = 1.4 * 215 + 622, 2455, 3374


def case(kind, mass, sigma, count, **more):
    """A case: `count` trajectories (for "generate": captures wanted) of one point (for "grid", of each point)."""
    c = {"kind": kind, "mass_gev": mass, "sigma_cm2": sigma, "count": count, "capture_mode": True, "mixed": False,
         "max_scatterings": 1000000, "grid_n": 1000, "dark_photon": False, "scan": False}
    c.update(more)
    return c


def listed():
    return [
        # a handful of trajectories replayed and looked at one by one: the smallest call
        case("records", 1.0, 1e-35, 64, name="records_64", max_scatterings=100000),
        # histories with their own radial histograms, kept on the GPU by a program with a fixed
        # memory budget; an odd count
        case("noalloc", 0.3, 1e-36, 127, name="histories_127", capture_mode=False, grid_n=200),
        # the Capture configuration: 16384 trajectories, cut at 1e5 scatterings
        case("run", 1.0, 1e-35, 16384, name="capture_16k", max_scatterings=100000),
        # the launch that keeps every lane busy
        case("run", 0.3, 1e-36, 1048576, name="capture_1m"),
        # a capture-rate scan: 20 points in one launch, a ragged number of trajectories each
        case("run", 0.0, 0.0, 10007, name="capture_scan_20", scan=True, max_scatterings=100000),
        # the run driver in Capture mode: rounds of the captures still missing
        case("generate", 1.0, 1e-35, 1000, name="generate_capture_1000", max_scatterings=100000),
        # evaporation histories (the Parameter-point configuration): a round of the run driver ...
        case("run", 0.3, 1e-36, 2048, name="point_2k", capture_mode=False),
        # ... and a batch
        case("run", 0.3, 1e-36, 16384, name="point_16k", capture_mode=False),
        # a heavy particle, cut off after 300 scatterings: every captured one is as long as the others
        case("run", 1.0, 1e-35, 4096, name="point_capped_4k", capture_mode=False, max_scatterings=300),
        # the mixed-precision form: every lane busy, and a batch of histories
        case("run", 0.3, 1e-36, 1048576, name="capture_mixed_1m", mixed=True),
        case("run", 0.3, 1e-36, 16384, name="point_mixed_16k", mixed=True, capture_mode=False),
        # the dark photon's General form factor
        case("run", 0.1, 1e-36, 16384, name="capture_dark_photon_16k", dark_photon=True),
    ]


def draw(rng):
    def sized(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["records", "noalloc", "generate", "scan", "point", "point", "capped", "capture", "capture", "capture"])
    mixed = rng.random() < 0.3
    grid_n = rng.choice([200, 300, 400, 1000, 1000])
    m, s = rng.choice(sorted(CAPTURE_WORK))
    if kind == "records":
        return case("records", m, s, sized(1, 1024), mixed=mixed, grid_n=grid_n, max_scatterings=100000)
    if kind == "noalloc":
        return case("noalloc", m, s, rng.randint(1, 128), grid_n=grid_n, max_scatterings=100000)
    if kind == "generate":
        return case("generate", 1.0, 1e-35, sized(100, 1000), grid_n=grid_n, max_scatterings=100000)
    if kind == "scan":
        return case("run", 0.0, 0.0, sized(500, 10000), scan=True, mixed=mixed, max_scatterings=100000)
    if kind == "point":
        m, s = rng.choice(sorted(POINT_WORK))
        return case("run", m, s, sized(64, 16384), capture_mode=False, mixed=mixed, grid_n=grid_n)
    if kind == "capped":
        m, s = rng.choice(CAPPED_POINTS)
        return case("run", m, s, sized(256, 4096), capture_mode=False, mixed=mixed, grid_n=grid_n,
                    max_scatterings=rng.randint(50, 300))
    return case("run", m, s, sized(256, 1000000), mixed=mixed, grid_n=grid_n)


_engine = None
_points = {}


def engine():
    """The process's engine context: a program creates one and keeps it."""
    global _engine
    if _engine is None:
        _engine = dms_b200.Engine(torch.cuda.current_device())
    return _engine


def point(mass, sigma, grid_n, dark_photon):
    """The point's id; its rate grid is built when it is first asked for."""
    key = (mass, sigma, grid_n, dark_photon)
    if key not in _points:
        if dark_photon:
            p = dms_b200.point_params(mass, 0.0, sigma_e_cm2=sigma, interpolation_points=grid_n,
                                      interaction=dms_b200.INTERACTION_DARK_PHOTON_GENERAL, mediator_mass_mev=1.0)
        else:
            p = dms_b200.point_params(mass, sigma, interpolation_points=grid_n)
        _points[key] = engine().add_point(p)
    return _points[key]


def prepare(case, seed):
    e = engine()
    if case["scan"]:
        points = [point(m, s, case["grid_n"], False) for m, s in GRID]
    else:
        points = [point(case["mass_gev"], case["sigma_cm2"], case["grid_n"], case["dark_photon"])]
    first = (seed % 65521) * 2097152
    opts = dms_b200.run_opts(seed=seed % (1 << 31), capture_mode=case["capture_mode"], max_scatterings=case["max_scatterings"],
                             precision=dms_b200.PRECISION_MIXED if case["mixed"] else dms_b200.PRECISION_FP64)
    state = {"case": case, "engine": e, "points": points, "first": first, "opts": opts, "seed": seed % (1 << 31)}
    if case["kind"] == "noalloc":
        import ctypes
        size = ctypes.sizeof(dms_b200.TrajRecord)
        state["records"] = torch.zeros(case["count"], size, dtype=torch.uint8, device="cuda")
        state["hists"] = torch.zeros(2, case["count"], dms_b200.NUM_BINS, dtype=torch.float64, device="cuda")
    return state


RECORD = np.dtype([("ids", "<u8"), ("scatterings", "<u8"), ("draws", "<u8"), ("point", "<u4"), ("reason", "<u4"), ("flags", "<u4"),
                   ("reserved", "<u4"), ("values", "<f8", (22,))])


def accumulated(per_point, first, count):
    """The results of one or several points as arrays; lifetimes and reflections by trajectory (-1 for the others)."""
    counters, columns = [], {}
    for k, r in enumerate(per_point):
        c = dict(r["counters"])
        reasons = c.pop("reasons")
        counters.append([c[k] for k in sorted(c)] + list(reasons))
        for name in ("events", "reflections"):
            if name in r:
                for f in r[name].dtype.names[1:]:
                    column = columns.setdefault(f, np.full((len(per_point), count), -1.0))
                    column[k, r[name]["trajectory_id"] - np.uint64(first + 1)] = r[name][f]
    return {"counters": np.array(counters, dtype=np.int64), "histograms": np.stack([r["histograms"] for r in per_point]), **columns}


def run(state):
    case, e, count = state["case"], state["engine"], state["case"]["count"]
    if case["kind"] == "records":
        r = e.run_records(state["points"][0], state["first"], count, state["opts"])["records"]
        a = np.frombuffer(r, dtype=RECORD)
        return {"whole": np.stack([a[f].astype(np.int64) for f in ("ids", "scatterings", "draws", "reason", "flags")]), "values": a["values"]}
    if case["kind"] == "noalloc":
        dt, v2dt = state["hists"]
        e.run_records_noalloc(state["points"][0], state["first"], count, state["opts"], state["records"].data_ptr(), dt.data_ptr(),
                              v2dt.data_ptr())
        words = state["records"].view(torch.int64)
        return {"whole": words[:, :5], "values": state["records"].view(torch.float64)[:, 5:], "hists": state["hists"]}
    if case["kind"] == "generate":
        p = state["points"][0]
        g = e.generate(p, count, seed=state["seed"], capture_mode=case["capture_mode"], max_scatterings=case["max_scatterings"],
                       sigma_p_cm2=case["sigma_cm2"])
        r = e.results(p)
        # Capture mode has no events
        return {"rounds": g["rounds"], "results": accumulated([r], 0, 1)}
    for p in state["points"]:
        e.reset_results(p)
    e.run([(p, state["first"], count) for p in state["points"]], state["opts"])
    # histories come with the reflected particles, whose spectrum the program forms
    reflections = 0 if case["capture_mode"] else count
    return accumulated([e.results(p, reflections_capacity=reflections) for p in state["points"]], state["first"], count)


def work(case):
    """Counted operations of the trajectories (means of the point), and the bytes of what comes back."""
    def per_trajectory(m, s):
        if case["dark_photon"]:
            steps, scatterings = 65, 2.7
        elif case["capture_mode"]:
            steps, scatterings = CAPTURE_WORK.get((m, s), (55, 0.5))
        elif (m, s) in CAPPED_POINTS:
            scatterings = 0.52 * case["max_scatterings"]
            steps = 47 + 25 * scatterings
        else:
            steps, scatterings = POINT_WORK[(m, s)] if (m, s) in POINT_WORK else CAPTURE_WORK[(m, s)]
        return steps * FLOP_STEP + scatterings * FLOP_SCATTER + FLOP_TRAJECTORY

    n = case["count"]
    points = GRID if case["scan"] else [(case["mass_gev"], case["sigma_cm2"])]
    if case["kind"] == "generate":
        n = 2 * n  # half of the trajectories are captured at this point
    flops = sum(n * per_trajectory(m, s) for m, s in points)
    out = 8 * dms_b200.NUM_BINS * 8 + 32 * 8
    if case["kind"] in ("records", "noalloc"):
        out = n * (216 + (16 * dms_b200.NUM_BINS if case["kind"] == "noalloc" else 0))
    # 9 radial tables of 1968 knots, 12 reachable columns of the rate grid per point
    return {"bytes": float(len(points) * (out + 8 * 12 * case["grid_n"]) + 9 * 8 * 1968), "flops": float(flops)}


def exact(case, seed):
    """No case has a value in plain 64-bit numpy or torch.  A trajectory is a chain of decisions
    (steps that land on the solar surface or beside it, scatterings accepted or not) that turns a
    different last bit into another trajectory, and the engine's values are defined by their order
    of operations; a Python loop over the steps would also take far longer than the engine."""
    return None
