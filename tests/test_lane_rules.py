"""The rules of the lane loop that need no GPU (csrc/dms_lane_rules.h), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

from dms_ctypes import PACKAGE_DIR, REPO

SHIM = r"""
#include <cstdint>
#include "dms_lane_rules.h"
#include "dms_math.h"
extern "C" {
int vote_sets() { return dms::lane::VOTE_SETS; }
int next_vote_set(int set) { return dms::lane::next_vote_set(set); }
int rare_phase_due(int* passes, int waiting, int stepping, int batch, int per, int wait, int lanes, int full)
{
	return dms::lane::rare_phase_due(*passes, waiting, stepping, batch, per, wait, lanes, full);
}
}

struct V { double x, y, z; };
static double dot(const V& a, const V& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
static V cross(const V& a, const V& b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
static V unit(const V& a) { const double n = sqrt(dot(a, a)); return {a.x / n, a.y / n, a.z / n}; }
static uint64_t seed_;
static double uniform(double a, double b)
{
	uint64_t x = seed_ += 0x9e3779b97f4a7c15ULL;
	x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
	x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
	return a + (b - a) * (static_cast<double>((x ^ (x >> 31)) >> 11) * 0x1p-53);
}

// States outside the surface, down to grazing ones, with steps about the time to the surface: how many of those that
// the radial speed calls far does the event's time to the surface bind all the same (*wrong)?  Returns how many it calls far.
extern "C" int far_from_surface(int n, uint64_t seed, int* wrong)
{
	seed_ = seed;
	int far = 0;
	*wrong = 0;
	for(int i = 0; i < n; i++)
	{
		// axes as prop_init makes them
		V ax = unit({uniform(-1, 1), uniform(-1, 1), uniform(-1, 1)});
		const V az = unit(cross(ax, {uniform(-1, 1), uniform(-1, 1), uniform(-1, 1)}));
		const V ay = unit(cross(az, ax));
		ax = unit(cross(ay, az));
		const double r = DMS_RSUN_KM * (1.0 + pow(10.0, uniform(-9, 0))), J = r * uniform(10.0, 2000.0), v_radial = -pow(10.0, uniform(-8, 3));
		double sp, cp;
		dms_sincos(uniform(0.0, 100.0), &sp, &cp);
		const double vt = J / r, vx = v_radial * cp - vt * sp, vy = v_radial * sp + vt * cp;
		const V x = {r * (cp * ax.x + sp * ay.x), r * (cp * ax.y + sp * ay.y), r * (cp * ax.z + sp * ay.z)};
		const V v = {vx * ax.x + vy * ay.x, vx * ax.y + vy * ay.y, vx * ax.z + vy * ay.z};
		const double speed = sqrt(v_radial * v_radial + J * J / r / r), along = dot(x, v);
		if(!(along < 0.0))
			continue;
		const double time = (r - DMS_RSUN_KM) / (-(along / r)), by_speed = (r - DMS_RSUN_KM) / -v_radial;
		const double step = i & 1 ? time + uniform(0.0, 1.0) * (by_speed - time) : time * (1.0 + pow(10.0, uniform(-16, -6)) * uniform(-1, 1));
		if(dms::lane::surface_is_far_by_speed(r, v_radial, speed, step))
		{
			far++;
			*wrong += time < step;
		}
	}
	return far;
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PACKAGE_DIR, "csrc"),
                    "-I", os.path.join(REPO, "include"), "-o", str(d / "rules.so"), str(d / "rules.cpp")], check=True)
    return ctypes.CDLL(str(d / "rules.so"))


def wrong_count_possible(warps, passes, sets, following, clear_after_barrier):
    """Whether some order of the warps' accesses gives a warp a wrong count.

    In each pass every warp adds 1 to the pass's set, waits for the others and reads the set; warp 0 also clears
    the set of the next pass, before the barrier or after its read.  All orders that the barrier allows are tried."""
    body = ["add", "wait", "read"]
    first = body + ["clear"] if clear_after_barrier else ["clear"] + body
    programs = [[(op, p) for p in range(passes) for op in (first if w == 0 else body)] for w in range(warps)]
    set_of = [0]
    for _ in range(passes):
        set_of.append(following(set_of[-1]))

    def passed(w, at):
        """Barriers that a warp at this position is past."""
        return sum(op == "wait" for op, _ in programs[w][:at])

    seen, todo = set(), [((0,) * warps, (0,) * sets)]  # positions, counts
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        at, counts = state
        for w in range(warps):
            if at[w] == len(programs[w]):
                continue
            op, p = programs[w][at[w]]
            # a barrier opens when every warp has reached it
            if op == "wait" and not all(passed(u, at[u]) > p or programs[u][at[u]] == ("wait", p) for u in range(warps)):
                continue
            if op == "read" and counts[set_of[p]] != warps:
                return True
            c = list(counts)
            if op == "add":
                c[set_of[p]] += 1
            elif op == "clear":
                c[set_of[p + 1]] = 0
            todo.append((at[:w] + (at[w] + 1,) + at[w + 1:], tuple(c)))
    return False


@pytest.mark.parametrize("warps", [2, 3])
def test_no_vote_of_a_block_in_lockstep_is_lost(rules, warps):
    assert not wrong_count_possible(warps, 5, rules.vote_sets(), rules.next_vote_set, clear_after_barrier=False)


def test_two_vote_sets_are_too_few():
    """The search finds the races that it is made for."""
    def other(s):
        return 1 - s
    assert wrong_count_possible(2, 3, 2, other, clear_after_barrier=True)
    assert wrong_count_possible(2, 3, 2, other, clear_after_barrier=False)


def test_radial_speed_calls_no_step_far_that_the_surface_binds(rules):
    """A team bounds a step outside the Sun without the event where it may; the step has to be that of a lone lane."""
    wrong = ctypes.c_int()
    rules.far_from_surface.argtypes = [ctypes.c_int, ctypes.c_uint64, ctypes.POINTER(ctypes.c_int)]
    far = rules.far_from_surface(2_000_000, 1, ctypes.byref(wrong))
    assert far > 10_000  # the states reach the rule
    assert wrong.value == 0


@pytest.mark.parametrize("lanes, per, unit", [(32, 32, 1), (128, 64, 2), (512, 64, 2), (640, 64, 2)])
@pytest.mark.parametrize("batch", [1, 8, 32])
@pytest.mark.parametrize("wait", [1, 5, 32])
def test_lanes_wait_for_their_batch_or_their_passes(rules, lanes, per, unit, batch, wait):
    """A batch of b lanes of 32 starts a phase, or the first lane's passes since it arrived; quiet passes before do not count."""
    def passes_until(waiting, quiet, stepping=1):
        state, n = ctypes.c_int(0), 0
        for _ in range(quiet):
            assert not rules.rare_phase_due(ctypes.byref(state), 0, stepping, unit * batch, per, wait, lanes, lanes)
        while True:
            n += 1
            if rules.rare_phase_due(ctypes.byref(state), waiting, stepping, unit * batch, per, wait, lanes, lanes):
                assert state.value == 0
                return n
    enough = batch * lanes // 32
    for quiet in (0, 1, 1000):
        assert passes_until(enough, quiet) == 1
        assert passes_until(enough - 1, quiet) == wait if enough > 1 else True
        assert passes_until(1, quiet, stepping=0) == 1
