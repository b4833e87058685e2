// Kernels of the trajectory engine.
//
// trajectory_kernel, trajectory_kernel_latency: a persistent launch per dms_run, and for a large one a second
// that finishes its last trajectories.  Every thread is a lane that owns one
// trajectory at a time; lanes claim work indices from a global queue (one warp-aggregated
// atomic per claim), and refill as soon as their trajectory terminates, so trajectories of
// wildly different length (0 to 10^6 scatterings) never hold a whole batch back.  A lane's
// trajectory is a state machine whose common state is one outer step of Propagate_Freely
// (src/Simulation_Trajectory.cpp:876-1116); segment starts, scatterings and terminations are
// rare branches.  The time-weighted radial histogram of the running trajectory lives in a
// per-lane scratch row (touched bin range tracked) and is flushed once, at termination, into
// the per-point sums and sums of squares (src/Data_Generation.cpp:787-822).
#include "dms_lane.cuh"
#include "dms_team.cuh"

namespace dms
{

namespace
{
using namespace lane;
using StrictLane = LaneT<Prop, Event>;


// ---------------------------------------------------------------------------------------------
// One pass of the Propagate_Freely loop body (src/Simulation_Trajectory.cpp:876-1116), split at the
// RK45 retry loop: when no step is in progress the pre-step bounds are applied and a step is opened
// (step_begin); every pass makes one RK45 attempt; an accepted attempt runs the optical-depth,
// boundary and commit logic (strict_step).  The propagator keeps the state at the start of the step
// until the step is committed, so a rejected step has nothing to restore.
//
// With every lane busy a pass of a warp executes 3 300 instructions, 17.9 of 32 lanes active, one every 15 cycles:
// 5.4 of them waiting for memory, 3.5 at the barrier, 2.5 for the result of an operation, 1.7 for instructions (an
// SM fetches full rate from 32 KB of instruction cache; measured with a straight-line FP32 loop: 1.2-1.4
// cycles per instruction of a warp up to 32 KB, 3.2 up to 128 KB, 6 beyond).  What some lane of a warp does in
// almost every pass (a depth rejection, the surface, a fresh segment, a scattering point) is written out in
// the pass, so that the step's values stay in registers instead of being handed over in local memory:
// 2^20 Capture-mode trajectories 38.4 -> 36.5 ms, and 40.9 -> 38.4 ms from the hot lane state in shared memory
// with these calls half removed.  In the latency form, where a warp has a scheduler and an instruction cache
// to itself, the same functions are called (CALL): a lone lane takes 3.40 us per step, and 3.51 with them
// written out.  What is rarer stays in non-inlined functions in both.

// The event, speed and scattering rate at the propagator's state, at the start of a free segment
// (later steps take them from the step before).
__device__ __forceinline__ void fresh_state_here(const DevSolar& S, const DevPoint* __restrict__ P, StrictLane& L)
{
	if(!L.hot().before_valid)
		L.hot().before = prop_event(L.hot().pr);
	L.hot().before_valid = L.hot().before_valid ? L.hot().before_valid : 1;
	const double r = prop_radius(L.hot().pr);
	L.hot().next_speed = prop_speed(L.hot().pr);
	L.hot().next_rate = r >= DMS_RSUN_KM ? 0.0 : rate_total(S, P, r, L.hot().next_speed);
	L.hot().next_valid = 1;
}
static __device__ __noinline__ void fresh_state_called(const DevSolar& S, const DevPoint* __restrict__ P, StrictLane& L) { fresh_state_here(S, P, L); }
template <bool CALL>
__device__ __forceinline__ void fresh_state(const DevSolar& S, const DevPoint* __restrict__ P, StrictLane& L)
{
	if constexpr(CALL)
		fresh_state_called(S, P, L);
	else
		fresh_state_here(S, P, L);
}

// Ends the trajectory at the propagator's state.
static __device__ __noinline__ int end_at_propagator(StrictLane& L, int reason)
{
	set_final(L, prop_event(L.hot().pr), true, reason);
	return PH_FINAL;
}

static __device__ __noinline__ double div_general(double a, double b) { return a / b; }

// The time to the surface as a bound of a step that starts at or outside it.
__device__ __forceinline__ double surface_step_here(const Event& before, double r, double step)
{
	const double along = dot3(before.x, before.v);
	if(r > DMS_RSUN_KM && along < 0.0)
	{
		const double est = (r - DMS_RSUN_KM) / (-(along / r));
		if(isfinite(est) && est > 0.0)
		{
			const double lim = est > DMS_RK45_ABS_MIN_STEP_S ? est : DMS_RK45_ABS_MIN_STEP_S;
			step = lim < step ? lim : step;
		}
	}
	return step;
}
static __device__ __noinline__ double surface_step_called(const Event& before, double r, double step) { return surface_step_here(before, r, step); }
template <bool CALL>
__device__ __forceinline__ double surface_step(const Event& before, double r, double step)
{
	if constexpr(CALL)
		return surface_step_called(before, r, step);
	else
		return surface_step_here(before, r, step);
}

// The optical-depth bound of a step that starts inside the Sun at scattering rate `rate`.
__device__ __forceinline__ double inside_step(const RunParams& R, double rate, double step)
{
	const double tau_limit = R.capture_mode ? DMS_CAPTURE_MAX_OPTICAL_DEPTH_STEP : DMS_MAX_OPTICAL_DEPTH_STEP;
	// the quotient is formed only where it can be the smaller one
	if(rate * step * (1.0 + 0x1p-50) > tau_limit)
	{
		bool ok = (rate > 0x1p-200) & (rate < 0x1p100);
		double lim = fast::div(tau_limit, fast::recip(rate, ok));
		if(!ok)
			lim = div_general(tau_limit, rate);
		step = lim < step ? lim : step;
	}
	return step;
}

// Pre-step bounds (src/Simulation_Trajectory.cpp:873-927).  Returns PH_STEP when an attempt is due,
// else the lane's next phase.
template <bool CALL>
__device__ __forceinline__ int step_begin(const RunParams& R, const DevPoint* __restrict__ P, StrictLane& L)
{
	if(!(L.hot().seg_steps < R.max_free_steps))
	{
		if(L.hot().before_valid == 2)  // otherwise L.cur holds the last committed event
		{
			L.cur = L.hot().before;
			L.cur.t += L.hot().origin;
		}
		L.reason = DMS_REASON_MAX_FREE_STEPS;
		return PH_FINAL;
	}
	if(wall_time_exceeded(R, L))  // "before_step", src/Simulation_Trajectory.cpp:873-874
		return end_at_propagator(L, DMS_REASON_WALL_TIME_LIMIT);
	if(!L.hot().next_valid)
		fresh_state<CALL>(R.S, P, L);
	const double r = prop_radius(L.hot().pr);
	double step = sanitized_step(L.hot().pr.time_step);
	double rate = 0.0;
	if(r >= DMS_RSUN_KM)
	{
		step = capped_step(r, L.hot().next_speed, step, R.boundary);
		if(!surface_is_far(r, dot3(L.hot().before.x, L.hot().before.v), step))
			step = surface_step<CALL>(L.hot().before, r, step);
	}
	else
	{
		rate = L.hot().next_rate;
		if(!isfinite(rate) || rate < 0.0)
			return end_at_propagator(L, DMS_REASON_NUMERICAL_FAILURE);
		step = inside_step(R, rate, step);
	}
	L.hot().rate_before = rate;
	L.hot().pr.time_step = step;
	L.hot().in_rk = 1;
	L.hot().rk_inner = 0;
	return PH_STEP;
}

// A step as an accepted attempt leaves it: the propagator after it, the events and radii before
// and after it, and its interval inside the Sun.
struct StepCtx
{
	const Event* before;  // the lane's own, not a copy
	Event after;
	double r_before, r_after, v_after, dt, s0, s1;
};

// Event_In_3D and the speed of a propagator with J = 0, a radius below 1 km or a value outside the
// range of dms_fastmath.cuh.
__device__ __forceinline__ void event_and_speed_general_here(const Prop& p, Event& e, double& speed)
{
	speed = prop_speed(p);
	e = prop_event(p);
}
static __device__ __noinline__ void event_and_speed_general_called(const Prop& p, Event& e, double& speed) { event_and_speed_general_here(p, e, speed); }
template <bool CALL>
__device__ __forceinline__ void event_and_speed_general(const Prop& p, Event& e, double& speed)
{
	if constexpr(CALL)
		event_and_speed_general_called(p, e, speed);
	else
		event_and_speed_general_here(p, e, speed);
}

template <bool CALL>
__device__ __forceinline__ void event_and_speed(const Prop& p, Event& e, double& speed)
{
	bool ok = (p.J > 0x1p-200) & (p.J < 0x1p200) & fast::in_radius_range(p.radius) & (p.radial_mode == 0) & (fabs(p.phi) < 0x1p20);
	const fast::Recip R = fast::recip(p.radius, ok);
	// prop_speed and prop_event with the quotients by the radius sharing its reciprocal
	speed = fast::sqrt(p.v_radial * p.v_radial + fast::div(fast::div(p.J * p.J, R), R), ok);
	if(!ok)
	{
		event_and_speed_general<CALL>(p, e, speed);
		return;
	}
	const double safe = p.radius;
	double sp, cp;
	sincos_fast(p.phi, sp, cp);
	const double vt = fast::div(p.J, R);
	const double vx = p.v_radial * cp - vt * sp;
	const double vy = p.v_radial * sp + vt * cp;
	e.t = p.time;
	e.x = mk(safe * (cp * p.ax.x + sp * p.ay.x), safe * (cp * p.ax.y + sp * p.ay.y), safe * (cp * p.ax.z + sp * p.ay.z));
	e.v = mk(vx * p.ax.x + vy * p.ay.x, vx * p.ax.y + vy * p.ay.y, vx * p.ax.z + vy * p.ay.z);
}

// Whether a chord with both ends clearly outside the Sun passes clear of it: it only recedes from or only
// approaches the Sun between its ends, or its line misses the Sun.  Solar_Interior_Fraction_Interval
// then finds no crossing in [0, 1]; the margin of 10^-6 is far above its rounding.
__device__ __forceinline__ bool chord_stays_outside(const Event& a, const Event& b, double ra, double rb)
{
	const Vec3 d = sub3(b.x, a.x);
	const double ad = dot3(a.x, d), bd = dot3(b.x, d), dd = dot3(d, d);
	const double lim = DMS_RSUN_KM * (1.0 + 1.0e-6);
	return (ra > lim) & (rb > lim) & ((ad >= 0.0) | (bd <= 0.0) | ((ra * ra - lim * lim) * dd > ad * ad * (1.0 + 1.0e-6)));
}

// Solar_Interior_Fraction_Interval for a chord with an end outside the Sun.
__device__ __forceinline__ bool interior_interval_outside_here(const Event& a, const Event& b, double ra, double rb, double& s0, double& s1)
{
	return interior_interval(a, b, ra, rb, s0, s1);
}
static __device__ __noinline__ bool interior_interval_outside_called(const Event& a, const Event& b, double ra, double rb, double& s0, double& s1)
{
	return interior_interval_outside_here(a, b, ra, rb, s0, s1);
}
template <bool CALL>
__device__ __forceinline__ bool interior_interval_outside(const Event& a, const Event& b, double ra, double rb, double& s0, double& s1)
{
	if constexpr(CALL)
		return interior_interval_outside_called(a, b, ra, rb, s0, s1);
	else
		return interior_interval_outside_here(a, b, ra, rb, s0, s1);
}

static __device__ __noinline__ double rate_total_general(const DevSolar& S, const DevPoint* __restrict__ P, double r, double v)
{
	return rate_total(S, P, r, v);
}

// rate_total at 0 <= r, v; r at or beyond the surface gives 0 (Scattering_Rate_At_Fraction).
__device__ __forceinline__ double rate_inside(const DevSolar& S, const DevPoint* __restrict__ P, double r, double v)
{
	if(r >= DMS_RSUN_KM)
		return 0.0;
	if(!((r < DMS_RSUN_KM) & (v <= __ldg(&P->grid_vmax))))
		return rate_total_general(S, P, r, v);  // no grid, a speed beyond it or a NaN
	const double rc = r * __ldg(&P->grid_inv_r), vc = v * __ldg(&P->grid_inv_v);
	const unsigned int N = static_cast<unsigned int>(__ldg(&P->grid_n));
	const double last = __ldg(&P->grid_last);  // N - 2
	double wr, wv;
	unsigned int ri = fast::floor_index(rc, wr), vi = fast::floor_index(vc, wv);
	ri = ri > N - 2 ? N - 2 : ri;
	vi = vi > N - 2 ? N - 2 : vi;
	const double rf = rc - (wr > last ? last : wr), vf = vc - (wv > last ? last : wv);
	DMS_CHECK_INDEX(ri, 0u, N - 1, BOUNDS_GRID);
	DMS_CHECK_INDEX(vi, 0u, N - 1, BOUNDS_GRID);
	const double* g = reinterpret_cast<const double*>(__ldg(reinterpret_cast<const unsigned long long*>(&P->grid))) + static_cast<size_t>(ri) * N + vi;
	const double g00 = __ldg(g), g01 = __ldg(g + 1);
	const double g10 = __ldg(g + N), g11 = __ldg(g + N + 1);
	const double lower_rate = g00 + vf * (g01 - g00);
	const double upper_rate = g10 + vf * (g11 - g10);
	const double rate = lower_rate + rf * (upper_rate - lower_rate);
	return isfinite(rate) ? (rate > 0.0 ? rate : 0.0) : NAN;
}

// One piece-boundary rate of a step (Scattering_Rate_At_Fraction at fraction f of the chord a - b)
// or, with `next`, the scattering rate at the state after the step (ra, va), which the next step's
// head needs.
__device__ __forceinline__ double piece_rate(const DevSolar& S, const DevPoint* __restrict__ P, const Vec3& ax, const Vec3& av, const Vec3& bx,
                                             const Vec3& bv, double f, bool next, double ra, double va)
{
	f = clamp_unit(f);
	const double x = ax.x + f * (bx.x - ax.x), vx = av.x + f * (bv.x - av.x);
	const double y = ax.y + f * (bx.y - ax.y), vy = av.y + f * (bv.y - av.y);
	const double z = ax.z + f * (bx.z - ax.z), vz = av.z + f * (bv.z - av.z);
	double r, v;
	sqrt2(x * x + y * y + z * z, vx * vx + vy * vy + vz * vz, r, v);
	r = next ? ra : r;
	v = next ? va : v;
	return rate_inside(S, P, r, v);
}

// The optical depth of a step: the trapezoid sum over its pieces (dtau), the two-piece estimate
// (tau2), whether a rate was invalid, and the rate at the state after the step.
struct Depth
{
	double dtau, tau2, next_rate;
	bool invalid;
};

// Adds piece boundary i at fraction f with its rate to the sums of Build_Optical_Depth_Pieces
// (src/Simulation_Trajectory.cpp:347-414), in the reference's order.  The two-piece estimate is over
// [0, 2] and [2, 4] of four pieces; with two pieces (Capture mode) it is the sum itself and not used.
struct DepthSums
{
	double f_prev, r_prev, f_0, r_0;
	__device__ __forceinline__ void add(Depth& d, int i, double f, double rate, double dt)
	{
		d.invalid |= !(rate >= 0.0) | !(rate < INFINITY);
		if(i == 0)
		{
			f_0 = f;
			r_0 = rate;
			d.tau2 = 0.0;
		}
		else
		{
			if(f > f_prev)
				d.dtau += 0.5 * (r_prev + rate) * (dt * (f - f_prev));
			if((i & 1) == 0)
			{
				d.tau2 += 0.5 * (r_0 + rate) * (dt * (f - f_0));
				f_0 = f;
				r_0 = rate;
			}
		}
		f_prev = f;
		r_prev = rate;
	}
};

// The depth of one lane's step, its boundary rates one after another.
__device__ __forceinline__ void lane_depth(const RunParams& R, const DevPoint* __restrict__ P, const StepCtx& c, double rate_before, bool first_known,
                                           int pieces, Depth& d)
{
	const double fraction = 1.0 / static_cast<double>(pieces), span = c.s1 - c.s0;  // 1/2 or 1/4, exact
	DepthSums sums = {};
#pragma unroll 1
	for(int i = 0; i <= pieces + 1; i++)
	{
		const double f = c.s0 + static_cast<double>(i) * fraction * span;
		double rate = rate_before;
		if(i > 0 || !first_known)
			rate = piece_rate(R.S, P, c.before->x, c.before->v, c.after.x, c.after.v, f, i > pieces, c.r_after, c.v_after);
		if(i <= pieces)
			sums.add(d, i, f, rate, c.dt);
		else
			d.next_rate = rate;
	}
}

// The depths of the steps of the lanes in `dm`, each boundary rate of each step on a lane of its own
// (the whole warp calls this): the owners of a round put their events into shared memory, 30 or 32
// lanes form one rate each, and every owner sums its own.  The same lookups with the same
// arguments as lane_depth, so the same numbers.  A rate is a dependent chain of some 600 cycles, so
// a warp with few finished steps is done in one chain per round instead of five.
constexpr int COOP_SLOT = 18;    // doubles of a step handed over
constexpr int COOP_SLOTS = 8;    // most steps of a round (Capture mode: 4 rates each)
constexpr int COOP_BUFFER = COOP_SLOT * COOP_SLOTS + 32;
__device__ __forceinline__ void warp_depth(const RunParams& R, const DevPoint* __restrict__ P, const StepCtx& c, double rate_before, bool first_known,
                                           int pieces, unsigned int dm, bool mine, double* buffer, Depth& d)
{
	const double fraction = 1.0 / static_cast<double>(pieces);
	const int rates = pieces + 2, slots = 32 / rates;
	const int me = threadIdx.x & 31;
	const int rank = __popc(dm & ((1u << me) - 1u));
	const int steps = __popc(dm);
	const int slot_of_job = pieces == 4 ? (me * 43) >> 8 : me >> 2, j = me - slot_of_job * rates;  // me / rates
	for(int base = 0; base < steps; base += slots)
	{
		const int slot = rank - base;
		const bool owner = mine && slot >= 0 && slot < slots;
		if(owner)
		{
			double* b = buffer + slot * COOP_SLOT;
			b[0] = c.before->x.x; b[1] = c.before->x.y; b[2] = c.before->x.z;
			b[3] = c.before->v.x; b[4] = c.before->v.y; b[5] = c.before->v.z;
			b[6] = c.after.x.x; b[7] = c.after.x.y; b[8] = c.after.x.z;
			b[9] = c.after.v.x; b[10] = c.after.v.y; b[11] = c.after.v.z;
			b[12] = c.s0; b[13] = c.s1 - c.s0;
			b[14] = c.r_after; b[15] = c.v_after;
			b[16] = __longlong_as_double(reinterpret_cast<long long>(P));
		}
		__syncwarp();
		double rate = 0.0;
		if(slot_of_job < slots && base + slot_of_job < steps)
		{
			const double* b = buffer + slot_of_job * COOP_SLOT;
			rate = piece_rate(R.S, reinterpret_cast<const DevPoint*>(__double_as_longlong(b[16])), mk(b[0], b[1], b[2]), mk(b[3], b[4], b[5]), mk(b[6], b[7], b[8]), mk(b[9], b[10], b[11]),
			                  b[12] + static_cast<double>(j) * fraction * b[13], j > pieces, b[14], b[15]);
		}
		buffer[COOP_SLOT * COOP_SLOTS + me] = rate;
		__syncwarp();
		if(owner)
		{
			const double* q = buffer + COOP_SLOT * COOP_SLOTS + slot * rates;
			const double span = c.s1 - c.s0;
			DepthSums sums = {};
			sums.add(d, 0, c.s0, first_known ? rate_before : q[0], c.dt);
			sums.add(d, 1, c.s0 + fraction * span, q[1], c.dt);
			sums.add(d, 2, c.s0 + 2.0 * fraction * span, q[2], c.dt);
			if(pieces == 4)
			{
				sums.add(d, 3, c.s0 + 3.0 * fraction * span, q[3], c.dt);
				sums.add(d, 4, c.s0 + 4.0 * fraction * span, q[4], c.dt);
			}
			d.next_rate = q[rates - 1];
		}
		__syncwarp();
	}
}

constexpr int PH_CONTINUE = -1;  // depth_reject: the step stands

// A step whose optical depth exceeds the limit or whose two estimates differ too much: the step is
// taken again, shorter (src/Simulation_Trajectory.cpp:975-1011).
__device__ __forceinline__ int depth_reject_here(StrictLane& L, const Event& before, double dtau, double apart, double scale, bool capture_mode, double dt,
                                                double tau_limit)
{
	const double rel = apart / scale;
	const bool reject_acc = !capture_mode && rel > DMS_OPTICAL_DEPTH_REL_TOL;
	if(!(dtau > tau_limit) && !reject_acc)
		return PH_CONTINUE;
	L.hot().retries++;
	if(L.hot().retries > DMS_MAX_OPTICAL_DEPTH_RETRIES)
	{
		set_final(L, before, true, DMS_REASON_NUMERICAL_FAILURE);
		return PH_FINAL;
	}
	double factor = DMS_RK45_MAX_STEP_FACTOR;
	if(dtau > tau_limit && dtau > 0.0 && 0.8 * tau_limit / dtau < factor)
		factor = 0.8 * tau_limit / dtau;
	if(reject_acc && rel > 0.0 && 0.8 * sqrt(DMS_OPTICAL_DEPTH_REL_TOL / rel) < factor)
		factor = 0.8 * sqrt(DMS_OPTICAL_DEPTH_REL_TOL / rel);
	if(factor > 1.0) factor = 1.0;
	if(factor < DMS_RK45_MIN_STEP_FACTOR) factor = DMS_RK45_MIN_STEP_FACTOR;
	L.hot().pr.time_step = sanitized_step(factor * dt);
	return PH_STEP;  // L.hot().before and the speed and rate at it still describe the propagator
}
static __device__ __noinline__ int depth_reject_called(StrictLane& L, const Event& before, double dtau, double apart, double scale,
                                                       bool capture_mode, double dt, double tau_limit)
{
	return depth_reject_here(L, before, dtau, apart, scale, capture_mode, dt, tau_limit);
}
template <bool CALL>
__device__ __forceinline__ int depth_reject(StrictLane& L, const Event& before, double dtau, double apart, double scale, bool capture_mode,
                                            double dt, double tau_limit)
{
	if constexpr(CALL)
		return depth_reject_called(L, before, dtau, apart, scale, capture_mode, dt, tau_limit);
	else
		return depth_reject_here(L, before, dtau, apart, scale, capture_mode, dt, tau_limit);
}

// The scattering point of a step whose depth reaches the remaining one (src/Simulation_Trajectory.cpp:
// 1013-1044).  The boundary rates are formed again: the same lookups, the same numbers.
__device__ __forceinline__ void scatter_point_here(const DevSolar& S, const DevPoint* __restrict__ P, const StepCtx& c, double rate_before, bool first_known,
                                                  bool depth, int pieces, double remaining, Event& accepted)
{
	if(depth)
	{
		const double fraction = 1.0 / static_cast<double>(pieces), span = c.s1 - c.s0;
		double f_prev = c.s0, r_prev = rate_before;
		if(!first_known)
			r_prev = rate_at_fraction(S, P, *c.before, c.after, f_prev);
#pragma unroll 1
		for(int k = 1; k <= pieces; k++)
		{
			const double f = c.s0 + static_cast<double>(k) * fraction * span;
			const double rate = rate_at_fraction(S, P, *c.before, c.after, f);
			if(f > f_prev)
			{
				const double pdt = c.dt * (f - f_prev);
				const double ptau = 0.5 * (r_prev + rate) * pdt;
				if(ptau >= remaining)
				{
					const double lf = solve_linear_rate(r_prev, rate, pdt, remaining);
					accepted = interpolate_event(*c.before, c.after, f_prev + lf * (f - f_prev));
					return;
				}
				remaining -= ptau;
			}
			f_prev = f;
			r_prev = rate;
		}
	}
	accepted = interpolate_event(*c.before, c.after, c.s1);
}
static __device__ __noinline__ void scatter_point_called(const DevSolar& S, const DevPoint* __restrict__ P, const StepCtx& c, double rate_before,
                                                         bool first_known, bool depth, int pieces, double remaining, Event& accepted)
{
	scatter_point_here(S, P, c, rate_before, first_known, depth, pieces, remaining, accepted);
}
template <bool CALL>
__device__ __forceinline__ void scatter_point(const DevSolar& S, const DevPoint* __restrict__ P, const StepCtx& c, double rate_before,
                                              bool first_known, bool depth, int pieces, double remaining, Event& accepted)
{
	if constexpr(CALL)
		scatter_point_called(S, P, c, rate_before, first_known, depth, pieces, remaining, accepted);
	else
		scatter_point_here(S, P, c, rate_before, first_known, depth, pieces, remaining, accepted);
}

__device__ void commit_event(const RunParams& R, double m_dm, StrictLane& L, double2* hist, const Event& local);

// A step that ends at or beyond the boundary radius (src/Simulation_Trajectory.cpp:1046-1086).
enum Boundary : int
{
	BOUNDARY_INSIDE = 0,    // nothing to do
	BOUNDARY_ESCAPE = 1,    // c.after is the outward escape
	BOUNDARY_RETURN = 2,    // the bound orbit was carried back to the boundary; the segment goes on
	BOUNDARY_FAILURE = 3,
};
static __device__ __noinline__ int boundary_step(const RunParams& R, double m_dm, StrictLane& L, double2* hist, StepCtx& c)
{
	const DevSolar& S = R.S;
	Event ev = c.after;
	double r_b = c.r_after, v_b = c.v_after;
	if(c.r_before < R.boundary && c.r_after >= R.boundary && c.r_after > c.r_before)
	{
		const double f = (R.boundary - c.r_before) / (c.r_after - c.r_before);
		ev = interpolate_event(*c.before, c.after, f);
		r_b = ev_radius(ev);
		v_b = ev_speed(ev);
	}
	if(!(r_b >= R.boundary && r_b >= c.r_before))
		return BOUNDARY_INSIDE;
	if(v_b > solar_vesc(S, r_b))
	{
		c.after = ev;
		return BOUNDARY_ESCAPE;
	}
	Event abs_b = ev;
	abs_b.t += L.hot().origin;
	if(uncaptured_bound(S, m_dm, L, abs_b))
	{
		set_final(L, abs_b, false, DMS_REASON_NUMERICAL_FAILURE);
		return BOUNDARY_FAILURE;
	}
	Event inbound;
	if(!bound_kepler_return(ev, inbound))
		return BOUNDARY_INSIDE;
	L.hot().seg_steps++;
	L.hot().steps++;
	L.hot().retries = 0;
	commit_event(R, m_dm, L, hist, ev);
	// reset_propagator_at_absolute_event, src/Simulation_Trajectory.cpp:814-822
	L.cur = inbound;
	L.cur.t += L.hot().origin;
	L.hot().origin = L.cur.t;
	Event local = inbound;
	local.t = 0.0;
	prop_init(L.hot().pr, local);
	L.hot().before_valid = 0;
	L.hot().next_valid = 0;
	if(!R.capture_mode && L.prev_time >= 0.0)
		L.prev_time = 0.0;
	return BOUNDARY_RETURN;
}

static __device__ __noinline__ double solar_vesc_general(const DevSolar& S, double r) { return solar_vesc(S, r); }

// drift / scale of Update_Capture_State where it can be the larger one.
static __device__ __noinline__ void relative_drift(StrictLane& L, double drift, double scale)
{
	const double rel = drift / scale;
	if(isfinite(rel) && rel > L.max_drift_rel)
		L.max_drift_rel = rel;
}

// Update_Capture_State(..., allow_new_capture = false) of a captured particle and the bincount, the
// parts of commit_accepted_event (src/Simulation_Trajectory.cpp:842-874, 640-721) at radius r and speed v.
__device__ __forceinline__ void commit_event_inline(const RunParams& R, double m_dm, StrictLane& L, double2* hist, double t, double r, double v)
{
	const double vv = v * v;
	if(!R.capture_mode)
	{
		if(L.prev_time >= 0.0)
			accumulate_bincount(L, hist, L.prev_r, L.prev_v2, t - L.prev_time);
		L.prev_time = t;
		L.prev_r = r;
		L.prev_v2 = vv;
	}
	if(!L.hot().is_captured)
		return;
	if(L.bound_state)
		L.t_last_bound = t + L.hot().origin;
	if(!isfinite(L.free_flight_E))
		return;
	// capture_energy_eV
	bool ok = (R.S.fast_tables != 0) & (r < 0x1p100);
	double w;  // v_esc^2 before its root
	if(r <= DMS_RSUN_KM)
		w = solar_vesc2_fast(R.S, r);
	else
		w = fast::div(2 * DMS_GMSUN_KM3S2, fast::recip(r, ok));
	double vesc = fast::sqrt(w, ok);
	if(!ok)
		vesc = solar_vesc_general(R.S, r);
	const double E = fast::div_const(0.5 * m_dm * fast::div_const(vv - vesc * vesc, DMS_C_KMS * DMS_C_KMS), 1.0e-9);
	const double drift = fabs(E - L.free_flight_E);
	if(drift < INFINITY)
	{
		if(drift > L.max_drift_eV)
			L.max_drift_eV = drift;
		const double ref = fabs(L.free_flight_E);
		const double scale = ref > DMS_FREE_ENERGY_DRIFT_REL_E_SCALE_EV ? ref : DMS_FREE_ENERGY_DRIFT_REL_E_SCALE_EV;
		if(drift * (1.0 + 0x1p-50) >= L.max_drift_rel * scale)
			relative_drift(L, drift, scale);
	}
}

// abort_if_uncaptured_bound on the committed event, src/Simulation_Trajectory.cpp:767-778, 1108: whether
// its capture energy is not finite and >= 0, whose sign is that of v^2 - v_esc^2.  r and v may be a
// rounding error off (the propagator's): what is not clearly faster than the escape speed is decided
// with the event's own radius and speed.
__device__ __forceinline__ bool not_free_general_here(const DevSolar& S, double m_dm, const Event& e)
{
	const double E = capture_energy_eV(S, m_dm, ev_radius(e), ev_speed(e));
	return !(isfinite(E) && E >= 0.0);
}
static __device__ __noinline__ bool not_free_general_called(const DevSolar& S, double m_dm, const Event& e) { return not_free_general_here(S, m_dm, e); }
template <bool CALL>
__device__ __forceinline__ bool not_free_general(const DevSolar& S, double m_dm, const Event& e)
{
	if constexpr(CALL)
		return not_free_general_called(S, m_dm, e);
	else
		return not_free_general_here(S, m_dm, e);
}
template <bool CALL>
__device__ __forceinline__ bool not_free(const RunParams& R, double m_dm, const Event& e, double r, double v)
{
	const bool inside = r <= DMS_RSUN_KM;
	const double vv = v * v;
	// outside the Sun v_esc^2 = 2 G M / r, compared without the division
	const double have = inside ? vv : vv * r;
	const double need = inside ? solar_vesc2_fast(R.S, r) : 2 * DMS_GMSUN_KM3S2;
	const bool clear = (have > need * (1.0 + 0x1p-40)) & (vv < 1.0e200) & (r < 0x1p100) & (R.S.fast_tables != 0);
	return clear ? false : not_free_general<CALL>(R.S, m_dm, e);
}

__device__ __noinline__ void commit_event(const RunParams& R, double m_dm, StrictLane& L, double2* hist, const Event& local)
{
	commit_event_inline(R, m_dm, L, hist, local.t, ev_radius(local), ev_speed(local));
}

// Steps of a warp whose depths are formed by the whole warp rather than by each lane: one round of
// lookups serves 5 steps (8 in Capture mode) and costs a third more than one lookup of lane_depth,
// which makes 5 (3) of them one after another.
constexpr int COOP_MAX_STEPS = 15;

// Commits a step whose outcome is decided (src/Simulation_Trajectory.cpp:1088-1116): the event c.after, and
// for a plain step the propagator after it with the scattering rate there (next_known when it was formed).
template <bool CALL>
__device__ __forceinline__ int finish_step(const RunParams& R, double m_dm, StrictLane& L, double2* hist, const StepCtx& c,
                                           bool scattering, int boundary, double time, double radius, double phi, double v_radial, double time_step,
                                           double next_rate, bool next_known)
{
	L.hot().seg_steps++;
	L.hot().steps++;
	L.hot().retries = 0;
	const bool plain = !scattering && boundary == BOUNDARY_INSIDE;
	// the committed event's own radius and speed; in Capture mode a plain step only asks whether the
	// particle is still free, which the propagator's decide
	double r_now = c.r_after, v_now = c.v_after;
	if(!R.capture_mode | L.hot().is_captured | !plain)
		sqrt2(dot3(c.after.x, c.after.x), dot3(c.after.v, c.after.v), r_now, v_now);
	commit_event_inline(R, m_dm, L, hist, c.after.t, r_now, v_now);
	const bool bound = !L.hot().is_captured && not_free<CALL>(R, m_dm, c.after, r_now, v_now);
	if(bound | !plain)
	{
		L.cur = c.after;
		L.cur.t += L.hot().origin;
		if(bound)
			L.reason = DMS_REASON_NUMERICAL_FAILURE;
		else if(!scattering)
			L.reason = DMS_REASON_OUTWARD_ESCAPE;
		else if(r_now < DMS_RSUN_KM)
			return PH_SCATTER;  // Simulate, src/Simulation_Trajectory.cpp:1313-1346; Sample_Target runs in the lane loop
		else
			L.reason = DMS_REASON_SCATTER;
		return PH_FINAL;
	}
	L.hot().pr.time = time;
	L.hot().pr.radius = radius;
	L.hot().pr.phi = phi;
	L.hot().pr.v_radial = v_radial;
	L.hot().pr.time_step = time_step;
	L.hot().before = c.after;
	L.hot().before_valid = 2;
	// the next step starts from this speed and rate; without a depth the rate at a state inside the
	// Sun is not known yet
	L.hot().next_speed = c.v_after;
	L.hot().next_rate = next_rate;
	L.hot().next_valid = next_known || c.r_after >= DMS_RSUN_KM;
	return PH_STEP;
}

// One pass for every lane of the warp (all 32 call it); returns the lane's next phase.
template <int UNROLL>
__device__ __forceinline__ int strict_step(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, StrictLane& L, double2* hist, int phase,
                                           double* buffer)
{
	constexpr bool CALL = UNROLL > 1;
	const int capture_mode = R.capture_mode;
	const int pieces = capture_mode ? DMS_CAPTURE_OPTICAL_DEPTH_PIECES : DMS_MAX_OPTICAL_DEPTH_PIECES;
	const double tau_limit = capture_mode ? DMS_CAPTURE_MAX_OPTICAL_DEPTH_STEP : DMS_MAX_OPTICAL_DEPTH_STEP;
	StepCtx c;
	Prop q;
	bool done = false, interior = false, depth = false;
	int reason = 0;
	if(phase == PH_STEP && !L.hot().in_rk)
		phase = step_begin<CALL>(R, P, L);
	if(phase == PH_STEP)
	{
		q = L.hot().pr;
		L.hot().rk_inner++;
		const int rk = rk45_attempt<UNROLL>(R.S, q, L.hot().rk_inner);
		if(rk == RK_RETRY)
			L.hot().pr.time_step = q.time_step;
		else
		{
			done = true;
			L.hot().in_rk = 0;
			L.hot().attempts += static_cast<uint64_t>(L.hot().rk_inner);
			c.before = &L.hot().before;
			c.r_before = prop_radius(L.hot().pr);
			c.dt = q.time - L.hot().pr.time;
			c.r_after = prop_radius(q);
			event_and_speed<CALL>(q, c.after, c.v_after);
			// the checks after an attempt, src/Simulation_Trajectory.cpp:930-960
			if(rk == RK_FORCED)
				reason = DMS_REASON_NUMERICAL_FAILURE;
			else if(!isfinite(c.r_after) || !isfinite(c.v_after) || !isfinite(c.dt) || c.dt <= 0.0)
				reason = DMS_REASON_NON_FINITE_STATE;
			else if(c.v_after > DMS_V_MAX_C * DMS_C_KMS)
				reason = DMS_REASON_SPEED_LIMIT;
			else if(wall_time_exceeded(R, L))  // "after_rk45_step", src/Simulation_Trajectory.cpp:953-954
				reason = DMS_REASON_WALL_TIME_LIMIT;
			else
			{
				c.s0 = 0.0;
				c.s1 = 1.0;
				interior = true;
				if(!(c.r_before < DMS_RSUN_KM && c.r_after < DMS_RSUN_KM))
				{
					c.s1 = 0.0;
					interior = false;
					if(!chord_stays_outside(*c.before, c.after, c.r_before, c.r_after))
						interior = interior_interval_outside<CALL>(*c.before, c.after, c.r_before, c.r_after, c.s0, c.s1);
				}
				depth = interior && c.s1 > c.s0;
			}
		}
	}
	const unsigned int dm = __ballot_sync(0xffffffffu, depth);
	Depth d = {0.0, 0.0, 0.0, false};
	const bool first_known = depth && c.r_before < DMS_RSUN_KM && c.s0 <= 1.0e-12;
	if(dm != 0u)
	{
		if(__popc(dm) <= COOP_MAX_STEPS)
			warp_depth(R, P, c, L.hot().rate_before, first_known, pieces, dm, depth, buffer, d);
		else if(depth)
			lane_depth(R, P, c, L.hot().rate_before, first_known, pieces, d);
	}
	if(!done)
		return phase;
	if(d.invalid || !isfinite(d.dtau) || d.dtau < 0.0)
		reason = DMS_REASON_NUMERICAL_FAILURE;
	if(reason != 0)
	{
		set_final(L, c.after, true, reason);
		return PH_FINAL;
	}
	bool scattering = false;
	if(interior)
	{
		const double scale = d.dtau > DMS_OPTICAL_DEPTH_ABS_TOL ? d.dtau : DMS_OPTICAL_DEPTH_ABS_TOL;
		const double apart = capture_mode ? 0.0 : fabs(d.dtau - d.tau2);
		if((d.dtau > tau_limit) | (!capture_mode & (apart > (DMS_OPTICAL_DEPTH_REL_TOL * (1.0 - 0x1p-50)) * scale)))
		{
			const int rejected = depth_reject<CALL>(L, *c.before, d.dtau, apart, scale, capture_mode != 0, c.dt, tau_limit);
			if(rejected != PH_CONTINUE)
				return rejected;
		}
		if(d.dtau >= L.hot().tau)
		{
			scatter_point<CALL>(R.S, P, c, L.hot().rate_before, first_known, depth, pieces, L.hot().tau, c.after);
			scattering = true;
		}
		else
			L.hot().tau -= d.dtau;
	}
	int boundary = BOUNDARY_INSIDE;
	if(!scattering && c.r_after >= R.boundary)
	{
		boundary = boundary_step(R, m_dm, L, hist, c);
		if(boundary == BOUNDARY_RETURN)
			return PH_STEP;
		if(boundary == BOUNDARY_FAILURE)
			return PH_FINAL;
	}
	return finish_step<CALL>(R, m_dm, L, hist, c, scattering, boundary, q.time, q.radius, q.phi, q.v_radial, q.time_step, d.next_rate, depth);
}

// ---------------------------------------------------------------------------------------------
// The three parts of a step made by a team (dms_team.cuh).
using StrictBox = TeamBox<Prop, Event>;

// The propagating warp's step: from s to n.  One lane.
__device__ __forceinline__ void strict_propagate(const RunParams& R, const StrictBox& b, const TeamState& s, TeamState& n)
{
	Prop q = team_prop(b, s);
	// step_begin; the event at the state is only needed where the time to the surface may bind
	const double r = s.radius;
	double step = sanitized_step(s.step);
	bool ok = true;
	if(r >= DMS_RSUN_KM)
	{
		step = capped_step(r, s.speed, step, R.boundary);
		if(!surface_is_far_by_speed(r, s.v_radial, s.speed, step))
		{
			Event before;
			double speed;
			event_and_speed<true>(q, before, speed);
			step = surface_step<true>(before, r, step);
		}
	}
	else
	{
		ok = (s.rate >= 0.0) & (s.rate < INFINITY);
		step = inside_step(R, s.rate, step);
	}
	q.time_step = step;
	int inner = 0, rk = RK_RETRY;
	while(ok && rk == RK_RETRY && inner <= DMS_RK45_MAX_INNER_RETRIES)
	{
		inner++;
		rk = rk45_attempt<6>(R.S, q, inner);
	}
	ok &= rk == RK_ACCEPTED;
	// prop_speed, as in event_and_speed
	ok &= fast::in_radius_range(q.radius) & (fabs(q.phi) < 0x1p20);
	const fast::Recip D = fast::recip(q.radius, ok);
	n.speed = fast::sqrt(q.v_radial * q.v_radial + fast::div(fast::div(b.pr.J * b.pr.J, D), D), ok);
	n.rate = ok ? rate_inside(R.S, b.P, q.radius, n.speed) : 0.0;
	n.time = q.time;
	n.radius = q.radius;
	n.phi = q.phi;
	n.v_radial = q.v_radial;
	n.step = q.time_step;
	n.inner = inner;
	n.ok = ok ? 1 : 0;
}

// The judging warp's step: from state s with event e to state n, whose event goes to en.  All 32 lanes;
// `mine` marks the lane whose trajectory it is.
__device__ __forceinline__ int strict_judge(const RunParams& R, const StrictBox& b, TeamState& s, const Event& e, const TeamState& n, Event& en, StrictLane& L,
                                          bool mine, double* buffer, StepCtx& c)
{
	const int capture_mode = R.capture_mode;
	const int pieces = capture_mode ? DMS_CAPTURE_OPTICAL_DEPTH_PIECES : DMS_MAX_OPTICAL_DEPTH_PIECES;
	const double tau_limit = capture_mode ? DMS_CAPTURE_MAX_OPTICAL_DEPTH_STEP : DMS_MAX_OPTICAL_DEPTH_STEP;
	bool interior = false, depth = false, stop = true;
	if(mine && n.ok)
	{
		const Prop q = team_prop(b, n);
		c.before = &e;
		c.r_before = s.radius;
		c.dt = n.time - s.time;
		c.r_after = n.radius;
		event_and_speed<true>(q, c.after, c.v_after);
		stop = !(isfinite(c.v_after) & (c.dt > 0.0) & (c.dt < INFINITY) & (c.v_after <= DMS_V_MAX_C * DMS_C_KMS) &
		         (L.hot().seg_steps + 4 < R.max_free_steps));
		if(!stop)
		{
			c.s0 = 0.0;
			c.s1 = 1.0;
			interior = true;
			if(!(c.r_before < DMS_RSUN_KM && c.r_after < DMS_RSUN_KM))
			{
				c.s1 = 0.0;
				interior = false;
				if(!chord_stays_outside(*c.before, c.after, c.r_before, c.r_after))
					interior = interior_interval_outside<true>(*c.before, c.after, c.r_before, c.r_after, c.s0, c.s1);
			}
			depth = interior && c.s1 > c.s0;
		}
	}
	const unsigned int dm = __ballot_sync(0xffffffffu, depth);
	Depth d = {0.0, 0.0, 0.0, false};
	if(dm != 0u)
		warp_depth(R, b.P, c, s.rate, c.r_before < DMS_RSUN_KM && c.s0 <= 1.0e-12, pieces, dm, depth, buffer, d);
	int verdict = VERDICT_STOP;
	if(mine && !stop)
	{
		const double scale = d.dtau > DMS_OPTICAL_DEPTH_ABS_TOL ? d.dtau : DMS_OPTICAL_DEPTH_ABS_TOL;
		const double apart = capture_mode ? 0.0 : fabs(d.dtau - d.tau2);
		verdict = VERDICT_PLAIN;
		if(d.invalid | !(d.dtau >= 0.0) | !(d.dtau < INFINITY))
			verdict = VERDICT_STOP;
		else if(interior & (d.dtau >= L.hot().tau))
			verdict = VERDICT_SCATTER;
		if(interior && ((d.dtau > tau_limit) | (!capture_mode & (apart > (DMS_OPTICAL_DEPTH_REL_TOL * (1.0 - 0x1p-50)) * scale))) && !d.invalid &&
		   d.dtau >= 0.0 && d.dtau < INFINITY)
		{
			// (a rejection comes before the scattering test; the last retry ends the trajectory)
			verdict = VERDICT_STOP;
			if(L.hot().retries < DMS_MAX_OPTICAL_DEPTH_RETRIES)
			{
				const int rejected = depth_reject<true>(L, *c.before, d.dtau, apart, scale, capture_mode != 0, c.dt, tau_limit);
				verdict = rejected == PH_STEP ? VERDICT_RESTART : (d.dtau >= L.hot().tau ? VERDICT_SCATTER : VERDICT_PLAIN);
			}
		}
		if(verdict == VERDICT_PLAIN && c.r_after >= R.boundary)
			verdict = VERDICT_BOUNDARY;
		if(verdict == VERDICT_PLAIN && !L.hot().is_captured && not_free<true>(R, b.m_dm, c.after, c.r_after, c.v_after))
			verdict = VERDICT_STOP;
		if(verdict != VERDICT_STOP)
			L.hot().attempts += static_cast<uint64_t>(n.inner);
		if(verdict == VERDICT_RESTART)
			s.step = L.hot().pr.time_step;
		if(interior && (verdict == VERDICT_PLAIN || verdict == VERDICT_BOUNDARY))
			L.hot().tau -= d.dtau;
		if(verdict == VERDICT_PLAIN)
		{
			L.hot().seg_steps++;
			L.hot().steps++;
			L.hot().retries = 0;
			en = c.after;
		}
	}
	return verdict;
}

// The committing warp's step: the bincount and energy drift of the event e.  One lane, whose own lane
// state serves as scratch.
__device__ __forceinline__ void strict_commit(const RunParams& R, const StrictBox& b, StrictLane& L, const Event& e)
{
	double r, v;
	if(!R.capture_mode | L.hot().is_captured)
	{
		sqrt2(dot3(e.x, e.x), dot3(e.v, e.v), r, v);
		commit_event_inline(R, b.m_dm, L, b.hist, e.t, r, v);
	}
}

struct StrictTeam
{
	using Lane = StrictLane;
	using Box = StrictBox;
	using Ctx = StepCtx;
	static __device__ __forceinline__ void fresh(const RunParams& R, const DevPoint* __restrict__ P, StrictLane& L) { fresh_state<true>(R.S, P, L); }
	// what the fast functions cover; other states go to the one-lane pass
	static __device__ __forceinline__ bool fits(const StrictLane& L)
	{
		return (L.hot().pr.radial_mode == 0) & (L.hot().pr.J > 0x1p-200) & (L.hot().pr.J < 0x1p200) & fast::in_radius_range(L.hot().pr.radius) & (fabs(L.hot().pr.phi) < 0x1p20);
	}
	static __device__ __forceinline__ void propagate(const RunParams& R, const Box& b, const TeamState& s, TeamState& n) { strict_propagate(R, b, s, n); }
	static __device__ __forceinline__ int judge(const RunParams& R, const Box& b, TeamState& s, const Event& e, const TeamState& n, Event& en, StrictLane& L,
	                                            bool mine, double* buffer, StepCtx& c)
	{
		return strict_judge(R, b, s, e, n, en, L, mine, buffer, c);
	}
	static __device__ __forceinline__ void commit(const RunParams& R, const Box& b, StrictLane& L, const Event& e) { strict_commit(R, b, L, e); }
	// The end of a step that reaches the boundary or a scattering, as in strict_step: `phase` is the lane's next.
	static __device__ __forceinline__ void finish(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, StrictLane& L, double2* hist, StepCtx& c,
	                                              const TeamState& n, bool scattering, int& phase)
	{
		int boundary = BOUNDARY_INSIDE;
		if(!scattering)
			boundary = boundary_step(R, m_dm, L, hist, c);
		else
		{
			const bool depth = c.s1 > c.s0;
			scatter_point<true>(R.S, P, c, L.hot().next_rate, depth && c.r_before < DMS_RSUN_KM && c.s0 <= 1.0e-12, depth,
			              R.capture_mode ? DMS_CAPTURE_OPTICAL_DEPTH_PIECES : DMS_MAX_OPTICAL_DEPTH_PIECES, L.hot().tau, c.after);
		}
		if(boundary == BOUNDARY_FAILURE)
			phase = PH_FINAL;
		else if(boundary != BOUNDARY_RETURN)
			phase = finish_step<true>(R, m_dm, L, hist, c, scattering, boundary, n.time, n.radius, n.phi, n.v_radial, n.step, n.rate, true);
	}
};

// Initial_Conditions + Hyperbolic_Kepler_Shift of every work index (src/Data_Generation.cpp:747-761,
// src/Simulation_Utilities.cpp:123-321), ahead of the trajectory launch.  A lane takes every n-th work index
// in turn and makes one rejection try per pass; the lanes of a warp make the kind of try that most of them
// are at, and finish trajectories when most of them have one, so that a lane whose tries are rejected does not
// hold 31 others.  Bound by FP64 and instruction supply: 3 200 instructions in all, the tries fit the
// instruction cache.  2^20 trajectories 11.0 -> 5.3 ms, 16 384 0.62 -> 0.31 ms, 64 0.30 -> 0.07 ms, against one
// trajectory per thread with everything inline (6 800 instructions).
enum InitPhase : int
{
	INIT_FETCH = 0,
	INIT_SPEED = 1,   // a try for the speed
	INIT_BOUND = 2,   // the bound of the cosine's density: the density at -1
	INIT_COSINE = 3,  // a try for the cosine
	INIT_FINISH = 4,
	INIT_DONE = 5,
};

__global__ void __launch_bounds__(128) initial_state_kernel(const RunParams R, int lanes_per_warp)
{
	constexpr unsigned int FULL_WARP = 0xffffffffu;
	const int in_warp = threadIdx.x & 31;
	const uint64_t warp = blockIdx.x * static_cast<uint64_t>(blockDim.x >> 5) + (threadIdx.x >> 5);
	const uint64_t lanes = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5) * lanes_per_warp;
	uint64_t w = warp * lanes_per_warp + in_warp;
	int phase = in_warp < lanes_per_warp && w < R.total ? INIT_FETCH : INIT_DONE, point = -1, tries = 0;
	bool ok = true;
	Draws D;
	Sampler h;
	double u = 0.0, cosine = 0.0, cos_max = 0.0, y_max = 0.0, normalization = 0.0;
	for(;;)
	{
		if(__all_sync(FULL_WARP, phase == INIT_DONE))
			break;
		if(phase == INIT_FETCH)
		{
			int k = find_range(R, w);
			DMS_CHECK_INDEX(k, 0, R.n_ranges, BOUNDS_RANGE);
			if(R.range_point[k] != point)
			{
				point = R.range_point[k];
				sampler_init(R.S, R.points + point, h);
			}
			D.seed = R.seed;
			D.point = static_cast<uint32_t>(point);
			D.traj = R.range_first[k] + (w - R.range_offset[k]);
			D.index = 0;
			tries = 0;
			ok = true;
			phase = INIT_SPEED;
		}
		const int n_speed = __popc(__ballot_sync(FULL_WARP, phase == INIT_SPEED));
		const int n_cosine = __popc(__ballot_sync(FULL_WARP, phase == INIT_BOUND || phase == INIT_COSINE));
		const int n_finish = __popc(__ballot_sync(FULL_WARP, phase == INIT_FINISH));
		if(n_finish >= n_speed + n_cosine)
		{
			if(phase == INIT_FINISH)
			{
				Event ic;
				if(ok)
					initial_event(R.S, h, D, u, cosine, ic);
				else
				{
					ic.t = 0.0;
					ic.x = mk(0.0, 0.0, 0.0);
					ic.v = mk(0.0, 0.0, 0.0);
					atomicOr(R.status, STATUS_IC_REJECTION);
				}
				const bool shifted = ok && hyperbolic_kepler_shift(ic, R.boundary);
				InitState st;
				st.ic = ic;
				st.draws = static_cast<uint32_t>(D.index);
				st.flags = (ok ? INIT_IC_OK : 0u) | (shifted ? INIT_SHIFT_OK : 0u);
				R.init[w] = st;
				w += lanes;
				phase = w < R.total ? INIT_FETCH : INIT_DONE;
			}
		}
		else if(n_speed >= n_cosine)
		{
			if(phase == INIT_SPEED)
			{
				const double x = draw_between(D, 0.0, h.v_max);
				const double y = draw_between(D, 0.0, DMS_IC_SPEED_YMAX_NATURAL / DMS_C_KMS);
				tries++;
				if(y <= pdf_initial_speed(h, x))
				{
					u = x;
					const double v_gal = h.v_max - h.v_sun;
					cos_max = (h.v_sun == 0.0) ? 1.0 : (v_gal * v_gal - h.v_sun * h.v_sun - u * u) / (2.0 * u * h.v_sun);
					if(cos_max > 1.0)
						cos_max = 1.0;
					normalization = 2.0 * DMS_PI * u * u / halo_pdf_speed(h, u);
					tries = 0;
					phase = INIT_BOUND;
				}
				else if(tries >= R.ic_max_attempts)
				{
					ok = false;
					phase = INIT_FINISH;
				}
			}
		}
		else if(phase == INIT_BOUND || phase == INIT_COSINE)
		{
			// (the bound takes no draws)
			const bool bound = phase == INIT_BOUND;
			double x = -1.0, y = 0.0;
			if(!bound)
			{
				x = draw_between(D, -1.0, cos_max);
				y = draw_between(D, 0.0, y_max);
				tries++;
			}
			const double density = pdf_cos_theta(h, x, u, normalization);
			if(bound)
			{
				y_max = density;
				phase = INIT_COSINE;
			}
			else if(y <= density)
			{
				cosine = x;
				phase = INIT_FINISH;
			}
			else if(tries >= R.ic_max_attempts)
			{
				ok = false;
				phase = INIT_FINISH;
			}
		}
	}
}

template <bool THROUGHPUT>
struct StrictStep : Team<StrictTeam>
{
	static constexpr bool throughput = THROUGHPUT;
	static constexpr int threads = THROUGHPUT ? MAX_THREADS : LATENCY_THREADS;
	// in both forms: four warps with a scheduler each share the instruction cache too (4 096 histories of
	// m = 1 GeV, 1e-35 cm^2 cut at 300 scatterings 196 -> 173 ms, 8 192 273 -> 208 ms)
	static constexpr bool lockstep = true;
	static constexpr int buffer = COOP_BUFFER;
	__device__ __forceinline__ int operator()(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, StrictLane& L, double2* hist, int phase,
	                                          double* buffer) const
	{
		return strict_step<THROUGHPUT ? 1 : 6>(R, P, m_dm, L, hist, phase, buffer);
	}
	static constexpr bool team = !THROUGHPUT;
	__device__ __forceinline__ double channel(const DevSolar& S, const DevPoint* __restrict__ P, int i, double dr, double T, double v, int k) const
	{
		return channel_rate(S, P, i, dr, T, v, k);
	}
	__device__ __forceinline__ bool scatter(const DevSolar& S, const DevPoint* __restrict__ P, Draws& D, Event& e, int target) const
	{
		return scatter_with_target(S, P, D, e, target);
	}
};

// The throughput form: up to 16 warps per SM in lockstep, 128 registers each.
__global__ void __launch_bounds__(MAX_THREADS, 1) trajectory_kernel(const RunParams R)
{
	lane_loop<StrictLane>(R, StrictStep<true>());
}

// The latency form: one warp per scheduler, no spills (196 registers).
__global__ void __launch_bounds__(LATENCY_THREADS, 1) trajectory_kernel_latency(const RunParams R)
{
	lane_loop<StrictLane>(R, StrictStep<false>());
}

__global__ void rate_grid_kernel(const DevSolar S, const DevPoint* __restrict__ P, double* grid, int n)
{
	const size_t total = static_cast<size_t>(n) * n;
	for(size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < total; k += static_cast<size_t>(gridDim.x) * blockDim.x)
	{
		const int i = static_cast<int>(k / n), j = static_cast<int>(k % n);
		// src/Solar_Model.cpp:438-447: radius = R i/(N-1), speed = Linear_Space(0, 0.75, N)[j]
		const double radius = DMS_RSUN_KM * static_cast<double>(i) / static_cast<double>(n - 1);
		const double vstep_c = (DMS_V_MAX_C - 0.0) / (n - 1);
		const double speed = (0.0 + j * vstep_c) * DMS_C_KMS;
		grid[k] = rate_computed(S, P, radius, speed, nullptr, nullptr);
	}
}

__global__ void rate_query_kernel(const DevSolar S, const DevPoint* __restrict__ P, int interpolated, const double* r, const double* v, double* out, size_t n)
{
	const size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
	if(k >= n)
		return;
	out[k] = interpolated ? rate_total(S, P, r[k], v[k]) : rate_computed(S, P, r[k], v[k], nullptr, nullptr);
}

// Independent DFMA chains: 8 accumulators per thread, `iters` iterations.
__global__ void __launch_bounds__(256) fp64_fma_probe_kernel(double* out, int iters, double b, double c)
{
	double a0 = threadIdx.x, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3, a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6, a7 = a0 + 7;
	for(int i = 0; i < iters; i++)
	{
		a0 = fma(a0, b, c);
		a1 = fma(a1, b, c);
		a2 = fma(a2, b, c);
		a3 = fma(a3, b, c);
		a4 = fma(a4, b, c);
		a5 = fma(a5, b, c);
		a6 = fma(a6, b, c);
		a7 = fma(a7, b, c);
	}
	const double s = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
	if(s == 1.2345)
		out[0] = s;
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
	x += 0x9e3779b97f4a7c15ULL;
	x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
	x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
	return x ^ (x >> 31);
}

// A double with random significand and an exponent uniform in [lo, hi].
__device__ __forceinline__ double random_double(uint64_t bits, int lo, int hi)
{
	const int e = lo + static_cast<int>((bits >> 52) % static_cast<uint64_t>(hi - lo + 1));
	const uint64_t mant = bits & 0x000fffffffffffffULL;
	return __longlong_as_double(static_cast<long long>((static_cast<uint64_t>(e + 1023) << 52) | mant));
}

// Self-test of the certified division and square root against IEEE `/` and sqrt on n random
// operand pairs: out[0] quotients inside the straight-line range whose bits differ from IEEE (must
// be 0), out[1] pairs outside that range, out[2] and out[3] the same for the root.
// Operands: random exponents in the ranges of the trajectory arithmetic, arbitrary bit patterns
// (NaN, infinities, subnormals, zeros), quotients within a few ulp of representable values, exact
// quotients (a power-of-two divisor), and the whole range of fast::div.  Division and square root never land exactly
// halfway between two doubles, so round-to-nearest has no ties to test.
__global__ void certified_math_check_kernel(uint64_t n, uint64_t seed, unsigned long long* out)
{
	unsigned long long c[4] = {0, 0, 0, 0};
	for(uint64_t k = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; k < n; k += static_cast<uint64_t>(gridDim.x) * blockDim.x)
	{
		const uint64_t h1 = splitmix64(seed ^ (k * 0x2545f4914f6cdd1dULL)), h2 = splitmix64(h1), h3 = splitmix64(h2);
		double a, b;
		switch((k & 7) == 7 ? 4 : static_cast<int>(k & 3))
		{
			case 0:  // the trajectory ranges: km, km/s, s, km^3/s^2
				a = random_double(h1, -40, 70);
				b = random_double(h2, -20, 40);
				break;
			case 1:  // any bit pattern
				a = __longlong_as_double(static_cast<long long>(h1));
				b = __longlong_as_double(static_cast<long long>(h2));
				break;
			case 2:
			{  // dividend a few ulp away from b * q for a random q
				b = random_double(h1, -30, 30);
				const double q = random_double(h2, -30, 30);
				const long long d = static_cast<long long>(h3 % 7) - 3;
				a = __longlong_as_double(__double_as_longlong(__dmul_rn(b, q)) + d);
				break;
			}
			case 3:
			{  // exact quotients: a power-of-two divisor
				const double m = random_double(h1, -10, 10);
				b = ldexp(1.0, static_cast<int>(h2 % 41) - 20);
				a = __dmul_rn(b, m);
				break;
			}
			default:  // the ends of the range
				a = random_double(h1, -700, 400);
				b = random_double(h2, -200, 399);
				break;
		}
		if(h3 & 1)
			a = -a;
		// pairs outside the range of fast::div count as fallbacks (a zero dividend's quotient has no sign there)
		bool ok = fast::in_division_range(a, b) & ((a != 0.0) | (__double_as_longlong(a) == 0 && b > 0.0));
		const double q = fast::div(a, fast::recip(b, ok));
		const double ref = a / b;
		if(!ok)
			c[1]++;
		else if(__double_as_longlong(q) != __double_as_longlong(ref) && !(isnan(q) && isnan(ref)))
			c[0]++;
		const double x = fabs(a);
		bool ok2 = true;
		const double sq = fast::sqrt(x, ok2);
		const double sref = sqrt(x);
		if(!ok2)
			c[3]++;
		else if(__double_as_longlong(sq) != __double_as_longlong(sref) && !(isnan(sq) && isnan(sref)))
			c[2]++;
	}
	for(int i = 0; i < 4; i++)
		if(c[i])
			atomicAdd(out + i, c[i]);
}

}	// namespace

void Check_Certified_Math(uint64_t n, uint64_t seed, unsigned long long* out, int sm_count, cudaStream_t stream)
{
	certified_math_check_kernel<<<sm_count * 8, 256, 0, stream>>>(n, seed, out);
}

double Measure_FP64_Peak(int sm_count, cudaStream_t stream)
{
	double* d = nullptr;
	if(cudaMalloc(&d, sizeof(double)) != cudaSuccess)
		return -1.0;
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	const int blocks = sm_count * 8, threads = 256, iters = 1 << 16;
	fp64_fma_probe_kernel<<<blocks, threads, 0, stream>>>(d, 1024, 0.999999, 1e-9);
	cudaEventRecord(e0, stream);
	fp64_fma_probe_kernel<<<blocks, threads, 0, stream>>>(d, iters, 0.999999, 1e-9);
	cudaEventRecord(e1, stream);
	float ms = 0.0f;
	const bool ok = cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess;
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaFree(d);
	if(!ok || ms <= 0.0f)
		return -1.0;
	const double flops = 2.0 * 8.0 * iters * static_cast<double>(blocks) * threads;
	return flops / (ms * 1.0e-3) / 1.0e12;
}

void Launch_Initial_States(const RunParams& p, cudaStream_t stream)
{
	// one warp per scheduler with as few lanes as will do (a lane alone makes only its own tries), then
	// whole warps, five blocks of four per SM
	const uint64_t few = 148 * 4;
	const int lanes = static_cast<int>(p.total >= 32 * few ? 32 : (p.total + few - 1) / few);
	if(lanes == 0)
		return;
	const uint64_t wanted = (p.total + 4 * lanes - 1) / (4 * lanes);
	const uint64_t blocks = wanted < 148 * 5 ? wanted : 148 * 5;
	initial_state_kernel<<<static_cast<unsigned int>(blocks), 128, 0, stream>>>(p, lanes);
}

void Launch_Trajectories(const RunParams& p, int blocks, int threads, cudaStream_t stream)
{
	const auto kernel = threads <= LATENCY_THREADS ? trajectory_kernel_latency : trajectory_kernel;
	Launch_With_Hot_States<StrictLane>(kernel, p, blocks, threads, stream);
}

void Launch_Rate_Grid(const DevSolar& S, const DevPoint* point, double* grid, int n, cudaStream_t stream)
{
	rate_grid_kernel<<<148 * 8, 256, 0, stream>>>(S, point, grid, n);
}

void Launch_Rate_Query(const DevSolar& S, const DevPoint* point, int interpolated, const double* r, const double* v, double* out,
                       size_t n, cudaStream_t stream)
{
	const int threads = 128;
	const int blocks = static_cast<int>((n + threads - 1) / threads);
	if(blocks > 0)
		rate_query_kernel<<<blocks, threads, 0, stream>>>(S, point, interpolated, r, v, out, n);
}

#ifdef DMS_CHECKED
bool Take_Form_Counts(unsigned long long* counts)
{
	const unsigned long long zero[FORM_COUNTS] = {};
	return cudaMemcpyFromSymbol(counts, dms_form_counts, sizeof zero) == cudaSuccess &&
	       cudaMemcpyToSymbol(dms_form_counts, zero, sizeof zero) == cudaSuccess && cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess;
}
#endif

unsigned int Take_Bounds_Status()
{
#ifdef DMS_CHECKED
	unsigned int bits = 0;
	const unsigned int zero = 0;
	if(cudaMemcpyFromSymbol(&bits, dms_bounds_status, sizeof bits) != cudaSuccess ||
	   cudaMemcpyToSymbol(dms_bounds_status, &zero, sizeof zero) != cudaSuccess ||
	   cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess)  // ahead of what runs on the context's stream
		return ~0u;
	return bits;
#else
	return 0;
#endif
}

}	// namespace dms
