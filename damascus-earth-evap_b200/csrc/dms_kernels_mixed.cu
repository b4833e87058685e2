// Mixed-precision trajectory kernel (the batched-FP32 form).  Compiled with FMA contraction;
// shares the lane state machine (dms_lane.cuh) with the FP64 kernel.
#define DMS_FMA_CONTRACTION 1
#include "dms_device_mixed.cuh"
#include "dms_lane.cuh"
#include "dms_team.cuh"

namespace dms
{
namespace mixed
{
// found by argument-dependent lookup from the lane state machine
__device__ __forceinline__ void init_propagator(PropF& p, const Event& e) { prop_init_f(p, e); }
}	// namespace mixed

namespace
{
using namespace lane;
using namespace mixed;
using MixedLane = LaneT<PropF, EventF>;

// The mixed-precision pass (see dms_kernels.cu for the FP64 one, whose structure this follows, and
// dms_device_mixed.cuh for what stays FP64): the Propagate_Freely loop body,
// src/Simulation_Trajectory.cpp:876-1116, split at the RK45 retry loop.

__device__ __forceinline__ DevSolarF tables_f(const RunParams& R) { return DevSolarF{R.sf_knots, R.sf_vesc2_s, R.sf_bucket, R.sf_scale, R.S.nbuckets, R.sf_single_step, R.S.n}; }

__device__ __forceinline__ const float* grid_f(const DevPoint* __restrict__ P)
{
	return reinterpret_cast<const float*>(__ldg(reinterpret_cast<const unsigned long long*>(&P->grid_f)));
}

// The event, speed and scattering rate at the propagator's state, at the start of a free segment.
__device__ __forceinline__ void fresh_state(const DevSolar& S, const DevPoint* __restrict__ P, MixedLane& L)
{
	if(!L.hot().before_valid)
		L.hot().before = prop_event_f(L.hot().pr);
	L.hot().before_valid = L.hot().before_valid ? L.hot().before_valid : 1;
	const double r = prop_radius_f(L.hot().pr);
	L.hot().next_speed = prop_speed_f(L.hot().pr);
	L.hot().next_rate = r >= DMS_RSUN_KM ? 0.0 : rate_total_f(S, P, grid_f(P), static_cast<float>(r), static_cast<float>(L.hot().next_speed));
	L.hot().next_valid = 1;
}

static __device__ __noinline__ int end_at_propagator(MixedLane& L, int reason)
{
	set_final(L, to_event64(prop_event_f(L.hot().pr)), true, reason);
	return PH_FINAL;
}

__device__ __forceinline__ double surface_step(const EventF& before, double r, double step)
{
	const double vr = (r > 0.0) ? static_cast<double>(dotf(before.x, before.v)) / r : 0.0;
	if(r > DMS_RSUN_KM && vr < 0.0)
	{
		const double est = (r - DMS_RSUN_KM) / (-vr);
		if(isfinite(est) && est > 0.0)
		{
			const double lim = est > DMS_RK45_ABS_MIN_STEP_S ? est : DMS_RK45_ABS_MIN_STEP_S;
			step = lim < step ? lim : step;
		}
	}
	return step;
}

// The bound of a step inside the Sun by its optical depth.
__device__ __forceinline__ double inside_step(const RunParams& R, double rate, double step)
{
	if(rate > 0.0)
	{
		const double tau_limit = R.capture_mode ? DMS_CAPTURE_MAX_OPTICAL_DEPTH_STEP : DMS_MAX_OPTICAL_DEPTH_STEP;
		const float lim = static_cast<float>(tau_limit) / static_cast<float>(rate);
		if(static_cast<double>(lim) < step)
			step = static_cast<double>(lim);
	}
	return step;
}

// Pre-step bounds (src/Simulation_Trajectory.cpp:873-927).
__device__ __forceinline__ int mixed_begin(const RunParams& R, const DevPoint* __restrict__ P, MixedLane& L)
{
	if(!(L.hot().seg_steps < R.max_free_steps))
	{
		if(L.hot().before_valid == 2)  // otherwise L.cur holds the last committed event
		{
			L.cur = to_event64(L.hot().before);
			L.cur.t += L.hot().origin;
		}
		L.reason = DMS_REASON_MAX_FREE_STEPS;
		return PH_FINAL;
	}
	if(wall_time_exceeded(R, L))  // "before_step", src/Simulation_Trajectory.cpp:873-874
		return end_at_propagator(L, DMS_REASON_WALL_TIME_LIMIT);
	if(!L.hot().next_valid)
		fresh_state(R.S, P, L);
	const double r = prop_radius_f(L.hot().pr);
	double step = sanitized_step(L.hot().pr.time_step), rate = 0.0;
	if(r >= DMS_RSUN_KM)
	{
		step = capped_step(r, L.hot().next_speed, step, R.boundary);
		if(!surface_is_far(r, static_cast<double>(dotf(L.hot().before.x, L.hot().before.v)), step))
			step = surface_step(L.hot().before, r, step);
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

// A step as an accepted attempt leaves it.
struct StepCtxF
{
	const EventF* before;  // the lane's own, not a copy
	EventF after;
	double r_before, r_after, v_after, dt;
	float s0, s1;
};

// Whether a chord with both ends clearly outside the Sun passes clear of it (as in dms_kernels.cu, with a
// margin of 10^-4 for the FP32 events).
__device__ __forceinline__ bool chord_stays_outside(const EventF& a, const EventF& b, double ra, double rb)
{
	const F3 d = f3(b.x.x - a.x.x, b.x.y - a.x.y, b.x.z - a.x.z);
	const float ad = dotf(a.x, d), bd = dotf(b.x, d), dd = dotf(d, d);
	const float lim = static_cast<float>(DMS_RSUN_KM * (1.0 + 1.0e-4)), r = static_cast<float>(ra);
	return (ra > static_cast<double>(lim)) & (rb > static_cast<double>(lim)) &
	       ((ad >= 0.0f) | (bd <= 0.0f) | ((r - lim) * (r + lim) * dd > ad * ad * 1.0001f));
}

__device__ __forceinline__ bool interior_interval_outside(const EventF& a, const EventF& b, double ra, double rb, float& s0, float& s1)
{
	return interior_interval_f(a, b, ra, rb, s0, s1);
}

// One piece-boundary rate of a step or, with `next`, the scattering rate at the state after it.
__device__ __forceinline__ float piece_rate_f(const DevSolar& S, const DevPoint* __restrict__ P, const float* __restrict__ grid, const EventF& a,
                                              const EventF& b, float f, bool next, float ra, float va)
{
	f = f < 0.0f ? 0.0f : (f > 1.0f ? 1.0f : f);
	const float x = a.x.x + f * (b.x.x - a.x.x), vx = a.v.x + f * (b.v.x - a.v.x);
	const float y = a.x.y + f * (b.x.y - a.x.y), vy = a.v.y + f * (b.v.y - a.v.y);
	const float z = a.x.z + f * (b.x.z - a.x.z), vz = a.v.z + f * (b.v.z - a.v.z);
	float r = sqrtf(fmaxf(x * x + y * y + z * z, 0.0f));
	float v = sqrtf(fmaxf(vx * vx + vy * vy + vz * vz, 0.0f));
	if(!next && r >= static_cast<float>(DMS_RSUN_KM))
		return 0.0f;
	r = next ? ra : r;
	v = next ? va : v;
	return rate_total_f(S, P, grid, r, v);
}

// The optical depth of a step in FP32 (at most 0.1), as in dms_kernels.cu.
struct DepthF
{
	float dtau, tau2, next_rate;
	bool invalid;
};

struct DepthSumsF
{
	float f_prev, r_prev, f_0, r_0;
	__device__ __forceinline__ void add(DepthF& d, int i, float f, float rate, float dt)
	{
		if(!isfinite(rate) || rate < 0.0f)
			d.invalid = true;
		if(i == 0)
		{
			f_0 = f;
			r_0 = rate;
		}
		else
		{
			if(f > f_prev)
				d.dtau += 0.5f * (r_prev + rate) * (dt * (f - f_prev));
			if((i & 1) == 0)
			{
				d.tau2 += 0.5f * (r_0 + rate) * (dt * (f - f_0));
				f_0 = f;
				r_0 = rate;
			}
		}
		f_prev = f;
		r_prev = rate;
	}
};

__device__ __forceinline__ void lane_depth(const RunParams& R, const DevPoint* __restrict__ P, const StepCtxF& c, float rate_before, bool first_known,
                                           int pieces, DepthF& d)
{
	const float* grid = grid_f(P);
	const float fraction = pieces == 4 ? 0.25f : 0.5f, span = c.s1 - c.s0, dt = static_cast<float>(c.dt);
	DepthSumsF sums = {};
#pragma unroll 1
	for(int i = 0; i <= pieces + 1; i++)
	{
		const float f = c.s0 + static_cast<float>(i) * fraction * span;
		float rate = rate_before;
		if(i > 0 || !first_known)
			rate = piece_rate_f(R.S, P, grid, *c.before, c.after, f, i > pieces, static_cast<float>(c.r_after), static_cast<float>(c.v_after));
		if(i <= pieces)
			sums.add(d, i, f, rate, dt);
		else
			d.next_rate = rate;
	}
}

constexpr int COOP_SLOT_F = 18;  // floats of a step handed over (the point's address among them)
constexpr int COOP_SLOTS_F = 8;
constexpr int COOP_BUFFER_F = (COOP_SLOT_F * COOP_SLOTS_F + 32) / 2;  // in doubles
__device__ __forceinline__ void warp_depth(const RunParams& R, const DevPoint* __restrict__ P, const StepCtxF& c, float rate_before, bool first_known,
                                           int pieces, unsigned int dm, bool mine, float* buffer, DepthF& d)
{
	const float fraction = pieces == 4 ? 0.25f : 0.5f, dt = static_cast<float>(c.dt);
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
			float* b = buffer + slot * COOP_SLOT_F;
			b[0] = c.before->x.x; b[1] = c.before->x.y; b[2] = c.before->x.z;
			b[3] = c.before->v.x; b[4] = c.before->v.y; b[5] = c.before->v.z;
			b[6] = c.after.x.x; b[7] = c.after.x.y; b[8] = c.after.x.z;
			b[9] = c.after.v.x; b[10] = c.after.v.y; b[11] = c.after.v.z;
			b[12] = c.s0; b[13] = c.s1 - c.s0;
			b[14] = static_cast<float>(c.r_after); b[15] = static_cast<float>(c.v_after);
			*reinterpret_cast<const DevPoint**>(b + 16) = P;
		}
		__syncwarp();
		float rate = 0.0f;
		if(slot_of_job < slots && base + slot_of_job < steps)
		{
			const float* b = buffer + slot_of_job * COOP_SLOT_F;
			const DevPoint* Po = *reinterpret_cast<const DevPoint* const*>(b + 16);
			const EventF before{0.0, f3(b[0], b[1], b[2]), f3(b[3], b[4], b[5])}, after{0.0, f3(b[6], b[7], b[8]), f3(b[9], b[10], b[11])};
			rate = piece_rate_f(R.S, Po, grid_f(Po), before, after, b[12] + static_cast<float>(j) * fraction * b[13], j > pieces, b[14], b[15]);
		}
		buffer[COOP_SLOT_F * COOP_SLOTS_F + me] = rate;
		__syncwarp();
		if(owner)
		{
			const float* q = buffer + COOP_SLOT_F * COOP_SLOTS_F + slot * rates;
			const float span = c.s1 - c.s0;
			DepthSumsF sums = {};
			sums.add(d, 0, c.s0, first_known ? rate_before : q[0], dt);
			sums.add(d, 1, c.s0 + fraction * span, q[1], dt);
			sums.add(d, 2, c.s0 + 2.0f * fraction * span, q[2], dt);
			if(pieces == 4)
			{
				sums.add(d, 3, c.s0 + 3.0f * fraction * span, q[3], dt);
				sums.add(d, 4, c.s0 + 4.0f * fraction * span, q[4], dt);
			}
			d.next_rate = q[rates - 1];
		}
		__syncwarp();
	}
}

// A step whose optical depth exceeds the limit or whose two estimates differ too much
// (src/Simulation_Trajectory.cpp:975-1011).
constexpr int PH_CONTINUE = -1;
__device__ __forceinline__ int depth_reject(MixedLane& L, const EventF& before, float dtau_f, float tau2, bool capture_mode, double dt, double tau_limit)
{
	const double dtau = static_cast<double>(dtau_f);
	const float scale = dtau_f > static_cast<float>(DMS_OPTICAL_DEPTH_ABS_TOL) ? dtau_f : static_cast<float>(DMS_OPTICAL_DEPTH_ABS_TOL);
	const double rel = static_cast<double>(fabsf(dtau_f - tau2) / scale);
	const bool reject_acc = !capture_mode && rel > DMS_OPTICAL_DEPTH_REL_TOL;
	if(!(dtau > tau_limit) && !reject_acc)
		return PH_CONTINUE;
	L.hot().retries++;
	if(L.hot().retries > DMS_MAX_OPTICAL_DEPTH_RETRIES)
	{
		set_final(L, to_event64(before), true, DMS_REASON_NUMERICAL_FAILURE);
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
	return PH_STEP;
}

// The scattering point (src/Simulation_Trajectory.cpp:1013-1044), the boundary rates formed again.
__device__ __forceinline__ void scatter_point(const DevSolar& S, const DevPoint* __restrict__ P, const StepCtxF& c, float rate_before, bool first_known,
                                                  bool depth, int pieces, double remaining, EventF& accepted)
{
	if(depth)
	{
		const float* grid = grid_f(P);
		const float fraction = pieces == 4 ? 0.25f : 0.5f, span = c.s1 - c.s0;
		float f_prev = c.s0, r_prev = rate_before;
		if(!first_known)
			r_prev = rate_at_fraction_f(S, P, grid, *c.before, c.after, f_prev);
#pragma unroll 1
		for(int k = 1; k <= pieces; k++)
		{
			const float f = c.s0 + static_cast<float>(k) * fraction * span;
			const float rate = rate_at_fraction_f(S, P, grid, *c.before, c.after, f);
			if(f > f_prev)
			{
				const double pdt = c.dt * static_cast<double>(f - f_prev);
				const double ptau = 0.5 * static_cast<double>(r_prev + rate) * pdt;
				if(ptau >= remaining)
				{
					const double lf = solve_linear_rate(r_prev, rate, pdt, remaining);
					accepted = interpolate_event_f(*c.before, c.after, f_prev + static_cast<float>(lf) * (f - f_prev));
					return;
				}
				remaining -= ptau;
			}
			f_prev = f;
			r_prev = rate;
		}
	}
	accepted = interpolate_event_f(*c.before, c.after, c.s1);
}

// commit_accepted_event (src/Simulation_Trajectory.cpp:842-874) for an FP32 event: bincount
// with FP64 times, capture energy of the drift statistics and the uncaptured-bound guard in FP32
// (m_dm / (2 c^2) in FP64 first).  Returns the energy when evaluated, NaN otherwise.
__device__ __forceinline__ double commit_event_mixed(const RunParams& R, double m_dm, MixedLane& L, double2* hist, const EventF& local)
{
	if(R.capture_mode && !L.hot().is_captured)
		return NAN;
	const float rf = normf(local.x), vf = normf(local.v);
	const double r_now = static_cast<double>(rf);
	const double v_now = static_cast<double>(vf);
	if(!R.capture_mode)
	{
		if(L.prev_time >= 0.0)
			accumulate_bincount(L, hist, L.prev_r, L.prev_v2, local.t - L.prev_time);
		L.prev_time = local.t;
		L.prev_r = r_now;
		L.prev_v2 = v_now * v_now;
	}
	const double t_abs = local.t + L.hot().origin;
	const DevSolarF F = tables_f(R);
	const double E = capture_energy_eV_f(F, m_dm, rf, vf);
	if(L.hot().is_captured && isfinite(L.free_flight_E))
	{
		const double drift = fabs(E - L.free_flight_E);
		if(isfinite(drift) && drift > L.max_drift_eV)
			L.max_drift_eV = drift;
		const double ref = fabs(L.free_flight_E);
		const double scale = ref > DMS_FREE_ENERGY_DRIFT_REL_E_SCALE_EV ? ref : DMS_FREE_ENERGY_DRIFT_REL_E_SCALE_EV;
		// the quotient is formed only where it can be the larger one
		if(drift * (1.0 + 0x1p-50) >= L.max_drift_rel * scale)
		{
			const double rel = drift / scale;
			if(isfinite(rel) && rel > L.max_drift_rel)
				L.max_drift_rel = rel;
		}
	}
	if(L.bound_state && L.hot().is_captured)
		L.t_last_bound = t_abs;
	return E;
}

// abort_if_uncaptured_bound (src/Simulation_Trajectory.cpp:767-778, 1108) in Capture mode, where the commit
// forms no energy: the FP64 energy of the event decides unless the FP32 speeds are far apart.
__device__ __forceinline__ bool not_free_general(const DevSolar& S, double m_dm, const EventF& e)
{
	const Event d = to_event64(e);
	const double E = capture_energy_eV(S, m_dm, ev_radius(d), ev_speed(d));
	return !(isfinite(E) && E >= 0.0);
}
__device__ __forceinline__ bool not_free(const RunParams& R, double m_dm, const EventF& e)
{
	const float r2 = dotf(e.x, e.x), v2 = dotf(e.v, e.v);
	const float r = sqrtf(r2);
	const bool inside = r < static_cast<float>(DMS_RSUN_KM * (1.0 - 1.0e-6));
	const DevSolarF F = tables_f(R);
	float need = static_cast<float>(2.0 * DMS_GMSUN_KM3S2);
	if(inside)
		need = vesc2_f(F, r);
	const float have = inside ? v2 : v2 * r;
	const bool clear = (have > need * 1.001f) & (v2 < 1.0e12f) & (r < 1.0e12f);
	return clear ? false : not_free_general(R.S, m_dm, e);
}

// A step that ends at or beyond the boundary radius (src/Simulation_Trajectory.cpp:1046-1086).
enum Boundary : int
{
	BOUNDARY_INSIDE = 0,
	BOUNDARY_ESCAPE = 1,
	BOUNDARY_RETURN = 2,
	BOUNDARY_FAILURE = 3,
};
static __device__ __noinline__ int boundary_step(const RunParams& R, double m_dm, MixedLane& L, double2* hist, StepCtxF& c)
{
	const DevSolar& S = R.S;
	EventF ev = c.after;
	double r_b = c.r_after, v_b = c.v_after;
	if(c.r_before < R.boundary && c.r_after >= R.boundary && c.r_after > c.r_before)
	{
		const double f = (R.boundary - c.r_before) / (c.r_after - c.r_before);
		ev = interpolate_event_f(*c.before, c.after, static_cast<float>(f));
		r_b = normf(ev.x);
		v_b = normf(ev.v);
	}
	if(!(r_b >= R.boundary && r_b >= c.r_before))
		return BOUNDARY_INSIDE;
	if(v_b > solar_vesc(S, r_b))
	{
		c.after = ev;
		return BOUNDARY_ESCAPE;
	}
	Event abs_b = to_event64(ev);
	abs_b.t += L.hot().origin;
	if(uncaptured_bound(S, m_dm, L, abs_b))
	{
		set_final(L, abs_b, false, DMS_REASON_NUMERICAL_FAILURE);
		return BOUNDARY_FAILURE;
	}
	Event inbound;
	if(!bound_kepler_return(to_event64(ev), inbound))
		return BOUNDARY_INSIDE;
	L.hot().seg_steps++;
	L.hot().steps++;
	L.hot().retries = 0;
	// (in place: its radius is contracted as r_b is, so that both lie on the same side of the outermost bin's edge)
	commit_event_mixed(R, m_dm, L, hist, ev);
	// reset_propagator_at_absolute_event, src/Simulation_Trajectory.cpp:814-822
	L.cur = inbound;
	L.cur.t += L.hot().origin;
	L.hot().origin = L.cur.t;
	Event local = inbound;
	local.t = 0.0;
	prop_init_f(L.hot().pr, local);
	L.hot().before_valid = 0;
	L.hot().next_valid = 0;
	if(!R.capture_mode && L.prev_time >= 0.0)
		L.prev_time = 0.0;
	return BOUNDARY_RETURN;
}

// as in dms_kernels.cu
constexpr int COOP_MAX_STEPS = 15;

// The end of a step that has not been rejected, for the committed event c.after and the propagator after it.
__device__ __forceinline__ int finish_step(const RunParams& R, double m_dm, MixedLane& L, double2* hist, const StepCtxF& c,
                                           bool scattering, int boundary, double time, double radius, double phi, double v_radial, double time_step,
                                           double next_rate, bool next_known)
{
	L.hot().seg_steps++;
	L.hot().steps++;
	L.hot().retries = 0;
	const double E = commit_event_mixed(R, m_dm, L, hist, c.after);
	const bool bound = !L.hot().is_captured && (isnan(E) ? not_free(R, m_dm, c.after) : !(isfinite(E) && E >= 0.0));
	if(bound | scattering | (boundary == BOUNDARY_ESCAPE))
	{
		L.cur = to_event64(c.after);
		L.cur.t += L.hot().origin;
		if(bound)
			L.reason = DMS_REASON_NUMERICAL_FAILURE;
		else if(!scattering)
			L.reason = DMS_REASON_OUTWARD_ESCAPE;
		else if(ev_radius(L.cur) < DMS_RSUN_KM)
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
	L.hot().next_speed = c.v_after;
	L.hot().next_rate = next_rate;
	L.hot().next_valid = next_known || c.r_after >= DMS_RSUN_KM;
	return PH_STEP;
}

// One pass for every lane of the warp (all 32 call it); returns the lane's next phase.
template <bool UNROLLED>
__device__ __forceinline__ int mixed_step(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, MixedLane& L, double2* hist, int phase,
                                          float* buffer)
{
	const int capture_mode = R.capture_mode;
	const int pieces = capture_mode ? DMS_CAPTURE_OPTICAL_DEPTH_PIECES : DMS_MAX_OPTICAL_DEPTH_PIECES;
	const double tau_limit = capture_mode ? DMS_CAPTURE_MAX_OPTICAL_DEPTH_STEP : DMS_MAX_OPTICAL_DEPTH_STEP;
	StepCtxF c;
	PropF q;
	bool done = false, interior = false, depth = false;
	int reason = 0;
	if(phase == PH_STEP && !L.hot().in_rk)
		phase = mixed_begin(R, P, L);
	if(phase == PH_STEP)
	{
		q = L.hot().pr;
		L.hot().rk_inner++;
		const int rk = rk45_attempt_f<UNROLLED>(tables_f(R), q, L.hot().rk_inner);
		if(rk == RK_RETRY)
			L.hot().pr.time_step = q.time_step;
		else
		{
			done = true;
			L.hot().in_rk = 0;
			L.hot().attempts += static_cast<uint64_t>(L.hot().rk_inner);
			c.before = &L.hot().before;
			c.r_before = prop_radius_f(L.hot().pr);
			c.dt = q.time - L.hot().pr.time;
			c.r_after = prop_radius_f(q);
			c.v_after = prop_speed_f(q);
			c.after = prop_event_f(q);
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
				c.s0 = 0.0f;
				c.s1 = 1.0f;
				interior = true;
				if(!(c.r_before < DMS_RSUN_KM && c.r_after < DMS_RSUN_KM))
				{
					c.s1 = 0.0f;
					interior = false;
					if(!chord_stays_outside(*c.before, c.after, c.r_before, c.r_after))
						interior = interior_interval_outside(*c.before, c.after, c.r_before, c.r_after, c.s0, c.s1);
				}
				depth = interior && c.s1 > c.s0;
			}
		}
	}
	const unsigned int dm = __ballot_sync(0xffffffffu, depth);
	DepthF d = {0.0f, 0.0f, 0.0f, false};
	const bool first_known = depth && c.r_before < DMS_RSUN_KM && c.s0 <= 1.0e-12f;
	const float rate_before = static_cast<float>(L.hot().rate_before);
	if(dm != 0u)
	{
		if(__popc(dm) <= COOP_MAX_STEPS)
			warp_depth(R, P, c, rate_before, first_known, pieces, dm, depth, buffer, d);
		else if(depth)
			lane_depth(R, P, c, rate_before, first_known, pieces, d);
	}
	if(!done)
		return phase;
	const double dtau = static_cast<double>(d.dtau);
	if(reason == 0 && (d.invalid || !isfinite(dtau) || dtau < 0.0))
		reason = DMS_REASON_NUMERICAL_FAILURE;
	if(reason != 0)
	{
		set_final(L, to_event64(c.after), true, reason);
		return PH_FINAL;
	}
	bool scattering = false;
	if(interior)
	{
		// the quotient of the two estimates is formed only where the step may be rejected
		const float scale = d.dtau > static_cast<float>(DMS_OPTICAL_DEPTH_ABS_TOL) ? d.dtau : static_cast<float>(DMS_OPTICAL_DEPTH_ABS_TOL);
		if((dtau > tau_limit) | (!capture_mode & (fabsf(d.dtau - d.tau2) > static_cast<float>(DMS_OPTICAL_DEPTH_REL_TOL * 0.999) * scale)))
		{
			const int rejected = depth_reject(L, *c.before, d.dtau, d.tau2, capture_mode != 0, c.dt, tau_limit);
			if(rejected != PH_CONTINUE)
				return rejected;
		}
		if(dtau >= L.hot().tau)
		{
			scatter_point(R.S, P, c, rate_before, first_known, depth, pieces, L.hot().tau, c.after);
			scattering = true;
		}
		else
			L.hot().tau -= dtau;
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
	return finish_step(R, m_dm, L, hist, c, scattering, boundary, q.time, q.radius, q.phi, q.v_radial, q.time_step,
	                   static_cast<double>(d.next_rate), depth);
}

// The three parts of a step made by a team (dms_team.cuh), as in dms_kernels.cu.
struct MixedTeam
{
	using Lane = MixedLane;
	using Box = TeamBox<PropF, EventF>;
	using Ctx = StepCtxF;
	static __device__ __forceinline__ void fresh(const RunParams& R, const DevPoint* __restrict__ P, MixedLane& L) { fresh_state(R.S, P, L); }
	static __device__ __forceinline__ bool fits(const MixedLane& L) { return L.hot().pr.radial_mode == 0; }

	static __device__ __forceinline__ void propagate(const RunParams& R, const Box& b, const TeamState& s, TeamState& n)
	{
		PropF q = team_prop(b, s);
		const double r = prop_radius_f(q);
		double step = sanitized_step(s.step);
		bool ok = true;
		if(r >= DMS_RSUN_KM)
		{
			const EventF before = prop_event_f(q);
			step = capped_step(r, s.speed, step, R.boundary);
			if(!surface_is_far(r, static_cast<double>(dotf(before.x, before.v)), step))
				step = surface_step(before, r, step);
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
			rk = rk45_attempt_f<true>(tables_f(R), q, inner);
		}
		const double r_after = prop_radius_f(q);
		n.speed = prop_speed_f(q);
		ok &= (rk == RK_ACCEPTED) & (r_after < INFINITY) & (n.speed < INFINITY);
		n.rate = ok && r_after < DMS_RSUN_KM ? static_cast<double>(rate_total_f(R.S, b.P, grid_f(b.P), static_cast<float>(r_after), static_cast<float>(n.speed))) : 0.0;
		n.time = q.time;
		n.radius = q.radius;
		n.phi = q.phi;
		n.v_radial = q.v_radial;
		n.step = q.time_step;
		n.inner = inner;
		n.ok = ok ? 1 : 0;
	}

	static __device__ __forceinline__ int judge(const RunParams& R, const Box& b, TeamState& s, const EventF& e, const TeamState& n, EventF& en, MixedLane& L,
	                                            bool mine, double* buffer, StepCtxF& c)
	{
		const int capture_mode = R.capture_mode;
		const int pieces = capture_mode ? DMS_CAPTURE_OPTICAL_DEPTH_PIECES : DMS_MAX_OPTICAL_DEPTH_PIECES;
		const double tau_limit = capture_mode ? DMS_CAPTURE_MAX_OPTICAL_DEPTH_STEP : DMS_MAX_OPTICAL_DEPTH_STEP;
		bool interior = false, depth = false, stop = true;
		if(mine && n.ok)
		{
			const PropF q = team_prop(b, n);
			c.before = &e;
			c.r_before = s.radius < 0.0 ? 0.0 : s.radius;
			c.dt = n.time - s.time;
			c.r_after = prop_radius_f(q);
			c.v_after = n.speed;
			c.after = prop_event_f(q);
			stop = !((c.dt > 0.0) & (c.dt < INFINITY) & (c.v_after <= DMS_V_MAX_C * DMS_C_KMS) & (L.hot().seg_steps + 4 < R.max_free_steps));
			if(!stop)
			{
				c.s0 = 0.0f;
				c.s1 = 1.0f;
				interior = true;
				if(!(c.r_before < DMS_RSUN_KM && c.r_after < DMS_RSUN_KM))
				{
					c.s1 = 0.0f;
					interior = false;
					if(!chord_stays_outside(*c.before, c.after, c.r_before, c.r_after))
						interior = interior_interval_outside(*c.before, c.after, c.r_before, c.r_after, c.s0, c.s1);
				}
				depth = interior && c.s1 > c.s0;
			}
		}
		const unsigned int dm = __ballot_sync(0xffffffffu, depth);
		DepthF d = {0.0f, 0.0f, 0.0f, false};
		if(dm != 0u)
			warp_depth(R, b.P, c, static_cast<float>(s.rate), c.r_before < DMS_RSUN_KM && c.s0 <= 1.0e-12f, pieces, dm, depth,
			           reinterpret_cast<float*>(buffer), d);
		int verdict = VERDICT_STOP;
		const double dtau = static_cast<double>(d.dtau);
		if(mine && !stop && !d.invalid && (dtau >= 0.0) & (dtau < INFINITY))
		{
			verdict = interior & (dtau >= L.hot().tau) ? VERDICT_SCATTER : VERDICT_PLAIN;
			const float scale = d.dtau > static_cast<float>(DMS_OPTICAL_DEPTH_ABS_TOL) ? d.dtau : static_cast<float>(DMS_OPTICAL_DEPTH_ABS_TOL);
			if(interior && ((dtau > tau_limit) | (!capture_mode & (fabsf(d.dtau - d.tau2) > static_cast<float>(DMS_OPTICAL_DEPTH_REL_TOL * 0.999) * scale))))
			{
				// (a rejection comes before the scattering test; the last retry ends the trajectory)
				if(L.hot().retries >= DMS_MAX_OPTICAL_DEPTH_RETRIES)
					verdict = VERDICT_STOP;
				else if(depth_reject(L, *c.before, d.dtau, d.tau2, capture_mode != 0, c.dt, tau_limit) == PH_STEP)
					verdict = VERDICT_RESTART;
			}
			if(verdict == VERDICT_PLAIN && c.r_after >= R.boundary)
				verdict = VERDICT_BOUNDARY;
			if(verdict == VERDICT_PLAIN && !L.hot().is_captured)
			{
				// the energy that commit_event_mixed forms, or that of not_free
				const double E = capture_mode ? NAN : capture_energy_eV_f(tables_f(R), b.m_dm, normf(c.after.x), normf(c.after.v));
				if(isnan(E) ? not_free(R, b.m_dm, c.after) : !(isfinite(E) && E >= 0.0))
					verdict = VERDICT_STOP;
			}
			if(verdict != VERDICT_STOP)
				L.hot().attempts += static_cast<uint64_t>(n.inner);
			if(verdict == VERDICT_RESTART)
				s.step = L.hot().pr.time_step;
			if(interior && (verdict == VERDICT_PLAIN || verdict == VERDICT_BOUNDARY))
				L.hot().tau -= dtau;
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

	static __device__ __forceinline__ void commit(const RunParams& R, const Box& b, MixedLane& L, const EventF& e) { commit_event_mixed(R, b.m_dm, L, b.hist, e); }

	// The end of a step that reaches the boundary or a scattering, as in mixed_step: `phase` is the lane's next.
	static __device__ __forceinline__ void finish(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, MixedLane& L, double2* hist, StepCtxF& c,
	                                              const TeamState& n, bool scattering, int& phase)
	{
		int boundary = BOUNDARY_INSIDE;
		if(!scattering)
			boundary = boundary_step(R, m_dm, L, hist, c);
		else
		{
			const bool depth = c.s1 > c.s0;
			scatter_point(R.S, P, c, static_cast<float>(L.hot().next_rate), depth && c.r_before < DMS_RSUN_KM && c.s0 <= 1.0e-12f, depth,
			              R.capture_mode ? DMS_CAPTURE_OPTICAL_DEPTH_PIECES : DMS_MAX_OPTICAL_DEPTH_PIECES, L.hot().tau, c.after);
		}
		if(boundary == BOUNDARY_FAILURE)
			phase = PH_FINAL;
		else if(boundary != BOUNDARY_RETURN)
			phase = finish_step(R, m_dm, L, hist, c, scattering, boundary, n.time, n.radius, n.phi, n.v_radial, n.step, n.rate, true);
	}
};

template <int THREADS>
struct MixedStep : Team<MixedTeam>
{
	static constexpr int threads = THREADS;
	static constexpr bool throughput = THREADS > LATENCY_THREADS;
	// (in the latency form the barriers cost more than the fetches: 16 384 Capture-mode trajectories 2.8 / 3.0 ms)
	static constexpr bool lockstep = throughput;
	static constexpr int buffer = COOP_BUFFER_F;
	static constexpr bool team = !throughput;
	__device__ __forceinline__ int operator()(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, MixedLane& L, double2* hist, int phase,
	                                          double* buffer) const
	{
		return mixed_step<!throughput>(R, P, m_dm, L, hist, phase, reinterpret_cast<float*>(buffer));
	}
	__device__ __forceinline__ double channel(const DevSolar& S, const DevPoint* __restrict__ P, int i, double dr, double T, double v, int k) const
	{
		return channel_rate_f(S, P, i, dr, T, v, k);
	}
	__device__ __forceinline__ bool scatter(const DevSolar& S, const DevPoint* __restrict__ P, Draws& D, Event& e, int target) const
	{
		return scatter_with_target_f(S, P, D, e, target);
	}
};

// The throughput and the latency form, as in dms_kernels.cu.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) trajectory_kernel_mixed(const RunParams R)
{
	lane_loop<MixedLane>(R, MixedStep<THREADS>());
}

__global__ void __launch_bounds__(LATENCY_THREADS, 1) trajectory_kernel_mixed_latency(const RunParams R)
{
	lane_loop<MixedLane>(R, MixedStep<LATENCY_THREADS>());
}

__global__ void grid_to_float_kernel(const double* __restrict__ in, float* __restrict__ out, size_t n)
{
	for(size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < n; k += static_cast<size_t>(gridDim.x) * blockDim.x)
		out[k] = static_cast<float>(in[k]);
}

}	// namespace

void Launch_Trajectories_Mixed(const RunParams& p, int blocks, int threads, cudaStream_t stream)
{
	const auto kernel = threads <= LATENCY_THREADS ? trajectory_kernel_mixed_latency
	                    : threads <= MAX_THREADS   ? trajectory_kernel_mixed<MAX_THREADS>
	                                               : trajectory_kernel_mixed<MAX_THREADS_MIXED>;
	Launch_With_Hot_States<MixedLane>(kernel, p, blocks, threads, stream);
}

void Launch_To_Float(const double* in, float* out, size_t n, cudaStream_t stream)
{
	grid_to_float_kernel<<<148 * 4, 256, 0, stream>>>(in, out, n);
}

#ifdef DMS_CHECKED
bool Take_Form_Counts_Mixed(unsigned long long* counts)
{
	const unsigned long long zero[FORM_COUNTS] = {};
	return cudaMemcpyFromSymbol(counts, dms_form_counts, sizeof zero) == cudaSuccess &&
	       cudaMemcpyToSymbol(dms_form_counts, zero, sizeof zero) == cudaSuccess && cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess;
}
#endif

unsigned int Take_Bounds_Status_Mixed()
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
