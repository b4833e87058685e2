// Lane state machine shared by the FP64 and the mixed-precision trajectory kernels: lane state,
// work claims, trajectory start, free-segment start, capture bookkeeping, termination and
// aggregation.  The free step itself (the Propagate_Freely loop body) is supplied by each form.
#pragma once

#include <type_traits>

#include "dms_kernels.cuh"
#include "dms_lane_rules.h"

namespace dms
{
namespace lane
{

enum Phase : int
{
	PH_FETCH = 0,
	PH_SEGMENT = 1,
	PH_STEP = 2,
	PH_FINAL = 3,
	PH_DONE = 4,
	PH_SCATTER = 5,  // the committed event L.cur is a scattering point inside the Sun
};


// The part of a lane's state that every pass reads and writes.  It lies in shared memory (127 KB of a full FP64
// block): the states of a block's lanes are larger than its L1 cache, and in local memory more than half of
// their reads went to L2, the longest of the kernel's waits.  An odd number of 8-byte words keeps the lanes
// of a warp on different banks.  Together with the calls written out in the pass (dms_kernels.cu), 2^20
// Capture-mode trajectories take 40.9 -> 36.5 ms in FP64 and 25.3 -> 23.5 ms in the mixed form, the steady state
// of Parameter-point mode 855 -> 932 and 1 305 -> 1 407 Msteps/s; with the bincount and drift fields here too
// (160 KB) the tables lose their place in L1: 39.1 against 38.5 ms.
template <class PropT, class EvT>
struct HotFields
{
	PropT pr;            // propagator of the current free segment (local time)
	EvT before;          // Event_In_3D of the propagator at the start of the step (cached)
	double origin;       // absolute time of the segment's local t = 0
	double tau;          // remaining optical depth to the next scattering (minus_log_xi)
	double rate_before;  // scattering rate at the start of the step
	double next_speed, next_rate;
	uint64_t seg_steps;
	uint64_t steps;      // accepted free steps of the whole trajectory (work counter)
	uint64_t attempts;   // RK45 attempts of the whole trajectory (work counter)
	unsigned int retries;
	int before_valid;
	int in_rk;           // an RK45 step is in progress (retry pending)
	int rk_inner;        // passes of the current RK45 step
	int next_valid;      // next_speed / next_rate hold the propagator's speed and rate
	int is_captured;
};
template <class PropT, class EvT, bool EVEN = sizeof(HotFields<PropT, EvT>) / 8 % 2 == 0>
struct HotState : HotFields<PropT, EvT>
{
};
template <class PropT, class EvT>
struct HotState<PropT, EvT, true> : HotFields<PropT, EvT>
{
	double unused;
};
extern __shared__ double lane_hot_states[];

// Trajectory state of a lane (TrajectoryBincount + Trajectory_Simulator members,
// include/Simulation_Trajectory.hpp:53-154).
template <class PropT, class EvT>
struct LaneT
{
	// the FP64 form bins by the reference's division; the mixed form multiplies by the
	// reciprocal bin width (a bin edge can then move by one ulp)
	static constexpr bool exact_bins = std::is_same<PropT, Prop>::value;
	using Hot = HotState<PropT, EvT>;
	static_assert(sizeof(Hot) / 8 % 2 == 1, "lanes on different banks");
	static __device__ __forceinline__ Hot& hot() { return reinterpret_cast<Hot*>(lane_hot_states)[threadIdx.x]; }
	uint64_t work;
	int point;
	Draws D;
	Event cur;           // absolute event at segment boundaries and at termination
	uint64_t nscat;
	int shift_ok;
	int reason;
	// capture / evaporation state
	int bound_state;
	double t_capture, t_last_bound, t_final_unbinding;
	double free_flight_E;
	double max_drift_eV, max_drift_rel;
	// bincount anchor (left-endpoint rule)
	double prev_time, prev_r, prev_v2;
	int bmin, bmax;
	// the bin being visited, held in registers until the trajectory leaves it
	int cbin;
	double2 cval;
	uint64_t wall_start;  // %globaltimer at the start of the trajectory (wall-clock limit only)
};
// Nanoseconds of the device's global timer, one clock for every SM.
__device__ __forceinline__ uint64_t global_timer_ns()
{
	uint64_t t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}

// abort_if_wall_time_exceeded, src/Simulation_Trajectory.cpp:824-840: the trajectory's wall time
// since it started on its lane against max_trajectory_wall_time_sec (0 = no limit)
template <class Lane>
__device__ __forceinline__ bool wall_time_exceeded(const RunParams& R, const Lane& L)
{
	return R.wall_limit_ns != 0 && global_timer_ns() - L.wall_start > R.wall_limit_ns;
}

template <class Lane>
__device__ __forceinline__ void accumulate_bincount(Lane& L, double2* hist, double r, double v2, double dt)
{
	// Accumulate_Bincount_Step, src/Simulation_Trajectory.cpp:640-669
	if(!isfinite(dt) || dt <= 0.0)
		return;
	int bin = -1;
	if(isfinite(r) && r >= 0.0 && r < DMS_BIN_MAX_KM)
	{
		if constexpr(Lane::exact_bins)
		{
			double whole;
			bin = static_cast<int>(fast::floor_index(fast::div_const(r, DMS_BIN_WIDTH_KM), whole));
		}
		else
			bin = static_cast<int>(r * (1.0 / DMS_BIN_WIDTH_KM));
		if(bin < 0) bin = 0;
		if(bin >= DMS_NUM_BINS) bin = -1;
	}
	if(bin >= 0)
	{
		DMS_CHECK_INDEX(bin, 0, DMS_NUM_BINS, BOUNDS_BIN);
		// The row is read only when a visited bin is entered again and written when it is
		// left; the additions are the reference's, in its order.
		if(bin != L.cbin)
		{
			if(L.cbin >= 0)
				hist[L.cbin] = L.cval;
			L.cval = (bin >= L.bmin && bin <= L.bmax) ? hist[bin] : make_double2(0.0, 0.0);
			L.cbin = bin;
			L.bmin = bin < L.bmin ? bin : L.bmin;
			L.bmax = bin > L.bmax ? bin : L.bmax;
		}
		L.cval.x += dt;
		L.cval.y += v2 * dt;
	}
}

// Writes the bin being visited back to the lane's row (before the row is read out).
template <class Lane>
__device__ __forceinline__ void write_back_bin(Lane& L, double2* hist)
{
	if(L.cbin >= 0)
		hist[L.cbin] = L.cval;
	L.cbin = -1;
}

// Update_Capture_State, src/Simulation_Trajectory.cpp:689-760
template <class Lane>
__device__ __forceinline__ bool update_capture_state(const DevSolar& S, double m_dm, int capture_mode, Lane& L, double r, double v, double t, bool allow_new)
{
	if(capture_mode && !allow_new && !L.hot().is_captured)
		return false;
	const double E = capture_energy_eV(S, m_dm, r, v);
	const bool negative = E < 0.0;
	if(!allow_new)
	{
		if(L.hot().is_captured && isfinite(L.free_flight_E))
		{
			const double drift = fabs(E - L.free_flight_E);
			if(isfinite(drift) && drift > L.max_drift_eV)
				L.max_drift_eV = drift;
			const double ref = fabs(L.free_flight_E);
			const double scale = ref > DMS_FREE_ENERGY_DRIFT_REL_E_SCALE_EV ? ref : DMS_FREE_ENERGY_DRIFT_REL_E_SCALE_EV;
			const double rel = drift / scale;
			if(isfinite(rel) && rel > L.max_drift_rel)
				L.max_drift_rel = rel;
		}
		if(L.bound_state && L.hot().is_captured)
			L.t_last_bound = t;
		return false;
	}
	const int was_bound = L.bound_state;
	L.bound_state = negative;
	L.free_flight_E = E;
	if(negative)
	{
		if(!L.hot().is_captured)
		{
			L.hot().is_captured = 1;
			L.t_capture = t;
			L.t_last_bound = t;
		}
		else if(!was_bound)
			L.t_final_unbinding = NAN;
		L.t_last_bound = t;
		return true;
	}
	if(was_bound && L.hot().is_captured)
		L.t_final_unbinding = t;
	return false;
}

template <class Lane>
__device__ __forceinline__ bool uncaptured_bound(const DevSolar& S, double m_dm, const Lane& L, const Event& e)
{
	if(L.hot().is_captured)
		return false;
	const double E = capture_energy_eV(S, m_dm, ev_radius(e), ev_speed(e));
	if(isfinite(E) && E >= 0.0)
		return false;
	return true;
}

template <class Lane>
__device__ __forceinline__ void set_final(Lane& L, const Event& local_or_abs, bool is_local, int reason)
{
	L.cur = local_or_abs;
	if(is_local)
		L.cur.t += L.hot().origin;
	L.reason = reason;
}

__device__ __forceinline__ void init_propagator(Prop& p, const Event& e) { prop_init(p, e); }

// Start of a free segment: Simulate loop head + Propagate_Freely prologue,
// src/Simulation_Trajectory.cpp:1311-1313, 762-805
template <class Lane>
__device__ __forceinline__ int segment_start(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, Lane& L)
{
	if(!(L.nscat < R.max_scatterings))
	{
		L.reason = DMS_REASON_MAX_SCATTERINGS;
		return PH_FINAL;
	}
	if(outward_escaping(R.S, L.cur, R.boundary))
	{
		L.reason = DMS_REASON_OUTWARD_ESCAPE;
		return PH_FINAL;
	}
	if(uncaptured_bound(R.S, m_dm, L, L.cur))
	{
		L.reason = DMS_REASON_NUMERICAL_FAILURE;
		return PH_FINAL;
	}
	L.hot().origin = L.cur.t;
	Event local = L.cur;
	local.t = 0.0;
	init_propagator(L.hot().pr, local);
	L.hot().tau = -log_call(draw_positive(L.D));
	L.hot().seg_steps = 0;
	L.hot().retries = 0;
	L.hot().before_valid = 0;
	L.hot().next_valid = 0;
	L.hot().in_rk = 0;
	if(!R.capture_mode && L.prev_time >= 0.0)
		L.prev_time = 0.0;
	return PH_STEP;
}

__device__ __forceinline__ bool is_numerical_termination(int r)
{
	return r == DMS_REASON_NUMERICAL_FAILURE || r == DMS_REASON_NON_FINITE_STATE || r == DMS_REASON_SPEED_LIMIT ||
	       r == DMS_REASON_ENERGY_DRIFT_ESCAPE || r == DMS_REASON_UNKNOWN;
}

__device__ __forceinline__ bool is_computational_truncation(int r)
{
	return r == DMS_REASON_WALL_TIME_LIMIT || r == DMS_REASON_MAX_FREE_STEPS || r == DMS_REASON_MAX_SCATTERINGS;
}

// Termination: tail of Simulate (src/Simulation_Trajectory.cpp:1349-1399), classification and
// aggregation of simulate_one_trajectory (src/Data_Generation.cpp:745-861).
// The lane's histogram row still to be moved out at termination: copied into the record's
// histograms (records mode) or added with its squares to the per-point sums (accumulate mode),
// and zeroed either way.  Executed by the whole warp (cooperative_flush).
struct FlushJob
{
	double* dst0;  // records: dt row; accumulate: sum of dt
	double* dst1;  // records: v2dt row; accumulate: sum of v2dt
	double* dst2;  // accumulate: sum of dt^2
	double* dst3;  // accumulate: sum of v2dt^2
	int b0, b1;    // touched bins; b1 < b0 when there is nothing to do
	int mode;      // FLUSH_ZERO, FLUSH_COPY or FLUSH_ADD
};
constexpr int FLUSH_ZERO = 0, FLUSH_COPY = 1, FLUSH_ADD = 2;

template <class Lane>
__device__ __noinline__ void finalize(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, Lane& L, FlushJob& job)
{
	const DevSolar& S = R.S;
	int reason = L.reason;
	int survival_valid = 1, event_observed = 0, boundary_escape = 0, invalid_escape = 0;
	double t_boundary = NAN;
	const double t_term = L.cur.t;
	uint32_t flags = 0;
	if(L.shift_ok)
	{
		flags |= DMS_REC_SHIFT_OK;
		if(L.hot().is_captured)
		{
			const double r_f = ev_radius(L.cur), v_f = ev_speed(L.cur);
			const double vesc_f = solar_vesc(S, r_f);
			const double E_f = 0.5 * m_dm * ((v_f * v_f - vesc_f * vesc_f) / (DMS_C_KMS * DMS_C_KMS)) / 1.0e-9;
			if(reason == DMS_REASON_OUTWARD_ESCAPE && E_f >= 0.0)
			{
				if(isfinite(L.t_final_unbinding))
				{
					boundary_escape = 1;
					t_boundary = t_term;
					event_observed = 1;
				}
				else
				{
					reason = DMS_REASON_ENERGY_DRIFT_ESCAPE;
					survival_valid = 0;
					invalid_escape = 1;
				}
			}
		}
		switch(reason)
		{
			case DMS_REASON_ENERGY_DRIFT_ESCAPE:
			case DMS_REASON_NUMERICAL_FAILURE:
			case DMS_REASON_NON_FINITE_STATE:
			case DMS_REASON_SPEED_LIMIT:
			case DMS_REASON_WALL_TIME_LIMIT:
			case DMS_REASON_MAX_FREE_STEPS:
			case DMS_REASON_MAX_SCATTERINGS:
			case DMS_REASON_UNKNOWN: survival_valid = 0; break;
			default: break;
		}
		if(L.hot().is_captured && !event_observed)
		{
			L.t_final_unbinding = NAN;
			if(reason != DMS_REASON_CAPTURE_MODE)
				survival_valid = 0;
		}
		if(L.hot().is_captured) flags |= DMS_REC_CAPTURED;
		if(event_observed) flags |= DMS_REC_EVENT_OBSERVED;
		if(survival_valid) flags |= DMS_REC_SURVIVAL_VALID;
		if(boundary_escape) flags |= DMS_REC_BOUNDARY_ESCAPE;
		if(invalid_escape) flags |= DMS_REC_INVALID_ESCAPE;
		if(!L.hot().is_captured && reason == DMS_REASON_OUTWARD_ESCAPE)
		{
			if(L.nscat == 0)
				flags |= DMS_REC_FREE;
			else
			{
				const double rf = ev_radius(L.cur);
				const double vesc = sqrt(2 * DMS_GMSUN_KM3S2 / rf);
				if(rf > DMS_RSUN_KM && ev_speed(L.cur) > vesc)
				{
					flags |= DMS_REC_REFLECTED;
					Event fin = L.cur;
					if(hyperbolic_kepler_shift(fin, DMS_AU_KM))
					{
						flags |= DMS_REC_REFLECT_SHIFT_OK;
						if(R.records == nullptr && R.reflections != nullptr)
						{
							// the reflection-spectrum sample, src/Data_Generation.cpp:829-840
							const double speed = ev_speed(fin);
							const double* vs = P->vel_obs;
							const double sun = sqrt(vs[0] * vs[0] + vs[1] * vs[1] + vs[2] * vs[2]);
							const double cosine = (fin.x.x * vs[0] + fin.x.y * vs[1] + fin.x.z * vs[2]) / ev_radius(fin) / sun;
							const unsigned long long k = atomicAdd(R.reflection_count + L.point, 1ULL);
							if(k < R.event_capacity)
							{
								dms_reflection rf;
								rf.trajectory_id = L.D.traj + 1;
								rf.speed_kms = speed;
								rf.cos_sun_velocity = cosine;
								R.reflections[static_cast<size_t>(L.point) * R.event_capacity + k] = rf;
							}
							else
								atomicAdd(R.counters + static_cast<size_t>(L.point) * DMS_NUM_COUNTERS + DMS_CNT_REFLECTIONS_DROPPED, 1ULL);
						}
					}
				}
			}
		}
	}
	else
	{
		reason = DMS_REASON_NUMERICAL_FAILURE;
		survival_valid = 0;
	}
	const bool invalid = invalid_escape || reason == DMS_REASON_ENERGY_DRIFT_ESCAPE;
	const bool valid = survival_valid && !invalid;
	const bool observed = valid && event_observed;
	const double life = observed ? L.t_final_unbinding - L.t_capture : -1.0;
	const double lifetime = (L.hot().is_captured && isfinite(life) && life >= 0.0) ? life : -1.0;

	job.b0 = L.bmin;
	job.b1 = L.bmax;
	job.mode = FLUSH_ZERO;
	if(R.records != nullptr)
	{
		dms_traj_record& rec = R.records[L.work - 0];
		rec.number_of_scatterings = L.nscat;
		rec.number_of_draws = L.D.index;
		rec.termination_reason = static_cast<uint32_t>(reason);
		rec.flags = flags;
		rec.final_time = L.cur.t;
		rec.final_position[0] = L.cur.x.x;
		rec.final_position[1] = L.cur.x.y;
		rec.final_position[2] = L.cur.x.z;
		rec.final_velocity[0] = L.cur.v.x;
		rec.final_velocity[1] = L.cur.v.y;
		rec.final_velocity[2] = L.cur.v.z;
		rec.t_capture = L.shift_ok ? L.t_capture : -1.0;
		rec.t_last_bound = L.shift_ok ? L.t_last_bound : -1.0;
		rec.t_final_unbinding_scatter = L.shift_ok ? L.t_final_unbinding : NAN;
		rec.t_boundary_escape = t_boundary;
		rec.t_termination = L.shift_ok ? t_term : -1.0;
		rec.max_free_energy_drift_eV = L.max_drift_eV;
		rec.max_free_energy_drift_rel = L.max_drift_rel;
		rec.lifetime_unbinding = lifetime;
		if(R.rec_hist_dt != nullptr)
		{
			job.mode = FLUSH_COPY;
			job.dst0 = R.rec_hist_dt + L.work * DMS_NUM_BINS;
			job.dst1 = R.rec_hist_v2dt + L.work * DMS_NUM_BINS;
		}
	}
	else
	{
		unsigned long long* c = R.counters + static_cast<size_t>(L.point) * DMS_NUM_COUNTERS;
		atomicAdd(c + DMS_CNT_TRAJECTORIES, 1ULL);
		atomicAdd(c + DMS_CNT_TOTAL_SCATTERINGS, static_cast<unsigned long long>(L.nscat));
		atomicAdd(c + DMS_CNT_RK_STEPS, static_cast<unsigned long long>(L.hot().steps));
		atomicAdd(c + DMS_CNT_RK_ATTEMPTS, static_cast<unsigned long long>(L.hot().attempts));
		atomicAdd(c + DMS_CNT_REASON_BASE + reason, 1ULL);
		if(!L.shift_ok)
		{
			atomicAdd(c + DMS_CNT_INITIAL_SHIFT_FAILURES, 1ULL);
			atomicAdd(c + DMS_CNT_NUMERICAL_FAILURES, 1ULL);
		}
		else if(is_numerical_termination(reason))
			atomicAdd(c + DMS_CNT_NUMERICAL_FAILURES, 1ULL);
		if(is_computational_truncation(reason))
			atomicAdd(c + DMS_CNT_COMPUTATIONAL_TRUNCATIONS, 1ULL);
		int hist_slot = -1;
		if(L.hot().is_captured)
		{
			atomicAdd(c + DMS_CNT_CAPTURED, 1ULL);
			if(!R.capture_mode)
			{
				atomicAdd(c + (event_observed ? DMS_CNT_COMPLETE_EVAPORATION : DMS_CNT_INVALID_SURVIVAL), 1ULL);
				hist_slot = 0;
				if(lifetime >= 0.0)
				{
					const unsigned long long k = atomicAdd(R.event_count + L.point, 1ULL);
					if(k < R.event_capacity)
					{
						// the lifetime is made visible before the id: a reader of a run in flight
						// takes a slot whose id is still 0 (ids start at 1) as not yet published
						dms_evaporation_event& ev = R.events[static_cast<size_t>(L.point) * R.event_capacity + k];
						ev.lifetime_unbinding = lifetime;
						__threadfence();
						*reinterpret_cast<volatile uint64_t*>(&ev.trajectory_id) = L.D.traj + 1;
					}
					else
						atomicAdd(c + DMS_CNT_EVENTS_DROPPED, 1ULL);
				}
			}
		}
		else if(reason == DMS_REASON_OUTWARD_ESCAPE)
		{
			atomicAdd(c + DMS_CNT_COMPLETED_OUTWARD, 1ULL);
			if(!R.capture_mode)
			{
				hist_slot = 2;
				if(flags & DMS_REC_FREE)
					atomicAdd(c + DMS_CNT_FREE, 1ULL);
				else if(flags & DMS_REC_REFLECTED)
				{
					atomicAdd(c + DMS_CNT_REFLECTED, 1ULL);
					if(!(flags & DMS_REC_REFLECT_SHIFT_OK))
					{
						atomicAdd(c + DMS_CNT_FINAL_REFLECTION_SHIFT_FAILURES, 1ULL);
						atomicAdd(c + DMS_CNT_NUMERICAL_FAILURES, 1ULL);
					}
				}
			}
		}
		if(hist_slot >= 0)
		{
			double* h = R.hists + static_cast<size_t>(L.point) * DMS_NUM_HISTS * DMS_NUM_BINS;
			job.mode = FLUSH_ADD;
			job.dst0 = h + (hist_slot + 0) * DMS_NUM_BINS;
			job.dst1 = h + (hist_slot + 1) * DMS_NUM_BINS;
			job.dst2 = h + (hist_slot + 4) * DMS_NUM_BINS;
			job.dst3 = h + (hist_slot + 5) * DMS_NUM_BINS;
		}
	}
}

// Moves the histogram rows of every lane of the group `grp` (the whole warp) that terminated in
// this iteration: all lanes of the group stride over one row at a time, so the row is read, the
// per-point sums are updated and the row is zeroed with coalesced accesses instead of one
// lane walking up to 2000 bins while the rest of its warp waits.
__device__ __forceinline__ void cooperative_flush(double2* hist, FlushJob& job, unsigned int grp)
{
	unsigned int pending = __ballot_sync(grp, job.b1 >= job.b0);
	if(pending == 0u)
		return;
	const int me = threadIdx.x & 31;
	const int rank = __popc(grp & ((1u << me) - 1u));
	const int size = __popc(grp);
	__syncwarp(grp);  // each owner's last write to its row is visible to the group
	while(pending != 0u)
	{
		const int leader = __ffs(pending) - 1;
		pending &= pending - 1u;
		double2* row = reinterpret_cast<double2*>(__shfl_sync(grp, reinterpret_cast<unsigned long long>(hist), leader));
		int b0 = __shfl_sync(grp, job.b0, leader);
		int b1 = __shfl_sync(grp, job.b1, leader);
		DMS_CHECK_INDEX(b0, 0, DMS_NUM_BINS, BOUNDS_ROW);
		DMS_CHECK_INDEX(b1, 0, DMS_NUM_BINS, BOUNDS_ROW);
		const int mode = __shfl_sync(grp, job.mode, leader);
		double* d0 = reinterpret_cast<double*>(__shfl_sync(grp, reinterpret_cast<unsigned long long>(job.dst0), leader));
		double* d1 = reinterpret_cast<double*>(__shfl_sync(grp, reinterpret_cast<unsigned long long>(job.dst1), leader));
		double* d2 = reinterpret_cast<double*>(__shfl_sync(grp, reinterpret_cast<unsigned long long>(job.dst2), leader));
		double* d3 = reinterpret_cast<double*>(__shfl_sync(grp, reinterpret_cast<unsigned long long>(job.dst3), leader));
		for(int b = b0 + rank; b <= b1; b += size)
		{
			const double2 x = row[b];
			if(mode == FLUSH_COPY)
			{
				d0[b] = x.x;
				d1[b] = x.y;
			}
			else if(mode == FLUSH_ADD && (x.x != 0.0 || x.y != 0.0))
			{
				atomicAdd(d0 + b, x.x);
				atomicAdd(d1 + b, x.y);
				atomicAdd(d2 + b, x.x * x.x);
				atomicAdd(d3 + b, x.y * x.y);
			}
			row[b] = make_double2(0.0, 0.0);
		}
	}
	__syncwarp(grp);  // the zeroed rows are visible to their owners before they are reused
	job.b1 = -1;
}

// Picks up work index `w`: the Simulate prologue (src/Simulation_Trajectory.cpp:1284-1308) from
// the initial state (Initial_Conditions + Hyperbolic_Kepler_Shift, src/Data_Generation.cpp:747-761)
// that initial_state_kernel computed for every work index before the launch.
template <class Lane>
__device__ __forceinline__ int start_trajectory(const RunParams& R, Lane& L, uint64_t w, const DevPoint*& P, double& m_dm)
{
	int k = find_range(R, w);
	DMS_CHECK_INDEX(k, 0, R.n_ranges, BOUNDS_RANGE);
	L.work = w;
	L.point = R.range_point[k];
	P = R.points + L.point;
	m_dm = __ldg(&P->m_dm);
	L.D.seed = R.seed;
	L.D.point = static_cast<uint32_t>(L.point);
	L.D.traj = R.range_first[k] + (w - R.range_offset[k]);
	L.D.index = 0;
	L.nscat = 0;
	L.hot().steps = 0;
	L.hot().attempts = 0;
	L.wall_start = R.wall_limit_ns != 0 ? global_timer_ns() : 0;
	L.hot().is_captured = 0;
	L.bound_state = 0;
	L.t_capture = -1.0;
	L.t_last_bound = -1.0;
	L.t_final_unbinding = NAN;
	L.free_flight_E = NAN;
	L.max_drift_eV = 0.0;
	L.max_drift_rel = 0.0;
	L.prev_time = -1.0;
	L.prev_r = 0.0;
	L.prev_v2 = 0.0;
	L.bmin = DMS_NUM_BINS;
	L.bmax = -1;
	L.cbin = -1;
	L.reason = DMS_REASON_UNKNOWN;
	const InitState& init = R.init[w];
	const Event ic = init.ic;
	L.D.index = init.draws;
	L.shift_ok = (init.flags & INIT_SHIFT_OK) != 0u;
	L.cur = ic;
	if(R.records != nullptr)
	{
		dms_traj_record& rec = R.records[w];
		rec.trajectory_id = L.D.traj;
		rec.point = static_cast<uint32_t>(L.point);
		rec.reserved = 0;
		rec.initial_time = ic.t;
		rec.initial_position[0] = ic.x.x;
		rec.initial_position[1] = ic.x.y;
		rec.initial_position[2] = ic.x.z;
		rec.initial_velocity[0] = ic.v.x;
		rec.initial_velocity[1] = ic.v.y;
		rec.initial_velocity[2] = ic.v.z;
	}
	if(!L.shift_ok)
	{
		L.reason = DMS_REASON_NUMERICAL_FAILURE;
		return PH_FINAL;
	}
	return PH_SEGMENT;
}

// Sample_Target for every lane of the group `grp` (the whole warp) at a scattering point.  The 64
// channel rates of one scattering lane (63 isotopes + electrons, the dominant cost of a
// scatter) are evaluated by all lanes of the group in parallel into shared memory; the
// scattering lane then validates, sums and picks sequentially in the reference's order, so
// the target and the draws consumed are those of the one-lane form.  `rates` is this warp's
// DMS_NUM_TARGETS + 1 doubles of shared memory.
template <class Lane, class Step>
__device__ __forceinline__ void cooperative_targets(const RunParams& R, Lane& L, int phase, double* rates, int& target, const Step& step,
                                                    unsigned int grp)
{
	unsigned int pending = __ballot_sync(grp, phase == PH_SCATTER);
	if(pending == 0u)
		return;
	const int me = threadIdx.x & 31;
	const int rank = __popc(grp & ((1u << me) - 1u));
	const int size = __popc(grp);
	const bool mine = phase == PH_SCATTER;
	const double my_r = mine ? ev_radius(L.cur) : 0.0;
	const double my_v = mine ? ev_speed(L.cur) : 0.0;
	while(pending != 0u)
	{
		const int leader = __ffs(pending) - 1;
		pending &= pending - 1u;
		const double r = __shfl_sync(grp, my_r, leader);
		const double v = __shfl_sync(grp, my_v, leader);
		const int point = __shfl_sync(grp, L.point, leader);
		bool bad = !(isfinite(r) && isfinite(v));
		if(!bad)
		{
			const DevPoint* P = R.points + point;
			const int i = knot_index(R.S, r);
			const double dr = r - __ldg(R.S.r + i);
			const double T = __ldg(R.S.temp + i) + dr * __ldg(R.S.temp_s + i);
			for(int k = rank; k <= DMS_NUM_TARGETS; k += size)
			{
				const double x = step.channel(R.S, P, i, dr, T, v, k);
				bad = bad || !(isfinite(x) && x >= 0.0);
				rates[k] = x;
			}
		}
		// validation: every channel finite and >= 0 (the reference throws otherwise)
		bad = __any_sync(grp, bad);
		__syncwarp(grp);
		double total = 0.0;
		if(me == leader && !bad)
			total = channel_total(rates);
		total = __shfl_sync(grp, total, leader);
		const bool ok = !bad && isfinite(total) && total > 0.0;
		// the 64 divisions by the total, in parallel: each lane replaces its channels by
		// their fractions, exactly the quotients the sequential pick forms
		if(ok)
			for(int k = rank; k <= DMS_NUM_TARGETS; k += size) rates[k] = rates[k] / total;
		__syncwarp(grp);
		if(me == leader)
			target = ok ? pick_from_fractions(L.D, rates) : TARGET_FAILED;
		__syncwarp(grp);
	}
}

// Simulate after a scattering point (src/Simulation_Trajectory.cpp:1313-1346): target
// velocity, angle and kinematics, then capture bookkeeping and the bincount anchor.
template <class Lane, class Step>
__device__ __forceinline__ int finish_scatter(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, Lane& L, int target, const Step& step)
{
	if(target != TARGET_FAILED)
		DMS_CHECK_INDEX(target, -1, DMS_NUM_TARGETS, BOUNDS_TARGET);
	if(target == TARGET_FAILED || !step.scatter(R.S, P, L.D, L.cur, target))
	{
		L.reason = DMS_REASON_NUMERICAL_FAILURE;
		return PH_FINAL;
	}
	L.nscat++;
	const double r = ev_radius(L.cur), v = ev_speed(L.cur);
	const bool captured = update_capture_state(R.S, m_dm, R.capture_mode, L, r, v, L.cur.t, true);
	if(!R.capture_mode)
	{
		// Reset_Bincount_Anchor, src/Simulation_Trajectory.cpp:671-680
		L.prev_time = L.cur.t;
		L.prev_r = r;
		L.prev_v2 = v * v;
	}
	if(R.capture_mode && captured)
	{
		L.reason = DMS_REASON_CAPTURE_MODE;
		return PH_FINAL;
	}
	return PH_SEGMENT;
}


// A trajectory in flight, handed from a throughput launch to the latency launch behind it.
template <class Lane>
struct Parked
{
	Lane L;
	typename Lane::Hot hot;
	double2* hist;          // its histogram row
	uint64_t q_next, q_end; // its lane's claimed ids
	uint64_t iter;
	int phase;
};

template <class Lane, class Step>
__device__ __forceinline__ void lane_loop(const RunParams& R, Step step)
{
	// R.lanes_per_block lanes of the block take trajectories and own a histogram row, dealt out to the warps
	// one by one; the others only help in the collective steps
	const int in_warp = threadIdx.x & 31;
	const int slot = in_warp * (blockDim.x >> 5) + (threadIdx.x >> 5);
	const bool takes_work = slot < R.lanes_per_block;
	double2* hist = R.lane_hist + (static_cast<size_t>(blockIdx.x) * R.lanes_per_block + (takes_work ? slot : 0)) * DMS_NUM_BINS;
	// per warp: the 64 channel rates of a scattering, or the steps and rates of Step's own lookups
	constexpr int BUFFER = Step::buffer > DMS_NUM_TARGETS + 1 ? Step::buffer : DMS_NUM_TARGETS + 1;
	__shared__ double coop_rates[Step::threads / 32][BUFFER];
	double* rates = coop_rates[threadIdx.x >> 5];
	// Lockstep: the warps of a block make every pass together, so that an instruction fetched once serves
	// all of them (until few lanes are left: R.lockstep_min).  The block votes on its rare phases: lanes
	// stepping, at a scattering point and at a termination, counted per pass in the sets of
	// dms_lane_rules.h in turn.
	__shared__ int votes[VOTE_SETS][4];
	if(threadIdx.x < VOTE_SETS * 4)
		votes[threadIdx.x >> 2][threadIdx.x & 3] = 0;
	int vote_set = 0;
	bool lockstep = Step::lockstep;
	bool team = false;  // this warp's lone lane has formed a team
	uint64_t next_check = 1023;
	if constexpr(Step::team)
		if(threadIdx.x == 0)
			step.team_init();
	int scatter_passes = 0, final_passes = 0;  // as rare_phase_due counts them
	__syncthreads();
	Lane L;
	FlushJob job;
	job.b0 = 0;
	job.b1 = -1;
	const DevPoint* P = R.points;
	double m_dm = 0.0;
	int phase = takes_work ? PH_FETCH : PH_DONE;
	uint64_t iter = 0;
	// the lane's claimed ids [q_next, q_end): R.queue_chunk ids per claim
	uint64_t q_next = 0, q_end = 0;
	const unsigned int lane_bit = 1u << (threadIdx.x & 31);
	static_assert(sizeof(Parked<Lane>) <= PARKED_BYTES, "a parked state fits its slot");
	if constexpr(!Step::throughput)
		if(R.resume)
		{
			// the parked trajectories dealt out to the blocks one by one, and to the warps within
			const unsigned int item = static_cast<unsigned int>(slot) * gridDim.x + blockIdx.x;
			phase = PH_DONE;
			if(item < *R.parked_count && item < R.parked_capacity)
			{
				const Parked<Lane>& s = *reinterpret_cast<const Parked<Lane>*>(R.parked + item * PARKED_BYTES);
				L = s.L;
				L.hot() = s.hot;
				hist = s.hist;
				q_next = s.q_next;
				q_end = s.q_end;
				phase = s.phase;
				iter = s.iter;
				P = R.points + L.point;
				m_dm = __ldg(&P->m_dm);
				DMS_COUNT_FORM(FORM_RESUMED, 1);
			}
			// one count per block: the warps in lockstep agree on it
			__shared__ unsigned long long first_iter;
			if(threadIdx.x == 0)
				first_iter = 0;
			__syncthreads();
			atomicMax(&first_iter, static_cast<unsigned long long>(iter));
			__syncthreads();
			iter = first_iter;
			next_check = iter + 1023;
		}
	// Every lane stays in the loop until its whole warp is done (a lane without work waits in
	// PH_DONE), and leaves only together with the others.  So the warp's collective steps
	// below (batching votes, cooperative target sampling into the warp's shared rates, the
	// histogram flush) always run with all 32 lanes, a fixed mask, instead of whichever lanes
	// happen to be converged at that point.
	constexpr unsigned int FULL_WARP = 0xffffffffu;
	bool drained = false;
	for(;; iter++)
	{
		bool go_scatter = false, go_final = false;
		bool alone = !team;  // the lanes make this pass's steps themselves
		if(Step::lockstep && lockstep)
		{
			int* v = votes[vote_set];
			vote_set = next_vote_set(vote_set);
			if(threadIdx.x < 3)
				votes[vote_set][threadIdx.x] = 0;
			const unsigned int b_step = __ballot_sync(FULL_WARP, phase == PH_STEP || phase == PH_FETCH || phase == PH_SEGMENT);
			const unsigned int b_scatter = __ballot_sync(FULL_WARP, phase == PH_SCATTER);
			const unsigned int b_final = __ballot_sync(FULL_WARP, phase == PH_FINAL);
			if(in_warp == 0)
			{
				if(b_step) atomicAdd(v + 0, __popc(b_step));
				if(b_scatter) atomicAdd(v + 1, __popc(b_scatter));
				if(b_final) atomicAdd(v + 2, __popc(b_final));
				// one thread looks whether the queue is empty and whether the host cancelled
				if(threadIdx.x == 0)
				{
					int flags = (iter & 15) == 15 && *reinterpret_cast<volatile unsigned long long*>(R.queue_head) >= R.total ? 1 : 0;
					flags |= (iter & 1023) == 1023 && *R.cancel != 0 ? 2 : 0;
					v[3] = flags;
				}
			}
			__syncthreads();
			const int n_step = v[0], n_scatter = v[1], n_final = v[2], flags = v[3];
			drained |= (flags & 1) != 0;
			// batches and waits are for a full block; in the tail of a throughput launch they shrink with the
			// lanes at work
			const int at_work = n_step + n_scatter + n_final, lanes = blockDim.x;
			const int full = Step::throughput && drained ? at_work : lanes;
			go_scatter = rare_phase_due(scatter_passes, n_scatter, n_step, R.block_scatter_batch, 64, R.scatter_wait, lanes, full);
			go_final = rare_phase_due(final_passes, n_final, n_step, R.block_final_batch, 64, R.final_wait, lanes, full);
			if(flags & 2)
			{
				if(in_warp == 0)
					atomicOr(R.status, STATUS_CANCELLED);
				break;
			}
			if((iter & 1023) == 1023 && iter > R.iteration_budget)
			{
				atomicOr(R.status, STATUS_BUDGET);
				break;
			}
			if(at_work == 0)
				break;
			// few lanes left and no more work: their trajectories go on in the latency launch, or the warps by
			// themselves
			if(drained && at_work <= R.lockstep_min)
			{
				if constexpr(Step::throughput)
				{
					// (at most lockstep_min lanes of a block come here, and the slots are for as many of every
					// block; a lane without one would end the run with an error)
					bool room = true;
					if(phase != PH_DONE && !(phase == PH_FETCH && q_next >= q_end))
					{
						const unsigned int at = atomicAdd(R.parked_count, 1u);
						room = at < R.parked_capacity;
						if(room)
						{
							Parked<Lane>& s = *reinterpret_cast<Parked<Lane>*>(R.parked + at * PARKED_BYTES);
							s.L = L;
							s.hot = L.hot();
							s.hist = hist;
							s.q_next = q_next;
							s.q_end = q_end;
							s.phase = phase;
							s.iter = iter;
							DMS_COUNT_FORM(FORM_PARKED, 1);
						}
						else
							atomicOr(R.status, STATUS_PARKED_FULL);
					}
					phase = room ? PH_DONE : phase;
					break;
				}
				lockstep = false;
			}
		}
		else
		{
			const unsigned int live = __ballot_sync(FULL_WARP, phase != PH_DONE);
			bool leave = live == 0u;
			if(iter >= next_check)
			{
				next_check = iter + 1024;
				if constexpr(Step::team)
					step.team_alive();
				if(__any_sync(FULL_WARP, *R.cancel != 0))
				{
					atomicOr(R.status, STATUS_CANCELLED);
					leave = true;
				}
				if(iter > R.iteration_budget)
				{
					atomicOr(R.status, STATUS_BUDGET);
					leave = true;
				}
			}
			if(leave)
			{
				if constexpr(Step::team)
				{
					if(team)
						step.team_dismiss();
					else if(live != 0u)
						step.team_forgo();
					else if(R.wall_limit_ns == 0 && blockDim.x == 128)
						step.team_help(R, L, rates);
				}
				break;
			}
			if constexpr(Step::team)
			{
				const bool mine = phase == PH_STEP && !L.hot().in_rk;
				alone |= __any_sync(FULL_WARP, phase == PH_STEP && L.hot().in_rk);
				if((live & (live - 1u)) == 0u && __any_sync(FULL_WARP, mine) && R.wall_limit_ns == 0)
				{
					if(!team)
						team = step.team_form();
					if(team)
						alone = step.team_run(R, P, m_dm, L, hist, mine, rates, phase, iter);
				}
			}
			const unsigned int stepping = __ballot_sync(FULL_WARP, phase == PH_STEP || phase == PH_FETCH || phase == PH_SEGMENT);
			const unsigned int waiting = __ballot_sync(FULL_WARP, phase == PH_SCATTER);
			const unsigned int ending = __ballot_sync(FULL_WARP, phase == PH_FINAL);
			// batches and waits are for a full warp and shrink with the lanes at work
			const int at_work = __popc(live);
			go_scatter = rare_phase_due(scatter_passes, __popc(waiting), static_cast<int>(stepping), R.scatter_batch, 32, R.scatter_wait, 32, at_work);
			go_final = rare_phase_due(final_passes, __popc(ending), static_cast<int>(stepping), R.final_batch, 32, R.final_wait, 32, at_work);
		}
		// Scatterings and terminations run for many lanes at once.  A lane's draws do not depend on
		// when it scatters.
		if(go_scatter)
		{
			int target = TARGET_FAILED;
			cooperative_targets(R, L, phase, rates, target, step, FULL_WARP);
			if(phase == PH_SCATTER)
				phase = finish_scatter(R, P, m_dm, L, target, step);
		}
		if(go_final)
		{
			if(phase == PH_FINAL)
			{
				write_back_bin(L, hist);
				finalize(R, P, m_dm, L, job);
				phase = PH_FETCH;
			}
			cooperative_flush(hist, job, FULL_WARP);
		}
		if(phase == PH_FETCH)
		{
			// warp-aggregated claim of R.queue_chunk work indices per lane whose claimed ids
			// are used up
			const unsigned int mask = __activemask();
			const bool need = !(q_next < q_end);
			const unsigned int need_mask = __ballot_sync(mask, need);
			if(need_mask != 0u)
			{
				const int leader = __ffs(need_mask) - 1;
				const unsigned int rank = __popc(need_mask & (lane_bit - 1u));
				unsigned long long base = 0;
				if((threadIdx.x & 31) == leader)
					base = atomicAdd(R.queue_head, static_cast<unsigned long long>(__popc(need_mask)) * R.queue_chunk);
				base = __shfl_sync(mask, base, leader);
				if(need)
				{
					q_next = base + static_cast<uint64_t>(rank) * R.queue_chunk;
					q_end = q_next + R.queue_chunk;
				}
			}
			const uint64_t w = q_next++;
			if(w >= R.total)
				phase = PH_DONE;
			else
				phase = start_trajectory(R, L, w, P, m_dm);
		}
		if(phase == PH_SEGMENT)
			phase = segment_start(R, P, m_dm, L);
		if(alone && __any_sync(FULL_WARP, phase == PH_STEP))
			phase = step(R, P, m_dm, L, hist, phase, rates);
	}
	const bool in_trajectory = phase != PH_FETCH && phase != PH_DONE;
	if(in_trajectory && L.bmax >= L.bmin)
		for(int b = L.bmin; b <= L.bmax; b++) hist[b] = make_double2(0.0, 0.0);
	if(in_trajectory && R.records == nullptr)
	{
		// stopped in mid-trajectory: count the work done so far
		unsigned long long* c = R.counters + static_cast<size_t>(L.point) * DMS_NUM_COUNTERS;
		atomicAdd(c + DMS_CNT_UNFINISHED_TRAJECTORIES, 1ULL);
		atomicAdd(c + DMS_CNT_UNFINISHED_SCATTERINGS, static_cast<unsigned long long>(L.nscat));
		atomicAdd(c + DMS_CNT_UNFINISHED_RK_STEPS, static_cast<unsigned long long>(L.hot().steps));
		atomicAdd(c + DMS_CNT_UNFINISHED_RK_ATTEMPTS, static_cast<unsigned long long>(L.hot().attempts));
	}
}

// The launch of a kernel that runs lane_loop, with the shared memory of its lanes.
template <class Lane>
void Launch_With_Hot_States(void (*kernel)(const RunParams), const RunParams& p, int blocks, int threads, cudaStream_t stream)
{
	const size_t bytes = sizeof(typename Lane::Hot) * threads;
	// (a refusal shows as the launch's error)
	cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
	kernel<<<blocks, threads, bytes, stream>>>(p);
}

}	// namespace lane
}	// namespace dms
