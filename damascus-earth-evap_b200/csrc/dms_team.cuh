// The team: three warps that make the steps of a lone lane together (latency form of the trajectory kernels).
#pragma once

#include "dms_lane.cuh"

namespace dms
{
namespace lane
{

// Team: a lane that runs alone in its block spends its step on one dependent chain, and a warp issues one
// instruction every 4.4 cycles of it.  Once the other warps of a 128-thread block have run out of work,
// two of them take over parts of the lone lane's steps, one step apart, with a barrier per step:
//   propagate  the bounds and the RK45 attempts of the next step, from its own last result
//   judge      (the lane's own warp) event, optical depth and decisions of the step before
//   commit     bincount and energy drift of the step before that
// (A lone lane's orbit of some 9 steps often leaves the boundary radius and comes back by Kepler's equation,
// which the lane solves with the team's step in hand.)
// The propagating warp runs ahead as if every step ended plainly.  A step that does not is not committed:
// a depth rejection restarts the propagation from the step's start with the shorter step; anything
// else (a scattering, the boundary, a failure) hands the state at the step's start back to the lane, which
// makes that step by itself.  Every value is formed by the functions of the one-lane pass from the same
// arguments, so the results are the same bits.  The barriers count whole warps that all run the same loop;
// the only wait by polling is that of a warp without work for a team to form, and it ends some time after the
// block's last sign of life.
// A lone lane's step takes 5.7 -> 3.3 us in FP64 and 4.4 -> 3.0 us in the mixed form; 16 384 Parameter-point
// trajectories of m = 0.3 GeV, 1e-36 cm^2 426 -> 259 ms in the mixed form, 128 25 -> 18 ms.
struct TeamState  // the propagator at the start of a step
{
	double time, radius, phi, v_radial, step, speed, rate;
	int inner, ok;  // attempts of the step that led here; whether the propagating warp could make it
};
template <class PropT, class EvT>
struct TeamBox
{
	int word;       // warps without work; TEAM_FORMED once a team has formed, negative when none can
	int alive;      // raised now and then by the warps that make steps
	int command;    // TEAM_RUN, TEAM_EXIT
	int verdict[2];
	int captured, bound, bmin, bmax, cbin;
	const DevPoint* P;
	double2* hist;
	double m_dm;
	PropT pr;       // the constants of the segment
	double origin, prev_time, prev_r, prev_v2, t_last_bound, free_flight_E, max_drift_eV, max_drift_rel;
	double2 cval;
	TeamState s[4];  // by step number modulo 4
	EvT e[4];        // the events at those states
};
constexpr int TEAM_FORMED = 0x100, TEAM_NEVER = -0x10000, TEAM_RUN = 0, TEAM_EXIT = 1;
enum Verdict : int
{
	VERDICT_PLAIN = 0,
	VERDICT_RESTART = 1,
	VERDICT_STOP = 2,
	VERDICT_BOUNDARY = 3,  // the step ends at or beyond the boundary radius
	VERDICT_SCATTER = 4,   // the remaining optical depth lies in the step
	VERDICT_PAUSE = 5,     // not judged: the lane loop is due
};
constexpr int TEAM_MAX_STEPS = 512;                      // per call: the lane loop looks at the cancel flag between calls
// How long a warp without work waits for a team after the last sign of life of its block, which the warps at
// work give every 1 024 passes, some 10 ms (~20 s; in the checked build ~50 ms, for its tests).
#ifdef DMS_CHECKED
constexpr long long TEAM_WAIT_CYCLES = 100000000ll;
#else
constexpr long long TEAM_WAIT_CYCLES = 40000000000ll;
#endif

__device__ __forceinline__ void team_barrier() { asm volatile("bar.sync 1, 96;" ::: "memory"); }

// The propagator at a state of the box.
template <class PropT, class EvT>
__device__ __forceinline__ PropT team_prop(const TeamBox<PropT, EvT>& b, const TeamState& s)
{
	PropT q = b.pr;
	q.time = s.time;
	q.radius = s.radius;
	q.phi = s.phi;
	q.v_radial = s.v_radial;
	q.radial_mode = 0;
	return q;
}

// The loop of the three warps: role 0 judges, 1 propagates, 2 commits.  Returns the number of the step at
// whose start the lane goes on by itself (the states and events are in the box).
template <class T>
__device__ __forceinline__ int team_loop(const RunParams& R, typename T::Box& b, typename T::Lane& L, int role, bool mine, double* buffer,
                                         typename T::Ctx& c, int& last)
{
	const bool lane0 = (threadIdx.x & 31) == 0;
	int j = 0;             // the step to judge
	bool have = false;     // ... whose result is there
	bool pending = false;  // step j - 1 is to be committed
	for(int pass = 0;; pass++)
	{
		if(role == 1)
		{
			const int from = have ? j + 1 : j;
			if(lane0)
				T::propagate(R, b, b.s[from & 3], b.s[(from + 1) & 3]);
		}
		else if(role == 0)
		{
			if(have)
			{
				int v = VERDICT_PAUSE;
				if(pass < TEAM_MAX_STEPS)
					v = T::judge(R, b, b.s[j & 3], b.e[j & 3], b.s[(j + 1) & 3], b.e[(j + 1) & 3], L, mine, buffer, c);
				if(mine)
					b.verdict[pass & 1] = v;
			}
		}
		else if(pending && lane0)
			T::commit(R, b, L, b.e[j & 3]);
		__syncwarp();
		team_barrier();
		pending = false;
		if(!have)
		{
			have = true;
			continue;
		}
		const int v = *reinterpret_cast<volatile int*>(&b.verdict[pass & 1]);
		last = v;
		if(v >= VERDICT_STOP)
			break;
		if(v == VERDICT_PLAIN)
		{
			j++;
			pending = true;
		}
		else
			have = false;
	}
	return j;
}

// T supplies the parts of a step: fresh, fits, propagate, judge, commit and finish, for its Lane, Box and Ctx types.
template <class T>
struct Team
{
	using Lane = typename T::Lane;
	using Box = typename T::Box;
	static __device__ __forceinline__ Box& box()
	{
		__shared__ Box b;
		return b;
	}
	__device__ __forceinline__ void team_init() const
	{
		box().word = 0;
		box().alive = 0;
		box().command = TEAM_RUN;
	}
	// Called now and then by a whole warp at work, for those that wait.
	__device__ __forceinline__ void team_alive() const
	{
		if((threadIdx.x & 31) == 0)
			atomicAdd(&box().alive, 1);
	}
	// Called by a whole warp without work: it helps a lone lane of its block, if one forms a team, until that
	// lane's trajectory has ended.
	__device__ __noinline__ void team_help(const RunParams& R, Lane& L, double* buffer) const
	{
		Box& b = box();
		const bool lane0 = (threadIdx.x & 31) == 0;
		int rank = 0;
		if(lane0)
			rank = atomicAdd(&b.word, 1);
		rank = __shfl_sync(0xffffffffu, rank, 0);
		if(rank == 3)
		{
			team_forgo();  // the last warp of the block: nobody is left to help
			return;
		}
		long long t0 = clock64();
		int seen_alive = 0;
		for(unsigned int poll = 1;; poll++)
		{
			int word = 0;
			if(lane0)
			{
				word = *reinterpret_cast<volatile int*>(&b.word);
				const int alive = *reinterpret_cast<volatile int*>(&b.alive);
				if(alive != seen_alive)
				{
					seen_alive = alive;
					t0 = clock64();
				}
				bool leave = clock64() - t0 > TEAM_WAIT_CYCLES;
				const bool gave_up = leave;
				if((poll & 255u) == 0u)
					leave |= *R.cancel != 0;
				// a warp leaves by putting the count out of reach, which no formed team can follow
				if(leave && word >= 0 && word < TEAM_FORMED)
				{
					const int seen = atomicCAS(&b.word, word, TEAM_NEVER);
					if(gave_up && seen == word)
						DMS_COUNT_FORM(FORM_HELPERS_GAVE_UP, 1);
					word = seen == word ? TEAM_NEVER : seen;
				}
			}
			word = __shfl_sync(0xffffffffu, word, 0);
			if(word < 0)
				return;
			if(word >= TEAM_FORMED)
				break;
			__nanosleep(1000);
		}
		if(rank > 1)
			return;  // two helpers are enough
		for(;;)
		{
			team_barrier();  // the owner has filled the box
			if(*reinterpret_cast<volatile int*>(&b.command) == TEAM_EXIT)
				return;
			if(rank == 1)
			{
				L.hot().is_captured = b.captured;
				L.bound_state = b.bound;
				L.bmin = b.bmin;
				L.bmax = b.bmax;
				L.cbin = b.cbin;
				L.cval = b.cval;
				L.hot().origin = b.origin;
				L.prev_time = b.prev_time;
				L.prev_r = b.prev_r;
				L.prev_v2 = b.prev_v2;
				L.t_last_bound = b.t_last_bound;
				L.free_flight_E = b.free_flight_E;
				L.max_drift_eV = b.max_drift_eV;
				L.max_drift_rel = b.max_drift_rel;
			}
			typename T::Ctx c;
			int last;
			team_loop<T>(R, b, L, rank == 0 ? 1 : 2, false, buffer, c, last);
			if(rank == 1 && lane0)
			{
				b.bmin = L.bmin;
				b.bmax = L.bmax;
				b.cbin = L.cbin;
				b.cval = L.cval;
				b.prev_time = L.prev_time;
				b.prev_r = L.prev_r;
				b.prev_v2 = L.prev_v2;
				b.t_last_bound = L.t_last_bound;
				b.max_drift_eV = L.max_drift_eV;
				b.max_drift_rel = L.max_drift_rel;
			}
			__syncwarp();
			team_barrier();  // the owner may read the box
		}
	}
	// Called by the whole warp of a lone lane (`mine` on that lane, at the start of a step): forms the team if the
	// other three warps are without work.
	__device__ __forceinline__ bool team_form() const
	{
		Box& b = box();
		int formed = 0;
		if((threadIdx.x & 31) == 0)
			formed = *reinterpret_cast<volatile int*>(&b.word) == 3 && atomicCAS(&b.word, 3, TEAM_FORMED) == 3 ? 1 : 0;
		if(formed)
			DMS_COUNT_FORM(FORM_TEAMS, 1);
		return __shfl_sync(0xffffffffu, formed, 0) != 0;
	}
	// A warp that stops in mid-trajectory: no team can form any more.
	__device__ __forceinline__ void team_forgo() const
	{
		if((threadIdx.x & 31) == 0)
			atomicExch(&box().word, TEAM_NEVER);
	}
	__device__ __forceinline__ void team_dismiss() const
	{
		Box& b = box();
		if((threadIdx.x & 31) == 0)
			*reinterpret_cast<volatile int*>(&b.command) = TEAM_EXIT;
		__syncwarp();
		team_barrier();
	}
	// Steps of the lone lane made by the team; the lane's state is that at the start of a step before and
	// after (or `phase`, its phase, says otherwise).  Adds the number of steps to `iter`; returns whether
	// the lane must make its next step alone.
	__device__ __noinline__ bool team_run(const RunParams& R, const DevPoint* __restrict__ P, double m_dm, Lane& L, double2* hist, bool mine,
	                                     double* buffer, int& phase, uint64_t& iter) const
	{
		Box& b = box();
		if(mine && !L.hot().next_valid)
			T::fresh(R, P, L);
		const bool fit = mine && T::fits(L);
		if(!__any_sync(0xffffffffu, fit))
			return true;
		if(mine)
		{
			b.P = P;
			b.hist = hist;
			b.m_dm = m_dm;
			b.pr = L.hot().pr;
			b.captured = L.hot().is_captured;
			b.bound = L.bound_state;
			b.bmin = L.bmin;
			b.bmax = L.bmax;
			b.cbin = L.cbin;
			b.cval = L.cval;
			b.origin = L.hot().origin;
			b.prev_time = L.prev_time;
			b.prev_r = L.prev_r;
			b.prev_v2 = L.prev_v2;
			b.t_last_bound = L.t_last_bound;
			b.free_flight_E = L.free_flight_E;
			b.max_drift_eV = L.max_drift_eV;
			b.max_drift_rel = L.max_drift_rel;
			TeamState& s = b.s[0];
			s.time = L.hot().pr.time;
			s.radius = L.hot().pr.radius;
			s.phi = L.hot().pr.phi;
			s.v_radial = L.hot().pr.v_radial;
			s.step = L.hot().pr.time_step;
			s.speed = L.hot().next_speed;
			s.rate = L.hot().next_rate;
			b.e[0] = L.hot().before;
			b.e[0].t = L.hot().pr.time;
		}
		__syncwarp();
		team_barrier();
		typename T::Ctx c;
		int last = VERDICT_PLAIN;
		const int j = team_loop<T>(R, b, L, 0, mine, buffer, c, last);
		team_barrier();  // the committing warp has written its part back
		if(mine)
		{
			DMS_COUNT_FORM(FORM_TEAM_STEPS, j);
			const TeamState& s = b.s[j & 3];
			L.hot().pr.time = s.time;
			L.hot().pr.radius = s.radius;
			L.hot().pr.phi = s.phi;
			L.hot().pr.v_radial = s.v_radial;
			L.hot().pr.time_step = s.step;
			L.hot().next_speed = s.speed;
			L.hot().next_rate = s.rate;
			if(j > 0)
			{
				L.hot().before = b.e[j & 3];
				L.hot().before_valid = 2;
			}
			L.bmin = b.bmin;
			L.bmax = b.bmax;
			L.cbin = b.cbin;
			L.cval = b.cval;
			L.prev_time = b.prev_time;
			L.prev_r = b.prev_r;
			L.prev_v2 = b.prev_v2;
			L.t_last_bound = b.t_last_bound;
			L.max_drift_eV = b.max_drift_eV;
			L.max_drift_rel = b.max_drift_rel;
		}
		// a step that ends at the boundary or in a scattering is finished here with what the team made of it
		if(mine && (last == VERDICT_BOUNDARY || last == VERDICT_SCATTER))
			T::finish(R, P, m_dm, L, hist, c, b.s[(j + 1) & 3], last == VERDICT_SCATTER, phase);
		__syncwarp();
		iter += j;
		return last == VERDICT_STOP;
	}
};

}	// namespace lane
}	// namespace dms
