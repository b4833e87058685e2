// Kernel interfaces of the trajectory engine (launched from dms_capi.cu).
#pragma once

#include <cstdint>

#include "dms_device.cuh"

namespace dms
{

// The largest block of the trajectory kernels: all 16 warps that their registers allow per SM.
constexpr int MAX_THREADS = 512;
// The mixed form keeps less per lane: a launch with at least two trajectories for each lane of 20 warps runs
// that many, with 96 registers each.  2^20 Capture-mode trajectories with 512 / 640 / 768 / 1 024 threads took
// 27.0 / 25.3 / 25.9 / 27.3 ms; with 512 / 640 2^19 took 14.6 / 14.2, 2^18 8.5 / 8.3, 200 000 6.9 / 7.0, 2^17
// 5.3 / 5.5, 2^16 3.7 / 4.0.  The FP64 form took 40.9 / 41.4 / 44.6 / 48.6 ms for the first (448 / 384: 42.7 / 44.3).
constexpr int MAX_THREADS_MIXED = 640;
// Blocks of at most this many threads run the latency form of the kernels: one warp per scheduler, so
// the registers are not shared out among 16 warps.
constexpr int LATENCY_THREADS = 128;
// Room for one parked lane state.
constexpr size_t PARKED_BYTES = 1024;

// Status bits written by the kernels (device status word).
enum : unsigned int
{
	STATUS_CANCELLED = 1u,
	STATUS_BUDGET = 2u,
	STATUS_IC_REJECTION = 4u,
	STATUS_BAD_RANGE = 8u,
	STATUS_PARKED_FULL = 16u,  // more parked states than RunParams::parked_capacity
};

// Initial state of one work item, computed for the whole launch before the persistent kernel
// starts: the event after Initial_Conditions and the Kepler shift to the boundary (the raw
// initial event when the shift fails), and the uniform draws consumed.
enum : uint32_t
{
	INIT_IC_OK = 1u,     // initial conditions found within the attempt bound
	INIT_SHIFT_OK = 2u,  // Hyperbolic_Kepler_Shift succeeded
};
struct InitState
{
	Event ic;
	uint32_t draws;
	uint32_t flags;
};
static_assert(sizeof(InitState) == 64, "one initial state per 64 bytes");

struct RunParams
{
	DevSolar S;
	// FP32 images of the knot, G*M and G*M-slope tables (mixed-precision kernel only)
	const float4* sf_knots;
	const float* sf_vesc2_s;
	const uint16_t* sf_bucket;
	float sf_scale;
	int sf_single_step;
	const DevPoint* points;
	int n_points;
	// work: ranges and their prefix offsets (n_ranges + 1)
	const int32_t* range_point;
	const uint64_t* range_first;
	const uint64_t* range_offset;
	int n_ranges;
	uint64_t total;
	unsigned long long* queue_head;
	// options
	uint32_t seed;
	int capture_mode;
	uint64_t max_scatterings;
	uint64_t max_free_steps;
	double boundary;          // km
	uint64_t iteration_budget;
	uint64_t wall_limit_ns;  // per-trajectory wall-clock limit (max_trajectory_wall_time_sec); 0 = none
	// lane scheduling (dms_run_opts; never changes results): ids claimed per queue fetch and
	// the warp batching of scatterings and terminations
	uint32_t queue_chunk;
	int scatter_batch, scatter_wait, final_batch, final_wait;
	int block_scatter_batch, block_final_batch;  // the batches of a block in lockstep, in lanes of 64
	int lanes_per_block; // lanes of a block that take trajectories (all, fewer in a spread launch)
	int lockstep_min;    // lanes at work at which a block's warps leave the lockstep once the queue is empty
	// The tail of a throughput launch: a block with at most lockstep_min lanes at work and no more work parks
	// their states (PARKED_BYTES each) and ends; a latency launch behind it resumes them.
	unsigned char* parked;
	unsigned int parked_capacity;
	unsigned int* parked_count;
	int resume;          // 1: the lanes take the parked states instead of work indices
	int ic_max_attempts;
	// accumulators (accumulate mode)
	unsigned long long* counters;   // n_points x DMS_NUM_COUNTERS
	double* hists;                  // n_points x DMS_NUM_HISTS x DMS_NUM_BINS
	dms_evaporation_event* events;  // n_points x event_capacity
	unsigned long long* event_count;// n_points
	uint64_t event_capacity;
	dms_reflection* reflections;    // n_points x event_capacity
	unsigned long long* reflection_count; // n_points
	// records mode (records != nullptr): one record per work index
	dms_traj_record* records;
	double* rec_hist_dt;
	double* rec_hist_v2dt;
	// per-lane histogram scratch: lanes x DMS_NUM_BINS of (dt, v2dt)
	double2* lane_hist;
	// initial state of every work index (written by initial_state_kernel)
	InitState* init;
	const volatile int* cancel;
	unsigned int* status;
};

// Range of work index w: the largest k with range_offset[k] <= w (binary search).
__device__ __forceinline__ int find_range(const RunParams& R, uint64_t w)
{
	int lo = 0, hi = R.n_ranges - 1;
	while(lo < hi)
	{
		const int mid = (lo + hi + 1) >> 1;
		if(R.range_offset[mid] <= w)
			lo = mid;
		else
			hi = mid - 1;
	}
	return lo;
}

// Checked build: reads and clears the bounds-status bits of the FP64 and the mixed kernels'
// translation units (always 0 without DMS_CHECKED).
unsigned int Take_Bounds_Status();
unsigned int Take_Bounds_Status_Mixed();

#ifdef DMS_CHECKED
// The same for the counts of forms.
bool Take_Form_Counts(unsigned long long* counts);
bool Take_Form_Counts_Mixed(unsigned long long* counts);
#endif

// Initial states of all p.total work indices into p.init (one thread per work index); the
// trajectory kernels read them.  Launched on the same stream before every trajectory launch.
void Launch_Initial_States(const RunParams& p, cudaStream_t stream);
void Launch_Trajectories(const RunParams& p, int blocks, int threads, cudaStream_t stream);
void Launch_Rate_Grid(const DevSolar& S, const DevPoint* point, double* grid, int n, cudaStream_t stream);
void Launch_Rate_Query(const DevSolar& S, const DevPoint* point, int interpolated, const double* r, const double* v, double* out,
                       size_t n, cudaStream_t stream);
// mixed-precision (batched FP32) trajectory kernel and the FP32 image of a rate grid
void Launch_Trajectories_Mixed(const RunParams& p, int blocks, int threads, cudaStream_t stream);
void Launch_To_Float(const double* in, float* out, size_t n, cudaStream_t stream);
double Measure_FP64_Peak(int sm_count, cudaStream_t stream);
// Self-test of the certified division and square root (dms_fastmath.cuh) against IEEE on n
// random operand pairs; out (4 device counters, zeroed by the caller) as in dms_check_certified_math.
void Check_Certified_Math(uint64_t n, uint64_t seed, unsigned long long* out, int sm_count, cudaStream_t stream);

}	// namespace dms
