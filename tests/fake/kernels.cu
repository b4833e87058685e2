// Stand-ins for the engine's kernel launches, for tests of its host code without a GPU.  A trajectory launch is
// written down (fake_launches), and "runs" at fake_rate trajectories per second, 100 steps each, until its work is
// done or the host sets the cancel flag.
#include <chrono>
#include <cstring>
#include <string>
#include <vector>

#include "dms_host_model.h"
#include "dms_kernels.cuh"

extern "C" {
void fake_launched(cudaStream_t s, const char* what);
void fake_set_busy(int (*f)(void));
size_t fake_room(const void* p);
extern float fake_run_ms;

struct FakeLaunch
{
	uint64_t total, done, parked_room;
	int32_t blocks, threads, mixed, resume, lanes_per_block, lockstep_min;
	uint32_t queue_chunk;
	uint32_t parked_capacity;
	int32_t options[6];  // scatter_batch, scatter_wait, final_batch, final_wait; the batches of a block
};
double fake_rate = 1e9;
}

namespace dms
{
namespace
{
using Clock = std::chrono::steady_clock;
std::vector<FakeLaunch> launches;
RunParams running;
bool in_flight = false;
Clock::time_point started;

int busy()
{
	if(!in_flight)
		return 0;
	const double seconds = std::chrono::duration<double>(Clock::now() - started).count();
	const double done = seconds * fake_rate;
	const bool finished = done >= static_cast<double>(running.total), cancelled = *running.cancel != 0;
	if(!finished && !cancelled)
		return 1;
	const uint64_t n = finished ? running.total : static_cast<uint64_t>(done);
	*running.queue_head = n;
	*running.status = finished ? 0u : STATUS_CANCELLED;
	if(running.counters != nullptr)
		running.counters[static_cast<size_t>(running.range_point[0]) * DMS_NUM_COUNTERS + DMS_CNT_RK_STEPS] += 100 * n;
	fake_run_ms = static_cast<float>((finished ? static_cast<double>(running.total) / fake_rate : seconds) * 1e3);
	for(FakeLaunch& l : launches)
		if(l.done == ~0ULL)
			l.done = n;
	in_flight = false;
	return 0;
}

void launch(const RunParams& p, int blocks, int threads, cudaStream_t s, int mixed)
{
	fake_launched(s, "trajectories behind a legacy write");
	fake_set_busy(busy);
	FakeLaunch l{};
	l.total = p.total;
	l.done = ~0ULL;
	l.parked_room = p.parked ? fake_room(p.parked) : 0;
	l.parked_capacity = p.parked_capacity;
	l.blocks = blocks;
	l.threads = threads;
	l.mixed = mixed;
	l.resume = p.resume;
	l.lanes_per_block = p.lanes_per_block;
	l.lockstep_min = p.lockstep_min;
	l.queue_chunk = p.queue_chunk;
	l.options[0] = p.scatter_batch;
	l.options[1] = p.scatter_wait;
	l.options[2] = p.final_batch;
	l.options[3] = p.final_wait;
	l.options[4] = p.block_scatter_batch;
	l.options[5] = p.block_final_batch;
	launches.push_back(l);
	if(!p.resume)
	{
		running = p;
		started = Clock::now();
		in_flight = true;
	}
}
}	// namespace

void Launch_Initial_States(const RunParams&, cudaStream_t s) { fake_launched(s, "initial states behind a legacy write"); }
void Launch_Trajectories(const RunParams& p, int blocks, int threads, cudaStream_t s) { launch(p, blocks, threads, s, 0); }
void Launch_Trajectories_Mixed(const RunParams& p, int blocks, int threads, cudaStream_t s) { launch(p, blocks, threads, s, 1); }
void Launch_To_Float(const double*, float*, size_t, cudaStream_t s) { fake_launched(s, "grid image behind a legacy write"); }
void Launch_Rate_Grid(const DevSolar&, const DevPoint*, double*, int, cudaStream_t s) { fake_launched(s, "rate grid behind a legacy write"); }
void Launch_Rate_Query(const DevSolar&, const DevPoint*, int, const double*, const double*, double*, size_t, cudaStream_t s)
{
	fake_launched(s, "rate query behind a legacy write");
}
double Measure_FP64_Peak(int, cudaStream_t) { return 1.0; }
void Check_Certified_Math(uint64_t, uint64_t, unsigned long long*, int, cudaStream_t) {}
unsigned int Take_Bounds_Status() { return 0; }
unsigned int Take_Bounds_Status_Mixed() { return 0; }

}	// namespace dms

extern "C" int fake_take_launches(FakeLaunch* out, int capacity)
{
	const int n = static_cast<int>(dms::launches.size());
	for(int i = 0; i < n && i < capacity; i++) out[i] = dms::launches[i];
	dms::launches.clear();
	return n;
}
