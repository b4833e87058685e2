// A stand-in for the CUDA runtime calls of the engine's host code, for tests without a GPU.
//
// "Device" memory is host memory and every copy is made at once; what is modelled is the order.  A
// memset, a copy to the device and a copy on the device may still be under way when the call returns
// (the documented behaviour for pageable host memory).  Work on a non-blocking stream is not ordered behind
// it: a kernel launched, or memory touched, on such a stream before somebody waited for the legacy stream is
// recorded as a violation.
#include <cuda_runtime_api.h>

#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace
{
struct Range
{
	const char* p;
	size_t n;
};
std::vector<Range> legacy_pending;           // writes that may still be under way on the legacy stream
std::vector<std::string> violations;
std::map<const char*, size_t> allocations;
int (*run_busy)(void) = nullptr;             // set by the fake kernels: whether a run is in flight
cudaStream_t const STREAMS[2] = {reinterpret_cast<cudaStream_t>(0x100), reinterpret_cast<cudaStream_t>(0x200)};
int streams_made = 0;
std::map<cudaEvent_t, std::chrono::steady_clock::time_point> events;

bool is_legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }

// (fresh memory is zero, and nothing here writes to the large arrays)
void fill(void* p, int v, size_t n)
{
	if(v != 0 || n <= size_t{16} << 20)
		memset(p, v, n);
}

void touched(const void* p, size_t n, cudaStream_t s, const char* what)
{
	if(is_legacy(s))
		return;
	const char* a = static_cast<const char*>(p);
	for(const Range& r : legacy_pending)
		if(a < r.p + r.n && r.p < a + n)
		{
			violations.push_back(what);
			return;
		}
}
}	// namespace

extern "C" {

void fake_launched(cudaStream_t s, const char* what)
{
	if(!is_legacy(s) && !legacy_pending.empty())
		violations.push_back(what);
}
void fake_set_busy(int (*f)(void)) { run_busy = f; }
int fake_violations(char* text, int capacity)
{
	std::string all;
	for(const std::string& v : violations) all += v + "; ";
	const int n = static_cast<int>(violations.size());
	violations.clear();
	strncpy(text, all.c_str(), capacity - 1);
	return n;
}
// The size of the allocation that p lies in and p's place in it.
size_t fake_room(const void* p)
{
	auto it = allocations.upper_bound(static_cast<const char*>(p));
	if(it == allocations.begin())
		return 0;
	--it;
	const size_t at = static_cast<const char*>(p) - it->first;
	return at < it->second ? it->second - at : 0;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }

size_t fake_malloc_limit = ~size_t{0};  // a larger allocation fails
cudaError_t cudaMalloc(void** p, size_t n)
{
	if(n > fake_malloc_limit)
		return cudaErrorMemoryAllocation;
	*p = calloc(n ? n : 1, 1);
	allocations[static_cast<char*>(*p)] = n;
	return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p)
{
	allocations.erase(static_cast<char*>(p));
	free(p);
	return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int)
{
	*p = calloc(n, 1);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
	free(p);
	return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned int)
{
	*d = h;
	return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n)
{
	fill(p, v, n);
	legacy_pending.push_back({static_cast<char*>(p), n});
	return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s)
{
	touched(p, n, s, "memset on memory that the legacy stream still writes");
	fill(p, v, n);
	if(is_legacy(s))
		legacy_pending.push_back({static_cast<char*>(p), n});
	return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind)
{
	memcpy(d, s, n);
	if(kind == cudaMemcpyDeviceToHost)
		legacy_pending.clear();  // the copy is behind them, and is waited for
	else
		legacy_pending.push_back({static_cast<char*>(d), n});
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s)
{
	touched(d, n, s, "copy to memory that the legacy stream still writes");
	touched(src, n, s, "copy from memory that the legacy stream still writes");
	memcpy(d, src, n);
	return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int)
{
	*s = STREAMS[streams_made++ & 1];
	return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return run_busy && run_busy() ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
	if(is_legacy(s))
		legacy_pending.clear();
	return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e)
{
	*e = reinterpret_cast<cudaEvent_t>(malloc(1));
	return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
	free(e);
	return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
	events[e] = std::chrono::steady_clock::now();
	return cudaSuccess;
}
float fake_run_ms = 1.0f;  // the device time of the last run
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
	*ms = fake_run_ms;
	return cudaSuccess;
}

// what the compiler adds to a file with kernels
void** __cudaRegisterFatBinary(void*)
{
	static void* handle;
	return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned int __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t s)
{
	fake_launched(s, "kernel behind a legacy write");
	return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*)
{
	static char* scratch = static_cast<char*>(calloc(size_t{16} << 20, 1));
	*p = scratch;
	return cudaSuccess;
}

}	// extern "C"
