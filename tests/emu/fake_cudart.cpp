// A stand-in for the CUDA runtime: the library's host code runs without a GPU. Device memory is host memory, copies are
// done at once, kernels do nothing. It answers with errors where the runtime would: a copy from or to a null buffer, a
// launch with more dynamic shared memory than the kernel was allowed on the current device, an allocation beyond the
// device's memory (fake::limit bytes, pools included while they keep what was freed). Test harness only.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>

#include "fake_cudart.h"

namespace fake {
std::mutex mu;
size_t limit = 8ull << 30;
size_t used[kDevices];                       // bytes held on each device, by allocations and by pools
std::map<const void*, Block> blocks;         // live allocations
std::map<void*, Pool> pools;
std::set<std::pair<int, const void*>> allowed;
std::map<std::pair<int, const void*>, int> smem;
size_t launches[kDevices];
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
struct Call {
	dim3 grid, block;
	size_t smem;
	void* stream;
};
thread_local Call pushed;

cudaError_t Set(cudaError_t e)
{
	if (e != cudaSuccess) { last = e; }
	return e;
}

void* Token() { return std::malloc(16); }

cudaError_t Allocate(void** p, size_t bytes, bool host, void* pool)
{
	std::lock_guard<std::mutex> g(mu);
	Pool* from = pool ? &pools[pool] : nullptr;
	const size_t kept = from ? std::min(from->kept, bytes) : 0;
	if (!host && used[device] + bytes - kept > limit) { return Set(cudaErrorMemoryAllocation); }
	*p = std::malloc(bytes ? bytes : 1);
	if (from) { from->kept -= kept; }
	if (!host) { used[device] += bytes - kept; }
	blocks[*p] = Block{bytes, device, host, pool};
	return cudaSuccess;
}

cudaError_t Release(void* p)
{
	if (!p) { return cudaSuccess; }
	std::lock_guard<std::mutex> g(mu);
	const auto it = blocks.find(p);
	if (it == blocks.end()) { return Set(cudaErrorInvalidValue); }
	const Block b = it->second;
	blocks.erase(it);
	std::free(p);
	if (b.pool) { pools[b.pool].kept += b.bytes; }
	else if (!b.host) { used[b.device] -= b.bytes; }
	return cudaSuccess;
}

// A synchronisation returns what a pool holds above its threshold.
void Trim(void* pool, size_t keep)
{
	std::lock_guard<std::mutex> g(mu);
	for (auto& p : pools) {
		if (pool && p.first != pool) { continue; }
		const size_t to = pool ? keep : p.second.threshold;
		if (p.second.kept > to) {
			used[p.second.device] -= p.second.kept - to;
			p.second.kept = to;
		}
	}
}

cudaError_t Launch(const void* kernel, size_t bytes)
{
	std::lock_guard<std::mutex> g(mu);
	const auto it = smem.find({device, kernel});
	if (bytes > 48 * 1024 && (it == smem.end() || static_cast<size_t>(it->second) < bytes)) { return Set(cudaErrorInvalidValue); }
	++launches[device];
	return cudaSuccess;
}
}  // namespace fake

using namespace fake;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d)
{
	if (d < 0 || d >= kDevices) { return Set(cudaErrorInvalidDevice); }
	device = d;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaMalloc(void** p, size_t n) { return Allocate(p, n, false, nullptr); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return Allocate(p, n, false, nullptr); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) { return Allocate(p, n, false, pool); }
cudaError_t cudaMallocHost(void** p, size_t n) { return Allocate(p, n, true, nullptr); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return Allocate(p, n, true, nullptr); }
cudaError_t cudaFree(void* p) { return Release(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return Release(p); }
cudaError_t cudaFreeHost(void* p) { return Release(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *t = limit; *f = limit - used[device]; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps* props)
{
	std::lock_guard<std::mutex> g(mu);
	*pool = static_cast<cudaMemPool_t>(Token());
	pools[*pool] = Pool{props->location.id, 0, 0};
	return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t pool, cudaMemPoolAttr a, void* v)
{
	if (a == cudaMemPoolAttrReleaseThreshold) { pools[pool].threshold = *static_cast<uint64_t*>(v); }
	return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t pool, cudaMemPoolAttr a, void* v)
{
	size_t live = 0;
	for (auto& b : blocks) { live += b.second.pool == pool ? b.second.bytes : 0; }
	if (a == cudaMemPoolAttrReservedMemCurrent) { *static_cast<uint64_t*>(v) = pools[pool].kept + live; }
	return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) { Trim(pool, keep); return cudaSuccess; }
static cudaError_t Copy(void* d, const void* s, size_t n)
{
	if (n > 0 && (!d || !s)) { return Set(cudaErrorInvalidValue); }
	if (n > 0) { std::memcpy(d, s, n); }
	return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return Copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { return Copy(d, s, n); }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
	std::lock_guard<std::mutex> g(mu);
	*a = cudaPointerAttributes{};
	auto it = blocks.upper_bound(p);
	if (it != blocks.begin()) {
		--it;
		if (static_cast<const char*>(p) < static_cast<const char*>(it->first) + it->second.bytes) {
			a->type = it->second.host ? cudaMemoryTypeHost : cudaMemoryTypeDevice;
		}
	}
	return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*)
{
	static std::map<int, void*> at;
	void*& v = at[device];
	if (!v) { v = std::calloc(1, 8 << 20); }
	*p = v;
	return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorNotSupported; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = static_cast<cudaStream_t>(Token()); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { Trim(nullptr, 0); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = static_cast<cudaGraph_t>(Token()); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { std::free(g); return cudaSuccess; }
cudaError_t cudaGraphInstantiateWithFlags(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = static_cast<cudaGraphExec_t>(Token()); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = static_cast<cudaEvent_t>(Token()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v)
{
	std::lock_guard<std::mutex> g(mu);
	if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) { smem[{device, f}] = v; }
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t bytes, cudaStream_t) { return Launch(f, bytes); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return Launch(f, c->dynamicSmemBytes); }

unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t bytes, void* stream)
{
	pushed = Call{grid, block, bytes, stream};
	return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* bytes, void* stream)
{
	*grid = pushed.grid;
	*block = pushed.block;
	*bytes = pushed.smem;
	*static_cast<void**>(stream) = pushed.stream;
	return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
