// Exclusive prefix sums of uint32 in place, with the element counts either known on the host or read from device
// memory (so a chain of kernels needs no host round trip). data[n] receives the total; `total`, when given, too.
//
// One launch scans up to kMaxScans arrays in a single pass (decoupled look-back: Merrill and Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", 2016): a CTA takes the next tile of 4096 entries, publishes its sum,
// adds up its predecessors' published sums until one that carries its whole prefix, and writes the tile. Tiles are
// taken in order, so a tile's predecessors are always held by running CTAs; the wait for them is bounded all the same
// (an exhausted wait sets *fault and the host fails the call). Bound: launch latency, the arrays being short (a chunk
// of one frame has one tile per array). Scanning tiles, tile sums and offsets in three launches per array took 18 of a
// chunk's 45 segmentation launches, now 3.
#include <algorithm>

#include "pt_common.cuh"

namespace ptb {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;
constexpr int kScanPolls = 1 << 22;  // a predecessor's sum arrives within microseconds
// State of a tile: 0 nothing yet, else kSum | its sum or kPrefix | the sum up to and including it.
constexpr unsigned long long kSum = 1ull << 32, kPrefix = 2ull << 32;

struct Scans {
	ScanJob job[kMaxScans];
	unsigned long long* state[kMaxScans];  // [0] ticket, [1 + tile]
	uint32_t* fault;
};

__host__ __device__ __forceinline__ uint32_t Tiles(uint32_t n)
{
	return static_cast<uint32_t>((static_cast<unsigned long long>(n) + kScanTile - 1) / kScanTile);
}

// Block-wide exclusive scan of one value per thread; returns the block total in *total.
__device__ uint32_t BlockExclusive(uint32_t v, uint32_t* warpSums, uint32_t* total)
{
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	uint32_t x = v;
	#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
		if (lane >= d) { x += y; }
	}
	if (lane == 31) { warpSums[wid] = x; }
	__syncthreads();
	if (wid == 0) {
		uint32_t w = warpSums[lane];
		#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
			if (lane >= d) { w += y; }
		}
		warpSums[lane] = w;  // inclusive over warps
	}
	__syncthreads();
	const uint32_t warpBase = wid > 0 ? warpSums[wid - 1] : 0u;
	*total = warpSums[kScanThreads / 32 - 1];
	return warpBase + x - v;
}

// Sum of the tiles before `tile` (warp 0): 32 predecessors at a time, back to the nearest with its whole prefix.
__device__ uint32_t LookBack(volatile unsigned long long* tiles, uint32_t tile, uint32_t* fault)
{
	const int lane = threadIdx.x & 31;
	uint32_t sum = 0;
	for (long long last = static_cast<long long>(tile) - 1; last >= 0; last -= 32) {
		const long long i = last - lane;
		unsigned long long s = kPrefix;  // before the first tile: a prefix of zero
		for (int poll = 0; poll < kScanPolls; ++poll) {
			if (i >= 0) { s = tiles[i]; }
			if (__ballot_sync(0xffffffffu, s == 0) == 0) { break; }
		}
		if (__ballot_sync(0xffffffffu, s == 0) != 0) {
			if (lane == 0) { atomicExch(fault, 1u); }
			return sum;
		}
		const unsigned full = __ballot_sync(0xffffffffu, (s & kPrefix) != 0);
		const int stop = full ? __ffs(full) - 1 : 31;
		uint32_t v = lane <= stop ? static_cast<uint32_t>(s) : 0u;
		#pragma unroll
		for (int d = 16; d > 0; d >>= 1) { v += __shfl_xor_sync(0xffffffffu, v, d); }
		sum += v;
		if (full) { break; }
	}
	return sum;
}

__global__ void __launch_bounds__(kScanThreads) ScanKernel(Scans s)
{
	PTB_AFTER_PREVIOUS();
	__shared__ uint32_t warpSums[32];
	__shared__ uint32_t tileOf, before;
	const ScanJob job = s.job[blockIdx.y];
	unsigned long long* state = s.state[blockIdx.y];
	const uint32_t n = job.nptr ? min(*job.nptr, job.cap) : job.nconst;
	const uint32_t tiles = max(Tiles(n), 1u);
	while (true) {
		if (threadIdx.x == 0) { tileOf = atomicAdd(reinterpret_cast<unsigned int*>(state), 1u); }
		__syncthreads();
		const uint32_t tile = tileOf;
		if (tile >= tiles) { return; }
		const unsigned long long first = static_cast<unsigned long long>(tile) * kScanTile + threadIdx.x * kScanItems;
		uint32_t v[kScanItems] = {0u, 0u, 0u, 0u};
		const bool whole = first + kScanItems <= n;
		if (whole) {
			const uint4 q = *reinterpret_cast<const uint4*>(job.data + first);
			v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
		}
		else {
			#pragma unroll
			for (int k = 0; k < kScanItems; ++k) { v[k] = first + k < n ? job.data[first + k] : 0u; }
		}
		uint32_t total;
		uint32_t off = BlockExclusive(v[0] + v[1] + v[2] + v[3], warpSums, &total);
		if (threadIdx.x < 32) {
			volatile unsigned long long* mine = state + 1 + tile;
			if (threadIdx.x == 0) { *mine = (tile == 0 ? kPrefix : kSum) | total; }
			const uint32_t prefix = tile == 0 ? 0u : LookBack(state + 1, tile, s.fault);
			if (threadIdx.x == 0) {
				if (tile > 0) { *mine = kPrefix | static_cast<uint32_t>(prefix + total); }
				before = prefix;
				if (tile + 1 == tiles) {
					job.data[n] = prefix + total;
					if (job.total) { *job.total = prefix + total; }
				}
			}
		}
		__syncthreads();
		off += before;
		if (whole) { *reinterpret_cast<uint4*>(job.data + first) = make_uint4(off, off + v[0], off + v[0] + v[1], off + v[0] + v[1] + v[2]); }
		else {
			#pragma unroll
			for (int k = 0; k < kScanItems; ++k) {
				if (first + k < n) { job.data[first + k] = off; }
				off += v[k];
			}
		}
	}
}

}  // namespace

size_t ScanStateWords(uint32_t cap) { return static_cast<size_t>(Tiles(cap)) + 2; }

// state: the jobs' words (ScanStateWords of each capacity, one after the other), zeroed before the launch; fault: a
// device word set when a wait runs out. data must be 16-byte aligned and hold cap + 1 entries.
bool ExclusiveScans(const ScanJob* jobs, int count, unsigned long long* state, uint32_t* fault, cudaStream_t st)
{
	Scans s{};
	uint32_t blocks = 1;
	for (int k = 0; k < count; ++k) {
		s.job[k] = jobs[k];
		s.state[k] = state;
		state += ScanStateWords(jobs[k].cap);
		// a count known only on the device is a few per cent of its capacity: a CTA per 16 tiles of that
		blocks = std::max(blocks, jobs[k].nptr ? Tiles(jobs[k].cap) / 16 : Tiles(jobs[k].nconst));
	}
	s.fault = fault;
	const bool ok = LaunchChained(ScanKernel, dim3(std::min<uint32_t>(blocks, 148u), count), kScanThreads, 0, st, s);
	CountLaunch();
	return ok;
}

}  // namespace ptb
