// Candidate construction from region sums, per-frame (Y, X) ordering of fitted rows and final row numbering.
//
// Reference: SegmentationInfo fields from ComputeStatistics (Segmentation2D.cpp:144-175); per-frame sort with
// std::weak_order on Y then X (FrameProcessor.cpp:35-39); Id / Plane / Index assignment (lib/Palm.cpp:24-43).
#include <algorithm>

#include "pt_common.cuh"

namespace ptb {

namespace {

// Region sums are exact integers in 2^-16 units, so x = sum(v j) / sum(v) is the reference's FP64 quotient exactly.
__global__ void BuildCandidates(Workspace ws)
{
	PTB_AFTER_PREVIOUS();
	const uint32_t n = min(ws.cnt->nfit, ws.capRows);
	for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
		const uint32_t r = ws.candRegion[k];
		const double sv = static_cast<double>(ws.regSumV[r]);
		Cand c;
		c.x = static_cast<double>(ws.regSumVJ[r]) / sv;
		c.y = static_cast<double>(ws.regSumVI[r]) / sv;
		c.intensity = sv * kW1Unit;
		c.surf = static_cast<double>(ws.regCount[r]);
		c.frame = static_cast<int>(ws.candFrame[k]);
		c.image = 0;
		ws.cand[k] = c;
	}
}

// Total order of std::weak_order on doubles: -NaN < -inf < ... < -0 == +0 < ... < +inf < +NaN.
__device__ __forceinline__ unsigned long long WeakKey(double d)
{
	if (d == 0.0) { d = 0.0; }
	unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(d));
	if (isnan(d)) { return (b >> 63) ? 0ull : ~0ull; }
	return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

constexpr int kSortThreads = 512;
constexpr int kSmemSort = 4096;  // rows sorted in shared memory (80 KB); larger frames sort in global scratch
constexpr int kSortBins = 2048;  // bands of Y
constexpr uint32_t kBandMax = 64;
constexpr size_t kSortSmemBytes = kSmemSort * (2 * sizeof(unsigned long long) + sizeof(uint32_t)) + kSortBins * sizeof(uint32_t);

__device__ __forceinline__ bool KeyLess(unsigned long long ya, unsigned long long xa, unsigned long long yb, unsigned long long xb)
{
	return ya < yb || (ya == yb && xa < xb);
}

// Bitonic sort of (ky, kx, idx) over a power-of-two length `len`; entries >= n hold +inf keys.
template <bool SMEM>
__device__ void Bitonic(unsigned long long* ky, unsigned long long* kx, uint32_t* id, uint32_t len)
{
	for (uint32_t size = 2; size <= len; size <<= 1) {
		for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
			for (uint32_t t = threadIdx.x; t < len / 2; t += blockDim.x) {
				const uint32_t lo = 2 * t - (t & (stride - 1));
				const uint32_t hi = lo + stride;
				const bool up = (lo & size) == 0;
				const bool swap = up ? KeyLess(ky[hi], kx[hi], ky[lo], kx[lo]) : KeyLess(ky[lo], kx[lo], ky[hi], kx[hi]);
				if (swap) {
					const unsigned long long a = ky[lo], b = kx[lo];
					const uint32_t c = id[lo];
					ky[lo] = ky[hi]; kx[lo] = kx[hi]; id[lo] = id[hi];
					ky[hi] = a; kx[hi] = b; id[hi] = c;
				}
			}
			if (SMEM) { __syncthreads(); }
			else { __syncthreads(); __threadfence_block(); }
		}
	}
}

// Order of a frame's n <= kSmemSort rows by bands of Y: the rows are dealt to kSortBins bands of equal height, then each
// row's place is its band's start plus the number of rows of the band before it. False (for every thread, with order
// undefined) when a band holds more than kBandMax rows, two rows have equal keys or a row has the padding's key: the
// bitonic network then gives those rows the order that it gives. bins: kSortBins words; list, order: n entries.
// SortFrames of one 1024 x 1024 frame with 2 400 rows: 114 us by the bitonic network (4 096 entries, 78 steps with a barrier
// each), 39 us by bands, 18 us with the rows written by 16 CTAs (4: 23, 8: 19); of 500 such frames 0.35 and 0.17 ms.
__device__ bool BandOrder(const unsigned long long* ky, const unsigned long long* kx, uint32_t n, int H, uint32_t* bins, uint16_t* list,
                          uint16_t* order)
{
	__shared__ uint32_t warpSum[kSortThreads / 32];
	constexpr int kPer = kSmemSort / kSortThreads, kBinsPer = kSortBins / kSortThreads;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int i = threadIdx.x; i < kSortBins; i += kSortThreads) { bins[i] = 0; }
	__syncthreads();
	// the key of y >= 0 is its bits with the sign set; y below 0 and the first NaN go to the first band, all beyond the
	// frame to the last (bands are monotone in the key)
	const double scale = static_cast<double>(kSortBins) / H;
	uint32_t band[kPer], slot[kPer];
	bool other = false;
	#pragma unroll
	for (int u = 0; u < kPer; ++u) {
		const uint32_t i = threadIdx.x + u * kSortThreads;
		if (i >= n) { continue; }
		const unsigned long long k = ky[i];
		const double y = __longlong_as_double(static_cast<long long>(k & 0x7fffffffffffffffull));
		band[u] = (k >> 63) == 0 ? 0u : (y * scale < kSortBins ? static_cast<uint32_t>(y * scale) : kSortBins - 1u);
		slot[u] = atomicAdd(bins + band[u], 1u);
		other |= slot[u] >= kBandMax || (k == ~0ull && kx[i] == ~0ull);
	}
	if (__syncthreads_or(other)) { return false; }
	// exclusive prefix of the bands
	uint32_t c[kBinsPer], sum = 0;
	#pragma unroll
	for (int u = 0; u < kBinsPer; ++u) {
		c[u] = sum;
		sum += bins[threadIdx.x * kBinsPer + u];
	}
	uint32_t upTo = sum;
	#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t t = __shfl_up_sync(0xffffffffu, upTo, d);
		if (lane >= d) { upTo += t; }
	}
	if (lane == 31) { warpSum[warp] = upTo; }
	__syncthreads();
	uint32_t before = upTo - sum;
	for (int w = 0; w < warp; ++w) { before += warpSum[w]; }
	#pragma unroll
	for (int u = 0; u < kBinsPer; ++u) { bins[threadIdx.x * kBinsPer + u] = before + c[u]; }
	__syncthreads();
	#pragma unroll
	for (int u = 0; u < kPer; ++u) {
		const uint32_t i = threadIdx.x + u * kSortThreads;
		if (i < n) { list[bins[band[u]] + slot[u]] = static_cast<uint16_t>(i); }
	}
	__syncthreads();
	bool tie = false;
	#pragma unroll
	for (int u = 0; u < kPer; ++u) {
		const uint32_t i = threadIdx.x + u * kSortThreads;
		if (i >= n) { continue; }
		const uint32_t b0 = bins[band[u]], b1 = band[u] + 1 < kSortBins ? bins[band[u] + 1] : n;
		uint32_t rank = b0;
		for (uint32_t b = b0; b < b1; ++b) {
			const uint32_t j = list[b];
			rank += KeyLess(ky[j], kx[j], ky[i], kx[i]) ? 1u : 0u;
			tie |= j != i && ky[j] == ky[i] && kx[j] == kx[i];
		}
		order[rank] = static_cast<uint16_t>(i);
	}
	return !__syncthreads_or(tie);
}

// Sorts each frame's rows by (Y, X) and writes them numbered to out (device memory). gridDim.y CTAs per frame order the
// same rows and write a share of them each; a frame that outgrows shared memory is left to the first. Ids continue from
// *rowBase (rows written by earlier chunks); with offsetOut the rows also land at out + *rowBase rows. The last CTA to
// finish adds the chunk's rows to *rowBase.
__global__ void __launch_bounds__(kSortThreads) SortFrames(Workspace ws, double* out, unsigned long long* rowBase,
                                                            int offsetOut, unsigned long long planeBase, uint32_t capScratch)
{
	extern __shared__ __align__(16) unsigned long long sortSmem[];
	unsigned long long* sy = sortSmem;
	unsigned long long* sx = sy + kSmemSort;
	uint32_t* si = reinterpret_cast<uint32_t*>(sx + kSmemSort);
	uint32_t* bins = si + kSmemSort;
	const int f = blockIdx.x;
	const uint32_t base = ws.frameOutBase[f];
	const uint32_t n = ws.frameOutBase[f + 1] - base;
	// every CTA has read *rowBase when the last one is counted
	const unsigned long long idBase = *rowBase;
	auto finished = [&]() {
		__syncthreads();
		if (threadIdx.x == 0) {
			__threadfence();
			if (atomicAdd(&ws.cnt->sorted, 1u) + 1u == gridDim.x * gridDim.y) { *rowBase = idBase + ws.frameOutBase[ws.g.B]; }
		}
	};
	if (n == 0 || (n > static_cast<uint32_t>(kSmemSort) && blockIdx.y > 0)) {
		finished();
		return;
	}
	const uint32_t parts = n > static_cast<uint32_t>(kSmemSort) ? 1u : gridDim.y;
	uint32_t len = 1;
	while (len < n) { len <<= 1; }
	const double* __restrict__ rows = ws.rows + static_cast<long long>(base) * kCols;
	unsigned long long *ky, *kx;
	uint32_t* id;
	const bool smem = len <= static_cast<uint32_t>(kSmemSort);
	if (smem) { ky = sy; kx = sx; id = si; }
	else {
		// global scratch of this frame: 2 * len keys from 4 * base and len indices from 2 * base (len < 2 n, so frames
		// never overlap; the key scratch holds 4 * capRows and the index scratch 2 * capRows entries)
		if (4ull * base + 2ull * len > 4ull * capScratch) {
			finished();
			return;
		}
		ky = reinterpret_cast<unsigned long long*>(ws.sortKey) + 4ull * base;
		kx = ky + len;
		id = ws.sortIdx + 2ull * base;
	}
	// keys: four rows per thread and pass, their loads issued before any key is stored
	for (uint32_t i0 = threadIdx.x; i0 < len; i0 += 4 * blockDim.x) {
		double y[4], x[4];
		#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const uint32_t i = i0 + u * blockDim.x;
			y[u] = x[u] = 0.0;
			if (i < n) {
				y[u] = __ldg(rows + static_cast<long long>(i) * kCols + cY);
				x[u] = __ldg(rows + static_cast<long long>(i) * kCols + cX);
			}
		}
		#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const uint32_t i = i0 + u * blockDim.x;
			if (i < len) {
				ky[i] = i < n ? WeakKey(y[u]) : ~0ull;
				kx[i] = i < n ? WeakKey(x[u]) : ~0ull;
				id[i] = i;
			}
		}
	}
	__syncthreads();
	// list and order share the words of the bitonic network's indices, which are written again when it has to be used
	uint16_t* order = reinterpret_cast<uint16_t*>(si) + kSmemSort;
	const bool banded = smem && BandOrder(ky, kx, n, ws.g.H, bins, reinterpret_cast<uint16_t*>(si), order);
	if (smem && !banded) {
		for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) { id[i] = i; }
		__syncthreads();
		Bitonic<true>(ky, kx, id, len);
	}
	else if (!smem) { Bitonic<false>(ky, kx, id, len); }
	double* __restrict__ dst = out + (offsetOut ? static_cast<long long>(idBase) * kCols : 0ll) + static_cast<long long>(base) * kCols;
	// numbered rows in sorted order, element by element (consecutive threads: consecutive columns of a row, then the
	// next row), four elements per thread and pass with their loads issued first
	const double plane = static_cast<double>(planeBase + f + 1);
	const uint32_t total = static_cast<uint32_t>(static_cast<unsigned long long>(n) * (blockIdx.y + 1) / parts) * kCols;
	const uint32_t begin = static_cast<uint32_t>(static_cast<unsigned long long>(n) * blockIdx.y / parts) * kCols;
	for (uint32_t e0 = begin + threadIdx.x; e0 < total; e0 += 4 * blockDim.x) {
		double v[4];
		#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const uint32_t e = e0 + u * blockDim.x;
			v[u] = 0.0;
			if (e < total) {
				const uint32_t i = e / kCols, c = e - i * kCols;
				v[u] = __ldg(rows + static_cast<long long>(banded ? order[i] : id[i]) * kCols + c);
			}
		}
		#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const uint32_t e = e0 + u * blockDim.x;
			if (e < total) {
				const uint32_t i = e / kCols, c = e - i * kCols;
				dst[e] = c == cId ? static_cast<double>(idBase + base + i + 1) : c == cPlane ? plane : c == cIndex ? static_cast<double>(i + 1) : v[u];
			}
		}
	}
	finished();
}

}  // namespace

bool LaunchBuildCandidates(const Workspace& ws, cudaStream_t st)
{
	const int blocks = static_cast<int>(std::min<uint32_t>(148 * 4, (ws.capRows + 255) / 256));
	const bool ok = LaunchChained(BuildCandidates, blocks, 256, 0, st, ws);
	CountLaunch();
	return ok;
}

// out: device destination of the rows. rowBase: device count of the rows written by earlier chunks (Ids continue
// from it; it is advanced by this chunk's rows); offsetOut: write at out + rowBase rows instead of out.
bool LaunchSortFrames(const Workspace& ws, double* out, unsigned long long* rowBase, bool offsetOut, unsigned long long planeBase,
                      cudaStream_t st)
{
	static std::atomic<uint64_t> devices{0};
	if (!AllowSmemOnDevice(reinterpret_cast<const void*>(SortFrames), kSortSmemBytes, devices)) { return false; }
	// with few frames several CTAs order and write each of them, up to the number of SMs (BandOrder has the measurements)
	const int parts = std::max(1, std::min(16, 148 / std::max(1, ws.g.B)));
	SortFrames<<<dim3(ws.g.B, parts), kSortThreads, kSortSmemBytes, st>>>(ws, out, rowBase, offsetOut ? 1 : 0, planeBase, ws.capRows);
	CountLaunch();
	return PTB_LAUNCHED();
}

}  // namespace ptb
