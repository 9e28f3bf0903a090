// Runs the segmentation of a chunk of frames on the CPU (each CUDA thread a host thread) in the library's
// launch order: per-component floods with both exactness tests and the re-flood, basin fusion, the frame-wide flood by a
// warp, region sums and the frames' offsets, with the library's prefix sums. Every device array is a separate
// allocation for AddressSanitizer. Test harness only.
// Usage: frame_emu order <seeds> <pixels> <first pixel> checks and times the order of a frame's seeds; frame_emu scan
// <entries> <capacity> <CTAs> and frame_emu lookback <tile> <prefix> <missing> check the prefix sums;
// frame_emu <in> <out> [warps [points per frame]]; in: int32 H, W, B, mode, int64 threshold (2^-16 units), double fusion ratio,
// B * H * W int64 W1 values (2^-16 units); warps: warps per block of the kernels that give a warp a group (0: as the
// library). out: B * H * W uint32 labels, B * H * W code bytes, B + 1 uint32 output offsets, then 7 uint32 (routed,
// rank-tested, re-flooded, groups fused in global memory, fits, fault, multi-label groups).
// PTB_UNORDERED: warp collectives that order no memory (for ThreadSanitizer); otherwise on barriers, which is faster.
#if defined(PTB_UNORDERED)
#include "warp_shim.h"
#else
#include "shim.h"
#endif

thread_local uint3 threadIdx;
thread_local uint3 blockIdx;
dim3 blockDim;
dim3 gridDim;
namespace emu {
std::barrier<>* blockBar;
std::vector<std::unique_ptr<std::barrier<>>> warpBar;
uint64_t xbuf[1024];
#if defined(PTB_UNORDERED)
Slot slots[2][1024];
thread_local uint32_t collectives;
#endif
}  // namespace emu

#include "scan_emu.inc"
#include "frame_emu.inc"

#include <chrono>
#include <cstdio>
#include <cstdlib>

namespace ptb {
void SetError(const std::string& m) { fprintf(stderr, "SetError %s\n", m.c_str()); }
bool CheckCuda(cudaError_t, const char*, const char*, int) { return true; }
void CountLaunch(uint64_t) {}

template <class T> static T* Alloc(size_t n)
{
	T* p = static_cast<T*>(malloc(std::max<size_t>(n, 1) * sizeof(T)));
	memset(static_cast<void*>(p), 0xAB, std::max<size_t>(n, 1) * sizeof(T));  // garbage, like uninitialised device memory
	return p;
}
}  // namespace ptb

using namespace ptb;

namespace {

// Each block's collectives are tagged from a number of its own (a launch has fewer than 256 blocks), so that a block's
// threads take no value left by another's.
template <class K, class... A> void Run(dim3 grid, int threads, K kernel, A... args)
{
#if defined(PTB_UNORDERED)
	memset(static_cast<void*>(emu::slots), 0, sizeof emu::slots);
#endif
	emu::Launch(grid, dim3(threads), [=]() {
#if defined(PTB_UNORDERED)
		emu::collectives = (blockIdx.y * grid.x + blockIdx.x) << 24;
#endif
		kernel(args...);
	});
}

// ExclusiveScans' launch.
void Scan(std::initializer_list<ScanJob> jobs, unsigned* fault)
{
	Scans s{};
	int k = 0;
	std::vector<unsigned long long*> states;
	for (const ScanJob& j : jobs) {
		s.job[k] = j;
		s.state[k] = Alloc<unsigned long long>(ScanStateWords(j.cap));
		memset(s.state[k], 0, ScanStateWords(j.cap) * sizeof(unsigned long long));
		states.push_back(s.state[k++]);
	}
	s.fault = fault;
	Run(dim3(2, k), kScanThreads, ScanKernel, s);
	for (auto* p : states) { free(p); }
}

void OrderKernel(const uint32_t* seeds, uint32_t n, uint32_t base, unsigned long long N, uint32_t* sorted)
{
	static uint32_t count[kSeedBuckets];
	OrderSeeds(seeds, n, base, N, sorted, count);
}

// `n` seeds of a frame of N pixels that starts at pixel `base`, in the order of a fixed shuffle: 0 when they come out
// ascending. Prints the milliseconds it took.
int OrderCheck(uint32_t n, unsigned long long N, uint32_t base)
{
	std::vector<uint32_t> want(n);
	for (uint32_t i = 0; i < n; ++i) { want[i] = base + static_cast<uint32_t>(i * N / n); }  // distinct for n <= N
	uint32_t* seeds = Alloc<uint32_t>(n);
	uint32_t* sorted = Alloc<uint32_t>(n);
	std::copy(want.begin(), want.end(), seeds);
	unsigned long long r = 88172645463325252ull;
	for (uint32_t i = n; i > 1; --i) {
		r ^= r << 13; r ^= r >> 7; r ^= r << 17;
		std::swap(seeds[i - 1], seeds[r % i]);
	}
	const auto t0 = std::chrono::steady_clock::now();
	Run(dim3(1), 32, OrderKernel, static_cast<const uint32_t*>(seeds), n, base, N, sorted);
	printf("%.3f\n", std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
	return std::equal(want.begin(), want.end(), sorted) ? 0 : 1;
}

// Prefix sums of n entries counted on the device (capacity cap), by the given number of CTAs: 0 when they are right.
int ScanCheck(uint32_t n, uint32_t cap, uint32_t blocks)
{
	const uint32_t held = std::min(n, cap);
	uint32_t* data = Alloc<uint32_t>(cap + 1);
	uint32_t* count = Alloc<uint32_t>(1);
	unsigned long long* state = Alloc<unsigned long long>(ScanStateWords(cap));
	std::vector<uint32_t> want(held + 1, 0);
	for (uint32_t i = 0; i < held; ++i) {
		data[i] = (i * 2654435761u) >> 20;
		want[i + 1] = want[i] + data[i];
	}
	memset(state, 0, ScanStateWords(cap) * sizeof(unsigned long long));
	*count = n;
	Scans s{};
	uint32_t total = 0, fault = 0;
	s.job[0] = ScanJob{data, count, 0, cap, &total};
	s.state[0] = state;
	s.fault = &fault;
	Run(dim3(blocks, 1), kScanThreads, ScanKernel, s);
	return fault == 0 && total == want[held] && std::equal(want.begin(), want.end(), data) ? 0 : 1;
}

void LookBackKernel(unsigned long long* tiles, uint32_t tile, uint32_t* fault, uint32_t* sum)
{
	const uint32_t s = LookBack(tiles, tile, fault);
	if (threadIdx.x == 0) { *sum = s; }
}

// The sum before `tile` from its predecessors' states: sums from `prefix` on, where a whole prefix is published (-1:
// nowhere), and with `missing` (-1: none) not published at all, which the bounded wait has to report.
int LookBackCheck(uint32_t tile, int prefix, int missing)
{
	unsigned long long* tiles = Alloc<unsigned long long>(tile);
	uint32_t want = 0, fault = 0, sum = 0;
	for (uint32_t i = 0; i < tile; ++i) {
		const uint32_t v = 1000 + i * 7;
		tiles[i] = kSum | v;
		if (static_cast<int>(i) == prefix) {
			tiles[i] = kPrefix | 123456u;
			want = 123456u;
		}
		else if (static_cast<int>(i) > prefix) { want += v; }
	}
	if (prefix < 0) { tiles[0] = kPrefix | 1000u; }
	if (missing >= 0) { tiles[missing] = 0; }
	Run(dim3(1), 32, LookBackKernel, tiles, tile, &fault, &sum);
	return missing >= 0 ? (fault == 1 ? 0 : 1) : (fault == 0 && sum == want ? 0 : 1);
}

}  // namespace

int main(int argc, char** argv)
{
	if (argc == 5 && !strcmp(argv[1], "scan")) {
		return ScanCheck(static_cast<uint32_t>(atoll(argv[2])), static_cast<uint32_t>(atoll(argv[3])), static_cast<uint32_t>(atoll(argv[4])));
	}
	if (argc == 5 && !strcmp(argv[1], "lookback")) { return LookBackCheck(static_cast<uint32_t>(atoll(argv[2])), atoi(argv[3]), atoi(argv[4])); }
	if (argc == 5 && !strcmp(argv[1], "order")) {
		return OrderCheck(static_cast<uint32_t>(atoll(argv[2])), static_cast<unsigned long long>(atoll(argv[3])), static_cast<uint32_t>(atoll(argv[4])));
	}
	if (argc < 3) { return 2; }
	const int warps = argc > 3 ? atoi(argv[3]) : 0;
	const uint32_t maxPoints = argc > 4 ? static_cast<uint32_t>(atoi(argv[4])) : 0xffffffffu;
	FILE* fp = fopen(argv[1], "rb");
	int dims[4] = {};
	long long thr = 0;
	double ratio = 0;
	if (!fp || fread(dims, 4, 4, fp) != 4 || fread(&thr, 8, 1, fp) != 1 || fread(&ratio, 8, 1, fp) != 1) { return 1; }
	const int H = dims[0], W = dims[1], B = dims[2], mode = dims[3];
	const size_t N = static_cast<size_t>(H) * W, P = N * B;
	std::vector<long long> w1u(P);
	if (fread(w1u.data(), 8, P, fp) != P) { return 1; }
	fclose(fp);

	Workspace ws{};
	Geometry g{};
	g.H = H; g.W = W; g.B = B; g.words = (W + 31) / 32; g.N = static_cast<long long>(N); g.P = static_cast<long long>(P);
	g.divN = MakeFastDiv(static_cast<uint32_t>(N));
	g.divW = MakeFastDiv(static_cast<uint32_t>(W));
	ws.g = g;
	const uint32_t capComp = static_cast<uint32_t>(((H + 1) / 2) * ((W + 1) / 2) * B + 1);
	ws.capDom = ws.capSeed = static_cast<uint32_t>(P);
	ws.capComp = ws.capRegion = capComp;
	ws.capRows = capComp;
	const uint32_t rows = static_cast<uint32_t>(B) * static_cast<uint32_t>(H), slots = RefloodSlots(g);
	ws.code = Alloc<uint8_t>(P); ws.w1 = Alloc<uint32_t>(P); ws.par = Alloc<uint32_t>(P); ws.lab = Alloc<uint32_t>(P);
	ws.rootmask = Alloc<uint32_t>(rows * static_cast<size_t>(g.words)); ws.rowcnt = Alloc<uint32_t>(rows + 1);
	ws.dom = Alloc<uint32_t>(P); ws.seeds = Alloc<uint32_t>(P);
	for (uint32_t** p : {&ws.compRoot, &ws.compSize, &ws.compNRoot, &ws.compNSeed, &ws.compRegion, &ws.multi, &ws.gReg, &ws.regCount,
	                     &ws.regFrame, &ws.fuMaxPos, &ws.fuWNPos, &ws.fuNeighbour, &ws.fuBecome, &ws.rfGroups}) { *p = Alloc<uint32_t>(capComp); }
	for (uint32_t** p : {&ws.gOff, &ws.gSeedOff, &ws.gRegOff, &ws.gCurPix, &ws.gCurSeed, &ws.gCurReg, &ws.regCand}) { *p = Alloc<uint32_t>(capComp + 1); }
	for (double** p : {&ws.fuMaxWN, &ws.fuMinP, &ws.fuMaxP}) { *p = Alloc<double>(capComp); }
	for (unsigned long long** p : {&ws.regSumVJ, &ws.regSumVI, &ws.regSumV}) { *p = Alloc<unsigned long long>(capComp); }
	ws.fuLocked = Alloc<uint8_t>(capComp);
	ws.gPix = Alloc<uint32_t>(P); ws.gSeed = Alloc<uint32_t>(P);
	ws.heapKey = Alloc<double>(P); ws.heapPix = Alloc<uint32_t>(P);
	for (uint32_t** p : {&ws.frameDom, &ws.frameSeeds, &ws.frameRoute, &ws.frameSuspect, &ws.frameReflood}) {
		*p = Alloc<uint32_t>(B + 1);
		memset(*p, 0, (B + 1) * sizeof(uint32_t));
	}
	for (uint32_t** p : {&ws.frameRegBase, &ws.frameCandBase, &ws.frameKeep, &ws.frameOutBase}) { *p = Alloc<uint32_t>(B + 1); }
	ws.rfVals = Alloc<uint32_t>(static_cast<size_t>(slots) * 2 * kRefloodCap);
	ws.rfGrp = Alloc<uint32_t>(static_cast<size_t>(slots) * 2 * kRefloodCap);
	ws.rfOff = Alloc<uint32_t>(static_cast<size_t>(slots) * 2 * (kRefloodBuckets + 1));
	ws.rfInfo = Alloc<uint32_t>(kRefloodSlots * 8);
	ws.rfPix = Alloc<uint32_t>(slots * N * kRfWords);
	ws.suspect = Alloc<uint4>(kSuspectCap); ws.capSuspect = kSuspectCap;
	ws.rankOrder = Alloc<uint32_t>(kSuspectCap); ws.rankSlotOff = Alloc<uint32_t>(kRankSlots + 1);
	ws.rankCount = Alloc<uint32_t>(2 * kSuspectCap);
	ws.candRegion = Alloc<uint32_t>(ws.capRows); ws.candFrame = Alloc<uint32_t>(ws.capRows);
	ws.cnt = Alloc<Counters>(1);
	memset(ws.cnt, 0, sizeof(Counters));
	memset(ws.rootmask, 0, sizeof(uint32_t) * rows * g.words);

	// the detection kernel's outputs
	auto v0 = [&](int f, int y, int x) -> long long {
		return (y < 0 || y >= H || x < 0 || x >= W) ? 0 : std::max(0ll, w1u[f * N + static_cast<size_t>(y) * W + x]);
	};
	for (int f = 0; f < B; ++f) {
		for (int y = 0; y < H; ++y) {
			for (int x = 0; x < W; ++x) {
				const size_t p = f * N + static_cast<size_t>(y) * W + x;
				const long long v = v0(f, y, x);
				const bool dom = v > thr && v > 0;
				long long m = 0;
				for (int t = 0; t < 9; ++t) { m = std::max(m, v0(f, y + t / 3 - 1, x + t % 3 - 1)); }
				const bool seed = dom && v >= m;
				ws.code[p] = static_cast<uint8_t>((dom ? kDomain : 0) | (seed ? kSeed : 0));
				if (dom) {
					ws.w1[p] = static_cast<uint32_t>(v);
					ws.dom[ws.cnt->ndom++] = static_cast<uint32_t>(p);
					++ws.frameDom[f];
				}
				if (seed) {
					ws.seeds[ws.cnt->nseed++] = static_cast<uint32_t>(p);
					++ws.frameSeeds[f];
				}
			}
		}
	}

	const dim3 one(1), two(2);
	const int boxThreads = 32 * (warps ? warps : kBoxWarps), fuseThreads = 32 * (warps ? warps : kFuseWarps),
	          rfThreads = 32 * (warps ? warps : kRfWarps);
	Run(two, 128, CclInit, ws);
	Run(two, 128, CclUnion, ws);
	Run(one, 256, CompEnumerate, ws);
	Run(two, 128, CompCount, ws);
	Run(two, 128, SeedParent, ws);
	Run(two, 128, RowCount, ws);
	Scan({{ws.rowcnt, nullptr, rows, rows, &ws.cnt->nregion}}, &ws.cnt->fault);
	Run(two, 128, SeedLabel, ws);
	const int rank = mode == 0 ? 1 : 0;
	const bool strict = mode == 1, fuse = static_cast<int>(ratio) > 0;
	const uint32_t frames = static_cast<uint32_t>(B), groupsStrict = strict ? frames : 0u;
	if (strict) {
		for (uint32_t* list : {ws.gOff, ws.gSeedOff, ws.gRegOff, ws.gCurPix, ws.gCurSeed, ws.gCurReg}) { memset(list, 0, sizeof(uint32_t) * (B + 1)); }
		Run(two, 128, GroupSizesStrict, ws);
		Scan({{ws.gOff, nullptr, frames, ws.capComp, nullptr}, {ws.gSeedOff, nullptr, frames, ws.capComp, nullptr},
		      {ws.gRegOff, nullptr, frames, ws.capComp, nullptr}}, &ws.cnt->fault);
	}
	else {
		Run(two, 128, GroupEnumerate, ws);
		Scan({{ws.gOff, &ws.cnt->nmulti, 0, ws.capComp, nullptr}, {ws.gSeedOff, &ws.cnt->nmulti, 0, ws.capComp, nullptr},
		      {ws.gRegOff, &ws.cnt->nmulti, 0, ws.capComp, nullptr}}, &ws.cnt->fault);
	}
	Run(two, 128, GroupScatter, ws, strict ? 1 : 0);
	if (strict) { Run(one, 32, FrameFlood, ws, 0); }
	else { Run(two, boxThreads, GroupFloodBox, ws, rank); }
	if (rank) {
		Run(one, kPlanThreads, SuspectPlan, ws);
		Run(two, 128, SuspectCount, ws);
		Run(two, 128, SuspectCheck, ws, 0);
		Run(one, kPlanThreads, RefloodPlan, ws);
		Run(two, 128, RefloodGather, ws);
		Run(dim3(slots * 2), kRfBucketThreads, RefloodBucket, ws);
		Run(two, 128, RefloodCounts, ws);
		Run(two, rfThreads, RefloodBox, ws);
	}
	if (fuse) {
		if (!strict) { Run(two, fuseThreads, GroupFuseBox, ws, ratio); }
		Run(one, kFloodThreads, GroupFuse, ws, groupsStrict, ratio, 0);
	}
	const uint32_t fusedGlobal = ws.cnt->nfuse, routed = ws.cnt->nroute;
	if (!strict) {
		Run(one, kRedoThreads, RedoOffsets, ws);
		Run(two, 128, GroupScatter, ws, 2);
		Run(two, 32, FrameFlood, ws, 1);
		if (fuse) { Run(one, kFloodThreads, GroupFuse, ws, frames, ratio, 1); }
	}
	Run(two, 128, RegionStats, ws);
	Run(two, 128, CandidateFlags, ws);
	Scan({{ws.regCand, &ws.cnt->nregion, 0, ws.capRegion, &ws.cnt->ncand}}, &ws.cnt->fault);
	Run(one, kOffsetThreads, FrameOffsets, ws, maxPoints);
	Run(two, 128, CandidateEmit, ws, maxPoints);
	FILE* lf = fopen(argv[2], "wb");
	fwrite(ws.lab, sizeof(uint32_t), P, lf);
	fwrite(ws.code, 1, P, lf);
	fwrite(ws.frameOutBase, sizeof(uint32_t), B + 1, lf);
	const uint32_t st[7] = {routed, ws.cnt->nslots, ws.cnt->nreflood, fusedGlobal, ws.cnt->nfit, ws.cnt->fault, ws.cnt->nmulti};
	fwrite(st, sizeof(uint32_t), 7, lf);
	fclose(lf);
	return 0;
}
