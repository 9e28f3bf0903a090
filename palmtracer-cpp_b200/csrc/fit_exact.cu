// Gaussian least-squares LM fits (modes 1-4) in FP64 with the reference's exact order of operations. This file is
// compiled with -fmad=false: every product and sum is rounded on its own, as in the reference built with
// -ffp-contract=off, so each ROI follows the reference's iteration path decision for decision; results differ from
// the reference only where CUDA's exp / sin / cos round differently from the host C library in the last place.
//
// Reference: lib/fit/GaussianFit.cpp:48-295, lib/fit/GaussianModel.cpp:19-52, lib/fit/Fitting.cpp:61-175,
// lib/signal_processing/Matrix.cpp:297-355.
//
// Two launches: ExactFitKernel iterates (parameters and a status are left in the output row), ExactFinalKernel forms
// the squared correlation and writes the row. Both come in two mappings of ROIs to lanes, chosen by the number of
// ROIs (LaunchExactFit); every pass of the persistent loop evaluates each busy ROI's model, error, gradient and
// curvature sums once, at its start point or at a trial point. The reference evaluates the error alone at a trial
// point and everything again at the same point once it is accepted: the same numbers, so they are formed once here.
//   * L = 1, a thread per ROI (many ROIs: FP64-issue-bound). The accumulators are the thread's registers, summed in
//     pixel order by construction; the state of the last accepted point is kept in shared memory, interleaved by
//     thread. A thread whose ROI ends takes the next one from a queue, so no lane idles on the others' iterations.
//   * L = 8 or 32, a group of lanes per ROI (few ROIs: bound by the latency of one ROI's serial iterations). The
//     lanes share the pixels and stage gradient and residual in shared memory; each accumulator is then owned by one
//     lane, which forms its products and adds them in pixel order; the damped matrix is inverted column-parallel.
// Bound: FP64 issue and, with few ROIs, the latency of dependent FP64 operations (8 cycles an operation, 114 a division).
// Before (one warp per ROI with shuffled solves and one summing lane per accumulator, all sizes) 365 738 ROIs of
// 7 x 7 in mode 2 took 25.3 ms; now 3.5 ms.
//
// Order of operations: every element of the inverse goes through exactly the reference's Gauss-Jordan operations
// (equilibration, partial pivoting, row normalisation, elimination), whose results do not depend on the order across
// columns: the columns of the matrix are eliminated first, keeping each step's multipliers in place of the column it
// cleared, and the columns of the inverse are then replayed one after the other and dotted with beta, j ascending.
#include <algorithm>

#include "pt_common.cuh"

namespace ptb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kThreads = 64;
constexpr uint32_t kNoRoi = 0xffffffffu;
constexpr int kStageUnit = 8;  // staged pixels come in whole units (the longest batch of the summing lanes)
// ExactFitKernel's hand-over in the output row: parameters in columns 0..6, this status in column kStatusCol.
constexpr int kStatusCol = 8;
constexpr double kStFitted = 1.0, kStSentinel = 0.0;

template <int MODE> struct NpOf;
template <> struct NpOf<kG2Fixed> { static constexpr int v = 4; };
template <> struct NpOf<kG2Sigma> { static constexpr int v = 5; };
template <> struct NpOf<kG3Fixed> { static constexpr int v = 6; };
template <> struct NpOf<kG3Theta> { static constexpr int v = 7; };

// Sums of one evaluation: error, gradient (NP), curvature (upper triangle, row major).
template <int MODE> struct SumsOf { static constexpr int v = 1 + NpOf<MODE>::v + NpOf<MODE>::v * (NpOf<MODE>::v + 1) / 2; };

// ---- Division by a divisor shared by many dividends ---------------------------------------------------------------
// The correctly rounded quotient a / b from the correctly rounded reciprocal y of b with fused multiply-adds
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990): a first correction
// brings a * y within one unit in the last place, and the correction of such a quotient with a correctly rounded
// reciprocal is the correctly rounded one. 5 operations; valid while no intermediate leaves the normal range: for
// divisors in [2^-60, 2^60) (Safe) and dividends that are zero or have magnitudes in [2^-960, 2^300). (A zero keeps
// its value but not its sign, which no sum here can tell.) Other operands are divided plainly.
__device__ __forceinline__ unsigned HighWord(double a) { return static_cast<unsigned>(__double2hiint(a)) & 0x7fffffffu; }
constexpr unsigned HighOfPow2(int e) { return static_cast<unsigned>(1023 + e) << 20; }
__device__ __forceinline__ bool Safe(double a) { return HighWord(a) - HighOfPow2(-60) < HighOfPow2(60) - HighOfPow2(-60); }
// Zero, or a magnitude of at least 2^E.
template <int E> __device__ __forceinline__ bool ZeroOrAbove(double a) { return a == 0.0 || HighWord(a) >= HighOfPow2(E); }

struct Divisor {
	double b, y;
	__device__ __forceinline__ void Set(double v) { b = v; y = 1.0 / v; }
	__device__ __forceinline__ double Quick(double a) const
	{
		const double q = a * y;
		const double q1 = __fma_rn(__fma_rn(-q, b, a), y, q);
		return __fma_rn(__fma_rn(-q1, b, a), y, q1);
	}
};

template <int MODE>
struct GModel {
	double off, amp, c, s, c2, s2, cs;
	Divisor sx, sy, sx2, sy2, sx3, sy3, twoSx2;
	bool quick;  // the quick division serves every dividend formed from these parameters

	__device__ void Make(const double* p, double sigma, double theta)
	{
		off = p[0];
		amp = p[1];
		// a pixel distance X - p[2] is then zero or at least 2^-60: X is a whole number
		quick = ZeroOrAbove<-60>(p[2]) && ZeroOrAbove<-60>(p[3]);
		if constexpr (MODE == kG2Fixed || MODE == kG2Sigma) {
			const double w = MODE == kG2Fixed ? sigma : p[4];
			sx2.Set(w * w);
			twoSx2.b = 2 * sx2.b;
			twoSx2.y = 0.5 * sx2.y;
			if constexpr (MODE == kG2Sigma) { sx3.Set(w * sx2.b); }
			quick = quick && Safe(w) && Safe(sx2.b) && (MODE == kG2Fixed || Safe(sx3.b)) && ZeroOrAbove<-40>(amp);
		}
		else {
			const double th = MODE == kG3Fixed ? theta : p[6];
			sx.Set(p[4]);
			sy.Set(p[5]);
			sx2.Set(p[4] * p[4]);
			sy2.Set(p[5] * p[5]);
			sx3.Set(p[4] * sx2.b);
			sy3.Set(p[5] * sy2.b);
			c = cos(th);
			s = sin(th);
			c2 = c * c;
			s2 = s * s;
			cs = c * s;
			// the dividends are sums of products of distances with these: zero or far above 2^-960
			quick = quick && Safe(sx.b) && Safe(sy.b) && Safe(sx2.b) && Safe(sy2.b) && Safe(sx3.b) && Safe(sy3.b) &&
			        ZeroOrAbove<-150>(c) && ZeroOrAbove<-150>(s) && ZeroOrAbove<-300>(cs);
		}
	}

	template <bool GRAD, bool QUICK>
	__device__ __forceinline__ double Form(double x, double y, double* g, double& e) const
	{
		auto div = [](double a, const Divisor& d) {
			if constexpr (QUICK) { return d.Quick(a); }
			else { return a / d.b; }
		};
		const double X2 = x * x, Y2 = y * y;
		if constexpr (MODE == kG2Fixed || MODE == kG2Sigma) {
			const double r2 = X2 + Y2;
			e = exp(div(-r2, twoSx2));
			const double P = amp * e;
			if constexpr (GRAD) {
				g[0] = 1;
				g[1] = e;
				g[2] = div(P * x, sx2);
				g[3] = div(P * y, sx2);
				if constexpr (MODE == kG2Sigma) { g[4] = div(P, sx3) * r2; }
			}
			return P + off;
		}
		else {
			const double xc = x * c, xs = x * s, yc = y * c, ys = y * s;
			const double f1 = div(xc - ys, sx), f2 = div(xs + yc, sy);
			e = exp(-((f1 * f1) + (f2 * f2)));
			const double P = amp * e;
			if constexpr (GRAD) {
				const double xy = x * y, f3 = 2 * xy * cs;
				g[0] = 1;
				g[1] = e;
				g[2] = P * (-div((-2 * c2 * x) + (2 * y * cs), sx2) - div((-2 * s2 * x) - (2 * y * cs), sy2));
				g[3] = P * (div((2 * s2 * y) - (2 * x * cs), sx2) - div((-2 * c2 * y) - (2 * x * cs), sy2));
				g[4] = P * div(2 * ((xc * xc) - f3 + (ys * ys)), sx3);
				g[5] = P * div(2 * ((xs * xs) + f3 + (yc * yc)), sy3);
				if constexpr (MODE == kG3Theta) {
					const double f4 = div(2 * xy, sx2) - div(2 * xy, sy2);
					g[6] = P * ((2 * cs * (div(X2 - Y2, sx2) + div(Y2 - X2, sy2))) - (s2 * f4) + (c2 * f4));
				}
			}
			return P + off;
		}
	}

	// Model values v and gradients g of B pixels, evaluated side by side: one evaluation is a chain of dependent
	// operations several hundred cycles long.
	template <bool GRAD, int B>
	__device__ __forceinline__ void Eval(const double (&x)[B], const double (&y)[B], double (&v)[B], double (*g)[NpOf<MODE>::v]) const
	{
		double e[B];
		#pragma unroll
		for (int b = 0; b < B; ++b) { v[b] = Form<GRAD, true>(x[b], y[b], GRAD ? g[b] : nullptr, e[b]); }
		bool again = !quick;
		if constexpr (MODE == kG2Fixed || MODE == kG2Sigma) {
			// these modes divide amp * e * distance: with e zero or at least 2^-860 it is zero or at least 2^-960
			#pragma unroll
			for (int b = 0; b < B; ++b) { again = again || (HighWord(e[b]) < HighOfPow2(-860) && e[b] != 0.0); }
		}
		if (again) {
			#pragma unroll
			for (int b = 0; b < B; ++b) { v[b] = Form<GRAD, false>(x[b], y[b], GRAD ? g[b] : nullptr, e[b]); }
		}
	}
};

// Exact conversion of a pixel value (below 2^32) to double.
__device__ __forceinline__ double ToDouble(uint32_t v) { return __hiloint2double(0x43300000, static_cast<int>(v)) - 4503599627370496.0; }

struct Roi {
	const uint16_t* base;
	int W, roi, n;
	double X0, Y0;  // frame coordinates of the first pixel
};

// Row i and column j of a pixel visited in steps of a fixed stride over the ROI's raster order; past the last pixel
// it stays inside the ROI's rows (its value is not used).
struct Cursor {
	int i, j;
	__device__ __forceinline__ void Set(int k, int roi) { i = k / roi; j = k - i * roi; }
	__device__ __forceinline__ void Step(int di, int dj, int roi)
	{
		i += di;
		j += dj;
		if (j >= roi) { j -= roi; ++i; }
	}
	__device__ __forceinline__ double Value(const Roi& R, double& X, double& Y) const
	{
		const int r = min(i, R.roi - 1);
		X = R.X0 + ToDouble(static_cast<uint32_t>(j));
		Y = R.Y0 + ToDouble(static_cast<uint32_t>(r));
		return ToDouble(__ldg(R.base + static_cast<long long>(r) * R.W + j));
	}
};

// False when the ROI crosses the frame border (the reference's test, Fitting.cpp).
__device__ __forceinline__ bool LocateRoi(const uint16_t* frame, int H, int W, const FitParams& fp, const Cand& cd, Roi& R)
{
	const bool nonneg = cd.x >= 0.0 && cd.y >= 0.0;
	const unsigned long long ux = nonneg ? static_cast<unsigned long long>(cd.x) : 0ull;
	const unsigned long long uy = nonneg ? static_cast<unsigned long long>(cd.y) : 0ull;
	const unsigned long long h = static_cast<unsigned long long>(fp.half);
	if (!nonneg || !RoiInside(ux, uy, fp.half, H, W)) { return false; }
	R.base = frame + static_cast<long long>(uy - h) * W + static_cast<long long>(ux - h);
	R.W = W;
	R.roi = fp.roi;
	R.n = fp.n;
	R.X0 = static_cast<double>(ux - h);
	R.Y0 = static_cast<double>(uy - h);
	return true;
}

template <int NP>
__device__ __forceinline__ int U(int a, int b) { return a <= b ? a * NP - (a * (a - 1)) / 2 + (b - a) : b * NP - (b * (b - 1)) / 2 + (a - b); }

template <int MODE>
__device__ __forceinline__ void Bounds(double x, double y, double (&lo)[NpOf<MODE>::v], double (&hi)[NpOf<MODE>::v])
{
	lo[0] = 0; lo[1] = 0; lo[2] = x - 1; lo[3] = y - 1;
	hi[0] = 65535; hi[1] = 65535; hi[2] = x + 1; hi[3] = y + 1;
	if constexpr (MODE == kG2Sigma) { lo[4] = 0.1; hi[4] = 20; }
	if constexpr (MODE == kG3Fixed || MODE == kG3Theta) { lo[4] = lo[5] = 0.1; hi[4] = hi[5] = 20; }
	if constexpr (MODE == kG3Theta) { lo[6] = -150; hi[6] = 150; }
}

// The theta derivative is dropped for a circular model (GaussianFit.cpp).
template <int MODE>
__device__ __forceinline__ bool Circular(const double* p)
{
	if constexpr (MODE == kG3Theta) { return fabs(p[4] - p[5]) <= 2.220446049250313e-16; }
	else { return false; }
}

template <int L>
__device__ __forceinline__ unsigned GroupMask()
{
	if constexpr (L >= 32) { return kFull; }
	else { return ((1u << L) - 1u) << ((threadIdx.x & 31) & ~(L - 1)); }
}

// ---- Shared memory of one ROI -------------------------------------------------------------------------------------
// Sums (error, beta, alpha) and parameters of the last accepted point, at s[q * stride]; for a group also the sums of
// the newest evaluation and the staged gradient and residual rows ([NP + 1][pitch], 16-byte aligned: pitch is even).
template <int MODE, int L>
struct Slot {
	static constexpr int NP = NpOf<MODE>::v, NT = SumsOf<MODE>::v;
	static constexpr int kHead = (2 * NT + NP + 1) / 2 * 2;
	double* s;
	double* stage;
	int stride, pitch;
	__device__ __forceinline__ Slot(double* smem, int pitchIn)
	{
		pitch = pitchIn;
		if constexpr (L == 1) {
			s = smem + threadIdx.x;
			stride = kThreads;
			stage = nullptr;
		}
		else {
			s = smem + (threadIdx.x / L) * (kHead + (NP + 1) * pitch);
			stride = 1;
			stage = s + kHead;
		}
	}
	__device__ __forceinline__ double& Err() const { return s[0]; }
	__device__ __forceinline__ double& Beta(int a) const { return s[(1 + a) * stride]; }
	__device__ __forceinline__ double& Alpha(int q) const { return s[(1 + NP + q) * stride]; }
	__device__ __forceinline__ double& P(int a) const { return s[(NT + a) * stride]; }
	__device__ __forceinline__ double* New() const { return s + NT + NP; }  // groups only
};

template <int MODE, int L>
size_t SlotBytes(int pitch)
{
	constexpr int NP = NpOf<MODE>::v, NT = SumsOf<MODE>::v;
	return L == 1 ? sizeof(double) * (NT + NP) * kThreads
	              : sizeof(double) * (Slot<MODE, L>::kHead + (NP + 1) * pitch) * (kThreads / L);
}

// Sums of one evaluation at p by one thread, in pixel order: out[0] error, then beta, then alpha. One pixel at a time:
// with many ROIs the issue rate counts, not one evaluation's latency (pixel pairs: 3.82 ms for the 3.49 ms above).
template <int MODE>
__device__ __forceinline__ void SumsThread(const Roi& R, const GModel<MODE>& m, const double* p, double (&out)[SumsOf<MODE>::v])
{
	constexpr int NP = NpOf<MODE>::v, NT = SumsOf<MODE>::v;
	const bool circular = Circular<MODE>(p);
	#pragma unroll
	for (int q = 0; q < NT; ++q) { out[q] = 0.0; }
	const uint16_t* row = R.base;
	double Y = R.Y0;
	for (int i = 0; i < R.roi; ++i, row += R.W, Y += 1.0) {
		const double y[1] = {Y - p[3]};
		double X = R.X0;
		for (int j = 0; j < R.roi; ++j, X += 1.0) {
			double hat[1], g[1][NP];
			const double v = ToDouble(__ldg(row + j));
			const double x[1] = {X - p[2]};
			m.template Eval<true, 1>(x, y, hat, g);
			const double d = v - hat[0];
			if (circular) { g[0][NP - 1] = 0.0; }
			out[0] += d * d;
			#pragma unroll
			for (int a = 0; a < NP; ++a) { out[1 + a] += g[0][a] * d; }
			int q = 1 + NP;
			#pragma unroll
			for (int a = 0; a < NP; ++a) {
				#pragma unroll
				for (int c = a; c < NP; ++c) { out[q++] += g[0][a] * g[0][c]; }
			}
		}
	}
}

// The two staged rows whose product accumulator q sums: rows 0..NP-1 the gradient, row NP the residual.
template <int NP>
__device__ __forceinline__ void SumRows(int q, int& a, int& b)
{
	if (q == 0) { a = b = NP; return; }
	if (q <= NP) { a = q - 1; b = NP; return; }
	int r = q - 1 - NP;
	a = 0;
	while (r >= NP - a) { r -= NP - a; ++a; }
	b = a + r;
}

// The same sums by a group of L lanes, into slot.New(): pixels spread over the lanes, up to pitch - 2 of them staged
// at a time (padded with zeros to whole batches), every accumulator then summed in pixel order by its owner
// (accumulators lane, lane + L, ...): the products of the next batch are formed while the chain of additions runs
// over the current one.
template <int MODE, int L>
__device__ __forceinline__ void SumsGroup(const Slot<MODE, L>& sl, const Roi& R, const GModel<MODE>& m, const double* p)
{
	constexpr int NP = NpOf<MODE>::v, NT = SumsOf<MODE>::v, OWN = (NT + L - 1) / L;
	constexpr int kPairs = L == 32 && OWN == 1 ? 4 : 2;  // pixel pairs per batch
	const unsigned mask = GroupMask<L>();
	const int gl = threadIdx.x & (L - 1);
	const bool circular = Circular<MODE>(p);
	const double2* ra[OWN];
	const double2* rb[OWN];
	double acc[OWN];
	#pragma unroll
	for (int t = 0; t < OWN; ++t) {
		int a, b;
		SumRows<NP>(min(gl + L * t, NT - 1), a, b);
		ra[t] = reinterpret_cast<const double2*>(sl.stage + a * sl.pitch);
		rb[t] = reinterpret_cast<const double2*>(sl.stage + b * sl.pitch);
		acc[t] = 0.0;
	}
	const int room = sl.pitch - 2;
	Cursor at[2];
	at[0].Set(gl, R.roi);
	at[1].Set(gl + L, R.roi);
	const int di = 2 * L / R.roi, dj = 2 * L - di * R.roi;
	for (int c0 = 0; c0 < R.n; c0 += room) {
		const int cnt = min(room, R.n - c0), padded = (cnt + kStageUnit - 1) / kStageUnit * kStageUnit;
		if (c0 > 0) {
			at[0].Set(c0 + gl, R.roi);
			at[1].Set(c0 + gl + L, R.roi);
		}
		for (int k = gl; k < padded; k += 2 * L) {
			double x[2], y[2], v[2], hat[2], g[2][NP];
			#pragma unroll
			for (int b = 0; b < 2; ++b) {
				double X, Y;
				v[b] = at[b].Value(R, X, Y);
				x[b] = X - p[2];
				y[b] = Y - p[3];
				at[b].Step(di, dj, R.roi);
			}
			m.template Eval<true, 2>(x, y, hat, g);
			#pragma unroll
			for (int b = 0; b < 2; ++b) {
				const int kb = k + b * L;
				const bool in = kb < cnt;
				if (circular) { g[b][NP - 1] = 0.0; }
				if (kb < padded) {
					#pragma unroll
					for (int a = 0; a < NP; ++a) { sl.stage[a * sl.pitch + kb] = in ? g[b][a] : 0.0; }
					sl.stage[NP * sl.pitch + kb] = in ? v[b] - hat[b] : 0.0;
				}
			}
		}
		__syncwarp(mask);
		double next[OWN][2 * kPairs];
		auto load = [&](int pair0) {
			#pragma unroll
			for (int u = 0; u < kPairs; ++u) {
				#pragma unroll
				for (int t = 0; t < OWN; ++t) {
					const double2 a = ra[t][pair0 + u], b = rb[t][pair0 + u];
					next[t][2 * u] = a.x * b.x;
					next[t][2 * u + 1] = a.y * b.y;
				}
			}
		};
		load(0);
		for (int pair0 = 0; pair0 < padded / 2; pair0 += kPairs) {
			double now[OWN][2 * kPairs];
			#pragma unroll
			for (int u = 0; u < 2 * kPairs; ++u) {
				#pragma unroll
				for (int t = 0; t < OWN; ++t) { now[t][u] = next[t][u]; }
			}
			if (pair0 + kPairs < padded / 2) { load(pair0 + kPairs); }
			#pragma unroll
			for (int u = 0; u < 2 * kPairs; ++u) {
				#pragma unroll
				for (int t = 0; t < OWN; ++t) { acc[t] += now[t][u]; }
			}
		}
		__syncwarp(mask);
	}
	#pragma unroll
	for (int t = 0; t < OWN; ++t) {
		if (gl + L * t < NT) { sl.New()[gl + L * t] = acc[t]; }
	}
	__syncwarp(mask);
}

// Largest entry of column I in rows [LO, HI), the first of equal ones as in a scan from LO on.
template <int I, int NP, int LO, int HI>
__device__ __forceinline__ void Pivot(const double (&A)[NP][NP], unsigned& piv, double& best)
{
	if constexpr (HI - LO == 1) { piv = LO; best = A[LO][I]; }
	else {
		constexpr int MID = (LO + HI) / 2;
		unsigned p2;
		double b2;
		Pivot<I, NP, LO, MID>(A, piv, best);
		Pivot<I, NP, MID, HI>(A, p2, b2);
		if (fabs(b2) > fabs(best)) { piv = p2; best = b2; }
	}
}

// Step I of the elimination of the matrix's own columns: pivot search and row exchange, then the later columns; the
// step's multipliers stay in column I (the reciprocal pivot in its diagonal entry). Recursive templates: the step
// index has to be a constant for the matrix to stay in registers.
template <int I, int NP>
__device__ __forceinline__ void EliminateStep(double (&A)[NP][NP], double tol, bool& good, unsigned& pivots, unsigned& moved)
{
	if constexpr (I < NP) {
		unsigned piv = I;
		double best = A[I][I];
		Pivot<I, NP, I, NP>(A, piv, best);
		good = good && isfinite(best) && !(fabs(best) <= tol);
		pivots |= piv << (4 * I);
		moved |= piv ^ static_cast<unsigned>(I);
		#pragma unroll
		for (int j = I + 1; j < NP; ++j) {
			if (piv == static_cast<unsigned>(j)) {
				#pragma unroll
				for (int c = I; c < NP; ++c) {
					const double t = A[I][c];
					A[I][c] = A[j][c];
					A[j][c] = t;
				}
			}
		}
		const double pinv = 1.0 / A[I][I];
		A[I][I] = pinv;
		#pragma unroll
		for (int c = I + 1; c < NP; ++c) {
			A[I][c] *= pinv;
			#pragma unroll
			for (int j = 0; j < NP; ++j) {
				if (j != I) { A[j][c] -= A[j][I] * A[I][c]; }
			}
		}
		EliminateStep<I + 1, NP>(A, tol, good, pivots, moved);
	}
}

template <int I, int C, int NP>
__device__ __forceinline__ void ReplayStep(const double (&A)[NP][NP], double (&v)[NP], unsigned pivots, unsigned moved)
{
	if constexpr (I < NP) {
		// without row exchanges the column is zero above its diagonal entry until step C
		if (I >= C || moved) {
			const unsigned piv = (pivots >> (4 * I)) & 15u;
			#pragma unroll
			for (int j = I + 1; j < NP; ++j) {
				if (piv == static_cast<unsigned>(j)) {
					const double t = v[I];
					v[I] = v[j];
					v[j] = t;
				}
			}
			v[I] *= A[I][I];
			#pragma unroll
			for (int j = 0; j < NP; ++j) {
				if (j != I) { v[j] -= A[j][I] * v[I]; }
			}
		}
		ReplayStep<I + 1, C, NP>(A, v, pivots, moved);
	}
}

// Columns C.. of the inverse, each replayed through the recorded steps and added to dp.
template <int C, int MODE, int L>
__device__ __forceinline__ void ReplayColumn(const double (&A)[NpOf<MODE>::v][NpOf<MODE>::v], const double (&scale)[NpOf<MODE>::v],
                                             const Slot<MODE, L>& sl, unsigned pivots, unsigned moved,
                                             double (&dp)[NpOf<MODE>::v], unsigned& high)
{
	constexpr int NP = NpOf<MODE>::v;
	if constexpr (C < NP) {
		double v[NP];
		#pragma unroll
		for (int r = 0; r < NP; ++r) { v[r] = r == C ? scale[C] : 0.0; }
		ReplayStep<0, C, NP>(A, v, pivots, moved);
		const double b = sl.Beta(C);
		#pragma unroll
		for (int i = 0; i < NP; ++i) {
			high = max(high, HighWord(v[i]));
			dp[i] += v[i] * b;
		}
		ReplayColumn<C + 1, MODE, L>(A, scale, sl, pivots, moved, dp, high);
	}
}

// Equilibrated Gauss-Jordan inverse of the damped matrix and dp = inverse * beta in the reference's order
// (Matrix.cpp:297-355, GaussianFit.cpp:85-106), in every lane's registers. Returns false where the reference's
// inversion throws. The lanes of a group solve the same system side by side: with a column per lane every multiplier
// takes two shuffles, more instructions than the whole elimination.
template <int MODE, int L>
__device__ __forceinline__ bool Solve(const Slot<MODE, L>& sl, double lambda, double (&dp)[NpOf<MODE>::v])
{
	constexpr int NP = NpOf<MODE>::v;
	double A[NP][NP], scale[NP];
	unsigned high = 0;
	#pragma unroll
	for (int r = 0; r < NP; ++r) {
		#pragma unroll
		for (int c = r; c < NP; ++c) {
			const double a = sl.Alpha(U<NP>(r, c));
			const double v = r == c ? (a == 0.0 ? 1.0 : (1.0 + lambda) * a) : a;
			high = max(high, HighWord(v));
			A[r][c] = v;
			A[c][r] = v;
		}
	}
	if (high >= 0x7ff00000u) { return false; }  // a non-finite entry
	bool zero = false, safe = true;
	unsigned low = 0xffffffffu;
	Divisor d[NP];
	#pragma unroll
	for (int r = 0; r < NP; ++r) {
		double m = fabs(A[r][0]);
		#pragma unroll
		for (int c = 1; c < NP; ++c) { m = fabs(A[r][c]) > m ? fabs(A[r][c]) : m; }
		#pragma unroll
		for (int c = r; c < NP; ++c) { low = A[r][c] == 0.0 ? low : min(low, HighWord(A[r][c])); }
		zero = zero || m == 0.0;
		safe = safe && Safe(m);
		d[r].Set(m);
		scale[r] = d[r].y;
	}
	if (zero) { return false; }
	if (safe && low >= HighOfPow2(-960)) {
		#pragma unroll
		for (int r = 0; r < NP; ++r) {
			#pragma unroll
			for (int c = 0; c < NP; ++c) { A[r][c] = d[r].Quick(A[r][c]); }
		}
	}
	else {
		#pragma unroll
		for (int r = 0; r < NP; ++r) {
			#pragma unroll
			for (int c = 0; c < NP; ++c) { A[r][c] /= d[r].b; }
		}
	}
	const double tol = 2.220446049250313e-16 * static_cast<double>(NP);
	bool good = true;
	unsigned pivots = 0, moved = 0;  // 4 bits per step: the pivot row; whether any step exchanged rows
	EliminateStep<0, NP>(A, tol, good, pivots, moved);
	if (!good) { return false; }
	#pragma unroll
	for (int i = 0; i < NP; ++i) { dp[i] = 0.0; }
	high = 0;
	ReplayColumn<0, MODE, L>(A, scale, sl, pivots, moved, dp, high);
	return high < 0x7ff00000u;
}

// The reference's step tests compare a quotient with a threshold. A comparison of the dividend with the threshold
// times the divisor decides them unless the two lie within 1e-4 of each other (the rounding of either side is far
// below that), and only then the quotient is formed.

// max |step| / max(|p|, 1e-12) < 1e-6
template <int NP>
__device__ __forceinline__ bool SmallStep(const double (&step)[NP], const double (&p)[NP])
{
	bool maybe = true;
	#pragma unroll
	for (int a = 0; a < NP; ++a) { maybe = maybe && !(fabs(step[a]) > 1.0001e-6 * fmax(fabs(p[a]), 1e-12)); }
	if (!maybe) { return false; }
	double r = 0.0;
	#pragma unroll
	for (int a = 0; a < NP; ++a) { r = fmax(r, fabs(step[a]) / fmax(fabs(p[a]), 1e-12)); }
	return r < 1e-6;
}

// gain / predicted > 1e-2
__device__ __forceinline__ bool GainRatioAbove(double gain, double predicted)
{
	if (predicted > 1e-280 && predicted < 1e280) {
		if (gain > 1.0001e-2 * predicted) { return true; }
		if (gain < 0.9999e-2 * predicted) { return false; }
	}
	return gain / predicted > 1e-2;
}

// sum / n < 1e-5
__device__ __forceinline__ bool MeanBelow(double sum, double n) { return !(sum > 1.0001e-5 * n) && sum / n < 1e-5; }

// Candidates for the lanes (groups) that need one: from a queue counter (zeroed before the launch), one atomic per
// warp, or, without one, in a fixed stride.
struct Taker {
	uint32_t n, next, stride;
	unsigned int* counter;
	bool out;  // the queue is exhausted
	__device__ __forceinline__ void Init(uint32_t count, unsigned int* ctr, int L)
	{
		n = count;
		counter = ctr;
		next = (blockIdx.x * blockDim.x + threadIdx.x) / L;
		stride = gridDim.x * blockDim.x / L;
		out = false;
	}
	// Called by all 32 lanes; need is set in the lanes (one per group) that take a candidate.
	__device__ __forceinline__ uint32_t Take(bool need)
	{
		if (counter == nullptr) {
			uint32_t k = kNoRoi;
			if (need && next < n) { k = next; next += stride; }
			out = __ballot_sync(kFull, need && k != kNoRoi) == 0;
			return k;
		}
		const unsigned mask = __ballot_sync(kFull, need);
		if (mask == 0 || out) { return kNoRoi; }
		const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
		uint32_t base = 0;
		if (lane == leader) { base = atomicAdd(counter, static_cast<unsigned>(__popc(mask))); }
		base = __shfl_sync(kFull, base, leader);
		out = base + static_cast<uint32_t>(__popc(mask)) >= n;
		const uint32_t k = base + static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)));
		return need && k < n ? k : kNoRoi;
	}
};

// Blocks per SM the thread-per-ROI kernels are held to: modes 1 and 2 fit 168 registers (3 warps per scheduler).
template <int MODE> struct ThreadBlocks { static constexpr int v = MODE == kG2Fixed ? 8 : MODE == kG2Sigma ? 6 : 4; };

// The LM iterations (GaussianFit.cpp:180-272). lo..hi: the ROI counts this launch serves (the other mappings' launches
// serve the rest). A fit needs 9 iterations on average in mode 2 and 15-18 in modes 3 and 4, but 2 % and 10 % of them
// run into the cap of 75, which sets the launch's tail: about 1 ms with a thread per ROI. Chains of two and three
// launches that pass fits beyond 8-30 iterations on to the next one, packed into full warps again, measured the same
// (365 738 ROIs: 3.49, 3.48 and 3.54 ms).
template <int MODE, int L>
__global__ void __launch_bounds__(kThreads, L == 1 ? ThreadBlocks<MODE>::v : 0) ExactFitKernel(const uint16_t* __restrict__ img, int H, int W, long long N,
                                                           const Cand* __restrict__ cands, const uint32_t* nptr,
                                                           uint32_t nconst, uint32_t lo, uint32_t hi, FitParams fp, int pitch,
                                                           double* rows, const uint8_t* only)
{
	extern __shared__ __align__(16) double exactSmem[];
	constexpr int NP = NpOf<MODE>::v, NT = SumsOf<MODE>::v;
	const uint32_t n = nptr ? *nptr : nconst;
	if (n < lo || n > hi) { return; }
	const Slot<MODE, L> sl(exactSmem, pitch);
	const unsigned mask = GroupMask<L>();
	const int gl = threadIdx.x & (L - 1), first = (threadIdx.x & 31) - gl;
	Taker taker;
	taker.Init(n, fp.mle.queue, L);
	uint32_t k = kNoRoi;
	bool fresh = false;
	double pTry[NP], lambda = 1e-2, denom = 0.0, cx = 0.0, cy = 0.0;
	int it = 0;
	Roi R;
	R.base = img;
	R.W = W;
	R.roi = fp.roi;
	R.n = fp.n;
	R.X0 = R.Y0 = 0.0;
	while (true) {
		uint32_t kk = taker.Take(gl == 0 && k == kNoRoi);
		if constexpr (L > 1) { kk = __shfl_sync(kFull, kk, first); }
		if (kk != kNoRoi && (!only || only[kk])) {
			const Cand cd = cands[kk];
			if (!LocateRoi(img + static_cast<long long>(cd.frame) * N, H, W, fp, cd, R)) {
				if (gl == 0) { rows[static_cast<long long>(kk) * kCols + kStatusCol] = kStSentinel; }
			}
			else {
				uint32_t vmin = 0xffffffffu, vmax = 0u;
				if constexpr (L == 1) {
					const uint16_t* row = R.base;
					for (int i = 0; i < R.roi; ++i, row += W) {
						for (int j = 0; j < R.roi; ++j) {
							const uint32_t v = __ldg(row + j);
							vmin = min(vmin, v);
							vmax = max(vmax, v);
						}
					}
				}
				else {
					for (int q = gl; q < R.n; q += L) {
						const int i = q / R.roi, j = q - i * R.roi;
						const uint32_t v = __ldg(R.base + static_cast<long long>(i) * W + j);
						vmin = min(vmin, v);
						vmax = max(vmax, v);
					}
					vmin = __reduce_min_sync(mask, vmin);
					vmax = __reduce_max_sync(mask, vmax);
				}
				cx = cd.x;
				cy = cd.y;
				pTry[0] = ToDouble(vmin);
				pTry[1] = ToDouble(vmax) - ToDouble(vmin);
				pTry[2] = cx;
				pTry[3] = cy;
				if constexpr (MODE == kG2Sigma) { pTry[4] = fp.sigmaX; }
				if constexpr (MODE == kG3Fixed || MODE == kG3Theta) {
					pTry[4] = 1.4142135623730951 * fp.sigmaX;
					pTry[5] = 1.4142135623730951 * fp.sigmaY;
				}
				if constexpr (MODE == kG3Theta) { pTry[6] = fp.theta; }
				k = kk;
				fresh = true;
			}
		}
		const bool busy = k != kNoRoi;
		if (__ballot_sync(kFull, busy) == 0) {
			if (taker.out) { break; }
			continue;
		}
		bool eval = busy && fresh, finish = false, failed = false;
		if (busy && !fresh) {
			// one LM step from the last accepted point: every branch that does not reach a trial point ends or damps
			double dp[NP];
			if (!Solve<MODE, L>(sl, lambda, dp)) {
				if (lambda < 1e7) { lambda = fmin(lambda * 11, 1e7); }
				else { failed = true; }
			}
			else {
				double lob[NP], hib[NP], p[NP];
				Bounds<MODE>(cx, cy, lob, hib);
				bool dpFin = true, tiny = true;
				#pragma unroll
				for (int i = 0; i < NP; ++i) {
					dpFin = dpFin && isfinite(dp[i]);
					p[i] = sl.P(i);
					pTry[i] = fmin(fmax(p[i] + dp[i], lob[i]), hib[i]);
					dp[i] = pTry[i] - p[i];
					tiny = tiny && fabs(dp[i]) < 1e-15;
				}
				if (!dpFin) { failed = true; }
				else if (tiny) {
					finish = lambda >= 1e7;
					lambda = fmin(lambda * 11, 1e7);
				}
				else {
					double quad = 0.0, lin = 0.0;
					denom = 0.0;
					#pragma unroll
					for (int i = 0; i < NP; ++i) {
						double t = 0.0;
						#pragma unroll
						for (int j = 0; j < NP; ++j) { t += sl.Alpha(U<NP>(i, j)) * dp[j]; }
						const double b = sl.Beta(i);
						quad += dp[i] * t;
						lin += dp[i] * b;
						denom += dp[i] * ((lambda * dp[i]) + b);
					}
					const double gain = (2.0 * lin) - quad;
					if (gain <= 0.0) {
						finish = lambda >= 1e7;
						lambda = fmin(lambda * 11, 1e7);
						finish = finish || (it >= 2 && SmallStep<NP>(dp, p));
					}
					else { eval = true; }
				}
			}
			if (!eval && !failed && !finish) {
				++it;
				finish = it >= kMaxIter;
			}
		}
		if (eval) {
			GModel<MODE> m;
			m.Make(pTry, fp.sigmaX, fp.theta);
			double out[L == 1 ? NT : 1];
			if constexpr (L == 1) { SumsThread<MODE>(R, m, pTry, out); }
			else { SumsGroup<MODE, L>(sl, R, m, pTry); }
			auto sum = [&](int q) {
				if constexpr (L == 1) { return out[q]; }
				else { return sl.New()[q]; }
			};
			const double errTry = sum(0);
			bool accept = fresh;
			if (fresh) {
				bool fin = isfinite(errTry);
				#pragma unroll
				for (int a = 0; a < NP; ++a) { fin = fin && isfinite(sum(1 + a)); }
				failed = !fin;
				lambda = 1e-2;
				it = 0;
			}
			else {
				accept = GainRatioAbove(sl.Err() - errTry, 2.0 * denom);
				if (accept) {
					const Divisor nine{9.0, 1.0 / 9.0};
					lambda = fmax(nine.Quick(lambda), 1e-7);  // lambda lies in [1e-7, 1e7]
				}
				else {
					finish = lambda >= 1e7;
					lambda = fmin(lambda * 11, 1e7);
				}
			}
			bool small = false;  // the step, against the parameters in force after it
			if (!fresh && it >= 2) {
				double step[NP], ref[NP];
				#pragma unroll
				for (int a = 0; a < NP; ++a) {
					const double old = sl.P(a);
					step[a] = pTry[a] - old;
					ref[a] = accept ? pTry[a] : old;
				}
				small = SmallStep<NP>(step, ref);
			}
			if constexpr (L > 1) { __syncwarp(mask); }
			if (accept) {
				if constexpr (L == 1) {
					#pragma unroll
					for (int q = 0; q < NT; ++q) { sl.s[q * kThreads] = out[q]; }
					#pragma unroll
					for (int a = 0; a < NP; ++a) { sl.P(a) = pTry[a]; }
				}
				else {
					for (int q = gl; q < NT; q += L) { sl.s[q] = sl.New()[q]; }
					#pragma unroll
					for (int a = 0; a < NP; ++a) {
						if (gl == a) { sl.P(a) = pTry[a]; }
					}
				}
			}
			if constexpr (L > 1) { __syncwarp(mask); }
			double mb = 0.0;
			#pragma unroll
			for (int a = 0; a < NP; ++a) { mb = fmax(mb, fabs(sl.Beta(a))); }
			if (fresh) { finish = mb < 1e-6; }
			else {
				if (it >= 2) { finish = finish || small || MeanBelow(sl.Err(), static_cast<double>(R.n)) || mb < 1e-6; }
				++it;
				finish = finish || it >= kMaxIter;
			}
			fresh = false;
		}
		if (failed || finish) {
			double* row = rows + static_cast<long long>(k) * kCols;
			if constexpr (L == 1) {
				#pragma unroll
				for (int a = 0; a < NP; ++a) { row[a] = sl.P(a); }
				row[kStatusCol] = failed ? kStSentinel : kStFitted;
			}
			else {
				if (gl < NP) { row[gl] = sl.P(gl); }
				if (gl == 0) { row[kStatusCol] = failed ? kStSentinel : kStFitted; }
				__syncwarp(mask);
			}
			k = kNoRoi;
		}
	}
}

__device__ __forceinline__ void StoreRow(double* row, const Cand& c, double x, double y, double off, double amp, double sx,
                                         double sy, double th, double qxy)
{
	row[cId] = 0;
	row[cPlane] = 0;
	row[cIndex] = 0;
	row[cChannel] = -1;
	row[cX] = x;
	row[cY] = y;
	row[cZ] = 0;
	row[cIntensity] = (amp > kEps && sx > kEps && sy > kEps) ? 2.0 * 3.141592653589793 * amp * sx * sy : -1;
	row[cSigmaX] = sx;
	row[cSigmaY] = sy;
	row[cTheta] = th;
	row[cQualityXY] = qxy;
	row[cQualityZ] = -1;
	row[cAmplitude] = amp;
	row[cOffset] = off;
	row[cSegIntensity] = c.intensity;
	row[cSurface] = c.surf;
	row[cCircularity] = (sx > kEps && sy > kEps) ? fmin(sx, sy) / fmax(sx, sy) : 1;
}

// Squared correlation on the model of the last accepted parameters (GaussianFit.cpp:274-295) and the output row. A
// group stages `pitch` model and data values at a time and every lane adds them in pixel order.
template <int MODE, int L>
__global__ void __launch_bounds__(kThreads) ExactFinalKernel(const uint16_t* __restrict__ img, int H, int W, long long N,
                                                             const Cand* __restrict__ cands, const uint32_t* nptr,
                                                             uint32_t nconst, uint32_t lo, uint32_t hi, FitParams fp, int pitch,
                                                             double* rows, const uint8_t* only)
{
	extern __shared__ __align__(16) double exactSmem[];
	constexpr int NP = NpOf<MODE>::v;
	const uint32_t n = nptr ? *nptr : nconst;
	if (n < lo || n > hi) { return; }
	const unsigned mask = GroupMask<L>();
	const int gl = threadIdx.x & (L - 1);
	double* sd = exactSmem + (threadIdx.x / L) * 2 * pitch;
	double* sm = sd + pitch;
	for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) / L; k < n; k += gridDim.x * blockDim.x / L) {
		if (only && !only[k]) { continue; }
		const Cand cd = cands[k];
		double* row = rows + static_cast<long long>(k) * kCols;
		const bool fitted = row[kStatusCol] == kStFitted;
		double p[NP];
		#pragma unroll
		for (int a = 0; a < NP; ++a) { p[a] = row[a]; }
		if constexpr (L > 1) { __syncwarp(mask); }  // the row is rewritten below
		Roi R;
		if (!fitted || !LocateRoi(img + static_cast<long long>(cd.frame) * N, H, W, fp, cd, R)) {
			if (gl == 0) { StoreRow(row, cd, cd.x, cd.y, -1, -1, -1, -1, -1, -1); }
			continue;
		}
		GModel<MODE> m;
		m.Make(p, fp.sigmaX, fp.theta);
		double muD = 0.0, muM = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
		if constexpr (L == 1) {
			for (int pass = 0; pass < 2; ++pass) {
				Cursor at[2];
				at[0].Set(0, R.roi);
				at[1].Set(1, R.roi);
				const int di = 2 / R.roi, dj = 2 - di * R.roi;
				for (int q = 0; q < R.n; q += 2) {
					double x[2], y[2], v[2], hat[2];
					#pragma unroll
					for (int b = 0; b < 2; ++b) {
						double X, Y;
						v[b] = at[b].Value(R, X, Y);
						x[b] = X - p[2];
						y[b] = Y - p[3];
						at[b].Step(di, dj, R.roi);
					}
					m.template Eval<false, 2>(x, y, hat, nullptr);
					#pragma unroll
					for (int b = 0; b < 2; ++b) {
						if (q + b >= R.n) { break; }
						if (pass == 0) { muD += v[b]; muM += hat[b]; }
						else {
							const double d = v[b] - muD, h = hat[b] - muM;
							t1 += d * h;
							t2 += d * d;
							t3 += h * h;
						}
					}
				}
				if (pass == 0) {
					muD /= static_cast<double>(R.n);
					muM /= static_cast<double>(R.n);
				}
			}
		}
		else {
			const bool once = R.n <= pitch;  // the staged values serve both passes
			for (int pass = 0; pass < 2; ++pass) {
				for (int c0 = 0; c0 < R.n; c0 += pitch) {
					const int cnt = min(pitch, R.n - c0);
					if (pass == 0 || !once) {
						for (int q = gl; q < cnt; q += L) {
							Cursor at;
							at.Set(c0 + q, R.roi);
							double X, Y, hat[1];
							sd[q] = at.Value(R, X, Y);
							const double x[1] = {X - p[2]}, y[1] = {Y - p[3]};
							m.template Eval<false, 1>(x, y, hat, nullptr);
							sm[q] = hat[0];
						}
						__syncwarp(mask);
					}
					if (pass == 0) {
						#pragma unroll 4
						for (int q = 0; q < cnt; ++q) { muD += sd[q]; muM += sm[q]; }
					}
					else {
						#pragma unroll 4
						for (int q = 0; q < cnt; ++q) {
							const double d = sd[q] - muD, h = sm[q] - muM;
							t1 += d * h;
							t2 += d * d;
							t3 += h * h;
						}
					}
					__syncwarp(mask);
				}
				if (pass == 0) {
					muD /= static_cast<double>(R.n);
					muM /= static_cast<double>(R.n);
				}
			}
		}
		const double Rr = t1 / sqrt(t2 * t3);
		const double rr = isnan(Rr) ? 0 : Rr * Rr;
		if (gl != 0) { continue; }
		if (rr < kEps) {
			StoreRow(row, cd, p[2], p[3], -1, -1, -1, -1, -1, -1);
			continue;
		}
		const double r2 = 1.4142135623730951;
		double sx = fp.sigmaX, sy = fp.sigmaY, th = fp.theta;
		if constexpr (MODE == kG2Fixed) { sx = sy = fp.sigmaX; th = 0; }
		if constexpr (MODE == kG2Sigma) { sx = p[4]; sy = sx; th = 0; }
		if constexpr (MODE == kG3Fixed || MODE == kG3Theta) { sx = p[4] / r2; sy = p[5] / r2; }
		if constexpr (MODE == kG3Theta) { th = p[6]; }
		StoreRow(row, cd, p[2], p[3], p[0], p[1], sx, sy, th, rr);
	}
}

// Pixels a group stages at a time: a 9 x 9 ROI whole.
constexpr int kStagePixels = 88;
// Mapping by the number of ROIs: a warp per ROI up to kWarpRois, 8 lanes up to GroupRois, a thread per ROI above. The
// lines lie where the measured times cross (us, L = 32 / 8 / 1, dense frames): mode 2 4 849 ROIs 583 / 610 / 1137,
// 19 596 1314 / 924 / 1593, 39 126 2362 / 1407 / 1742, 97 733 5416 / 2850 / 1995; mode 4 6 065 1878 / 1780 / 2304,
// 24 348 5816 / 3525 / 4261, 75 999 16963 / 8742 / 5333; mode 1 97 733 1940 / 1271 / 1389; mode 3 24 348 3539 / 2100 /
// 2976, 75 999 10083 / 4975 / 3502. The previous kernel: mode 2 741, 1869, 3584, 7793; mode 4 2527, 9680, 29923.
constexpr uint32_t kWarpRois = 5000;
template <int MODE> struct GroupRois {
	static constexpr uint32_t v = MODE == kG2Fixed ? 110000 : MODE == kG2Sigma ? 56000 : MODE == kG3Fixed ? 42000 : 32000;
};

int SmCount()
{
	int dev = 0, sms = 148;
	if (cudaGetDevice(&dev) == cudaSuccess) { cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
	return sms;
}

template <typename K>
uint32_t ResidentBlocks(K kernel, size_t bytes, int sms)
{
	if (bytes > 48 * 1024) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)); }
	int perSm = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, kThreads, bytes) != cudaSuccess || perSm < 1) { perSm = 1; }
	return static_cast<uint32_t>(sms * perSm);
}

template <int MODE, int L>
bool LaunchMapping(const uint16_t* img, int H, int W, long long N, const Cand* cands, const uint32_t* nptr, uint32_t nconst,
                   uint32_t lo, uint32_t hi, uint32_t cap, const FitParams& fp, double* rows, const uint8_t* only, cudaStream_t st)
{
	const int sms = SmCount();
	// whole batches and two more entries: even, so that pixel pairs are 16-byte aligned, and not a multiple of the banks
	const int pitch = (std::min(fp.n, kStagePixels) + kStageUnit - 1) / kStageUnit * kStageUnit + 2;
	const uint32_t most = std::max<uint32_t>(1, std::min(cap, hi));
	const uint32_t need = static_cast<uint32_t>((static_cast<unsigned long long>(most) * L + kThreads - 1) / kThreads);
	const size_t fitBytes = SlotBytes<MODE, L>(pitch);
	const size_t finalBytes = L == 1 ? 0 : sizeof(double) * 2 * pitch * (kThreads / L);
	const uint32_t fitBlocks = std::min(need, ResidentBlocks(ExactFitKernel<MODE, L>, fitBytes, sms));
	const uint32_t finalBlocks = std::min(need, static_cast<uint32_t>(sms) * 16u);
	if (fp.mle.queue && !PTB_CUDA(cudaMemsetAsync(fp.mle.queue, 0, sizeof(unsigned int), st))) { return false; }
	ExactFitKernel<MODE, L><<<fitBlocks, kThreads, fitBytes, st>>>(img, H, W, N, cands, nptr, nconst, lo, hi, fp, pitch, rows, only);
	ExactFinalKernel<MODE, L><<<finalBlocks, kThreads, finalBytes, st>>>(img, H, W, N, cands, nptr, nconst, lo, hi, fp, pitch, rows, only);
	CountLaunch(2);
	return PTB_LAUNCHED();
}

template <int MODE>
bool LaunchMode(const uint16_t* img, int H, int W, long long N, const Cand* cands, const uint32_t* nptr, uint32_t nconst,
                uint32_t cap, const FitParams& fp, double* rows, const uint8_t* only, cudaStream_t st)
{
	const uint32_t most = nptr ? cap : nconst, least = nptr ? 0 : nconst;
	bool ok = true;
	if (least <= kWarpRois) { ok = ok && LaunchMapping<MODE, 32>(img, H, W, N, cands, nptr, nconst, 0, kWarpRois, cap, fp, rows, only, st); }
	if (least <= GroupRois<MODE>::v && most > kWarpRois) {
		ok = ok && LaunchMapping<MODE, 8>(img, H, W, N, cands, nptr, nconst, kWarpRois + 1, GroupRois<MODE>::v, cap, fp, rows, only, st);
	}
	if (most > GroupRois<MODE>::v) {
		ok = ok && LaunchMapping<MODE, 1>(img, H, W, N, cands, nptr, nconst, GroupRois<MODE>::v + 1, 0xffffffffu, cap, fp, rows, only, st);
	}
	return ok;
}

}  // namespace

// fp.mle.queue: one work-queue counter (zeroed here), or null. Where the count is known only on the device, every
// mapping that could serve it is launched and the others return at once.
bool LaunchExactFit(const uint16_t* img, int H, int W, long long N, const Cand* cands, const uint32_t* nptr, uint32_t nconst,
                    uint32_t cap, const FitParams& fp, double* rows, const uint8_t* only, cudaStream_t st)
{
	switch (fp.mode) {
		case kG2Fixed: return LaunchMode<kG2Fixed>(img, H, W, N, cands, nptr, nconst, cap, fp, rows, only, st);
		case kG2Sigma: return LaunchMode<kG2Sigma>(img, H, W, N, cands, nptr, nconst, cap, fp, rows, only, st);
		case kG3Fixed: return LaunchMode<kG3Fixed>(img, H, W, N, cands, nptr, nconst, cap, fp, rows, only, st);
		case kG3Theta: return LaunchMode<kG3Theta>(img, H, W, N, cands, nptr, nconst, cap, fp, rows, only, st);
		default: return false;
	}
}

}  // namespace ptb
