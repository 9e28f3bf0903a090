// Cubic-spline PSF fit, EMCCD Poisson deviance (mode 5), one warp per ROI, FP64.
//
// Reference: lib/fit/SplineFit.cpp:53-318 with the bounds of lib/fit/Fitting.cpp:161-172, the centre of mass of
// lib/signal_processing/Matrix.cpp:245-269, its Cholesky (:272-294) and LU inverse (:358-410). Every behaviour of
// the reference is kept, including the ones that look accidental: the deviance accumulator starts at DBL_MAX and
// is never reset (so updates are always accepted and the loop stops after the third iteration unless the deviance
// turns NaN), the ROI row index drives the spline's x cell and the column index its y cell, and the output columns
// carry CRLB values (Offset = CRLB(bg), Intensity/Amplitude = CRLB(A), QualityXY = mean CRLB(x, y), QualityZ =
// deltaZ * CRLB(z)).
//
// The coefficient table lies on the device as [64][z][x][y] (the reference's [64][z][y][x] with x and y exchanged): all
// pixels of an evaluation share the 64 weights and differ in their cell only, and the lanes of a warp hold consecutive
// columns of the ROI, which are consecutive y cells. A load of one coefficient then reads 4-5 cache lines per warp. With
// the 64 coefficients of a cell in one run every lane read its own line: 32 tag lookups per load, which bound the
// kernel (2 347 ROIs of 9 x 9, table 17 x 17 x 41: 6.3 ms; with this layout 2.4 ms). What bounds it now is the serial
// part of an iteration (about 25 dependent divisions of the solve and the steps) beside the 64 x 4 products per pixel;
// three pixels per lane are evaluated side by side so that a coefficient's weights are read once for all of them, held
// to 168 registers: 3 140 ROIs 2.24 ms, 31 432 21.0 ms (before 6.35 and 60.2; with 128 registers 2.68 and 20.2).
#include <algorithm>

#include "pt_common.cuh"

namespace ptb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 4;

__device__ __forceinline__ double WarpSumD(double v)
{
	#pragma unroll
	for (int d = 16; d > 0; d >>= 1) { v += __shfl_xor_sync(kFull, v, d); }
	return v;
}

// Weights of the value and of its derivatives in x, y and z, per coefficient.
struct __align__(16) Patch {
	double2 fx[64], yz[64];
};

// Monomial weights x^k y^j z^i and their derivatives (SplineFit.cpp:296-318), two entries per lane.
__device__ void PatchWeights(Patch& P, double x, double y, double z)
{
	const int lane = threadIdx.x & 31;
	for (int id = lane; id < 64; id += 32) {
		const int i = id >> 4, j = (id >> 2) & 3, k = id & 3;
		double cz = 1.0, cy = 1.0, cx = 1.0, cxm = 1.0;
		for (int a = 0; a < i; ++a) { cz *= z; }
		for (int a = 0; a < j; ++a) { cy *= y; }
		for (int a = 0; a < k; ++a) { cxm = cx; cx *= x; }
		const double zy = cz * cy;
		P.fx[id] = make_double2(zy * cx, k > 0 ? static_cast<double>(k) * (zy * cxm) : 0.0);
		// derivative in y: j * x^k y^(j-1) z^i; in z: i * x^k y^j z^(i-1)
		double cym = 1.0, czm = 1.0;
		for (int a = 0; a + 1 < j; ++a) { cym *= y; }
		for (int a = 0; a + 1 < i; ++a) { czm *= z; }
		P.yz[id] = make_double2(j > 0 ? static_cast<double>(j) * (cz * cym * cx) : 0.0,
		                        i > 0 ? static_cast<double>(i) * (czm * cy * cx) : 0.0);
	}
	__syncwarp();
}

// size_t semantics of Vec3I::Clamp: a negative index wraps and clamps to the upper bound.
__device__ __forceinline__ long long ClampCell(long long v, int dim) { return (v < 0 || v > dim - 1) ? dim - 1 : v; }

// Pixels a lane evaluates side by side: each coefficient's weights are read from shared memory once for all of them.
constexpr int kSide = 3;

// Models and derivatives at the lane's pixels idx0, idx0 + 32, .. (those below npx; the others repeat the last pixel),
// SplineFit.cpp:219-240.
__device__ __forceinline__ void Eval(const FitParams& fp, const Patch& P, int idx0, int npx, int roi, long long xi, long long yi,
                                     long long zi, const double* p, double (&model)[kSide], double (&dudt)[kSide][5])
{
	const double* c[kSide];
	double s1[kSide], s2[kSide], s3[kSide], s4[kSide];
	const long long z = ClampCell(zi, fp.sz);
	#pragma unroll
	for (int t = 0; t < kSide; ++t) {
		const int idx = min(idx0 + 32 * t, npx - 1);
		const int i = idx / roi, j = idx - i * roi;
		const long long x = ClampCell(xi + i + fp.offsetXY, fp.sx), y = ClampCell(yi + j + fp.offsetXY, fp.sy);
		c[t] = fp.coeffs + ((z * fp.sx) + x) * fp.sy + y;
		s1[t] = s2[t] = s3[t] = s4[t] = 0;
	}
	constexpr int kBatch = 8;
	#pragma unroll 1
	for (int i0 = 0; i0 < 64; i0 += kBatch) {
		double v[kSide][kBatch];
		#pragma unroll
		for (int t = 0; t < kSide; ++t) {
			#pragma unroll
			for (int i = 0; i < kBatch; ++i) { v[t][i] = __ldg(c[t] + i * fp.splineSize); }
			c[t] += kBatch * fp.splineSize;
		}
		#pragma unroll
		for (int i = 0; i < kBatch; ++i) {
			const double2 fx = P.fx[i0 + i], yz = P.yz[i0 + i];
			#pragma unroll
			for (int t = 0; t < kSide; ++t) {
				s1[t] += fx.x * v[t][i];
				s2[t] += fx.y * v[t][i];
				s3[t] += yz.x * v[t][i];
				s4[t] += yz.y * v[t][i];
			}
		}
	}
	#pragma unroll
	for (int t = 0; t < kSide; ++t) {
		dudt[t][0] = 1;
		dudt[t][1] = s1[t];
		dudt[t][2] = s2[t] * (-1 * p[1]);
		dudt[t][3] = s3[t] * (-1 * p[1]);
		dudt[t][4] = s4[t] * p[1];
		model[t] = p[0] + (p[1] * dudt[t][1]);
	}
}

__device__ void StoreRow(double* row, double segI, double surf, double x, double y, double z, double off, double amp,
                         double qxy, double qz, bool sentinel)
{
	const int lane = threadIdx.x & 31;
	double v[kCols];
	v[cId] = 0; v[cPlane] = 0; v[cIndex] = 0; v[cChannel] = -1;
	v[cX] = x; v[cY] = y; v[cZ] = z;
	v[cIntensity] = amp;
	v[cSigmaX] = sentinel ? -1 : 0; v[cSigmaY] = sentinel ? -1 : 0; v[cTheta] = sentinel ? -1 : 0;
	v[cQualityXY] = qxy; v[cQualityZ] = qz;
	v[cAmplitude] = amp; v[cOffset] = off;
	v[cSegIntensity] = segI; v[cSurface] = surf;
	v[cCircularity] = 1.0;
	#pragma unroll
	for (int c = 0; c < kCols; ++c) {
		if (lane == c) { row[c] = v[c]; }
	}
}

__global__ void __launch_bounds__(32 * kWarps, 3) SplineFitKernel(const uint16_t* __restrict__ img, int H, int W, long long N,
                                                                const Cand* __restrict__ cands, const uint32_t* nptr,
                                                                uint32_t nconst, FitParams fp, double* rows)
{
	__shared__ Patch patches[kWarps];
	Patch& P = patches[threadIdx.x >> 5];
	const int lane = threadIdx.x & 31;
	const uint32_t n = nptr ? *nptr : nconst;
	const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
	const int roi = fp.roi, hh = fp.half, npx = fp.n;
	for (uint32_t k = warp; k < n; k += nw) {
		const Cand cd = cands[k];
		double* row = rows + static_cast<long long>(k) * kCols;
		const bool nonneg = cd.x >= 0.0 && cd.y >= 0.0;
		const unsigned long long ux = nonneg ? static_cast<unsigned long long>(cd.x) : 0ull;
		const unsigned long long uy = nonneg ? static_cast<unsigned long long>(cd.y) : 0ull;
		const unsigned long long h = static_cast<unsigned long long>(hh);
		if (!nonneg || !RoiInside(ux, uy, hh, H, W)) {
			StoreRow(row, cd.intensity, cd.surf, cd.x, cd.y, 0, -1, -1, -1, -1, true);
			continue;
		}
		const uint16_t* base = img + static_cast<long long>(cd.frame) * N + static_cast<long long>(uy - h) * W + static_cast<long long>(ux - h);
		// ROI min / max and centre of mass (rows weight y, columns weight x)
		double vmin = 1e300, vmax = -1e300, sx = 0, sy = 0, sv = 0;
		for (int idx = lane; idx < npx; idx += 32) {
			const int i = idx / roi, j = idx - i * roi;
			const double v = static_cast<double>(__ldg(base + static_cast<long long>(i) * W + j));
			vmin = fmin(vmin, v);
			vmax = fmax(vmax, v);
			sy += v * static_cast<double>(i);
			sx += v * static_cast<double>(j);
			sv += v;
		}
		#pragma unroll
		for (int d = 16; d > 0; d >>= 1) {
			vmin = fmin(vmin, __shfl_xor_sync(kFull, vmin, d));
			vmax = fmax(vmax, __shfl_xor_sync(kFull, vmax, d));
		}
		sx = WarpSumD(sx);
		sy = WarpSumD(sy);
		sv = WarpSumD(sv);
		double x0, y0;
		if (sv > 0) { x0 = sx / sv; y0 = sy / sv; }
		else { x0 = static_cast<double>(roi) / 2.0; y0 = static_cast<double>(roi) / 2.0; }
		const double roiC = (fp.roiParam - 1) / 2.0, roiD = fp.roiParam / 4.0;
		const double lo[5] = {-0.01, -1, roiC - roiD, roiC - roiD, 0};
		const double hi[5] = {0.01, 1, roiC + roiD, roiC + roiD, static_cast<double>(fp.sz)};
		double p[5] = {vmin, (vmax - vmin) * fp.intensityRatio, x0, y0, fp.initZ};
		#pragma unroll
		for (int a = 0; a < 5; ++a) { p[a] = fmin(fmax(p[a], lo[a]), hi[a]); }
		double jump[5] = {fmax(20.0, p[1]), fmax(100.0, p[1]), 1.0, 1.0, fmax(static_cast<double>(fp.sz) / 3.0, 2.0)};
		double lambda = 0.1, err = 1.7976931348623157e308, mu = 1 + lambda;
		double upd[5] = {0, 0, 0, 0, 0};
		auto cell = [&](const double* pp, long long& xi, long long& yi, long long& zi) {
			const double xr = -1 * (pp[2] - static_cast<double>(hh) + 0.5), yr = -1 * (pp[3] - static_cast<double>(hh) + 0.5);
			xi = static_cast<int>(floor(xr));
			yi = static_cast<int>(floor(yr));
			zi = static_cast<int>(floor(pp[4]));
			PatchWeights(P, xr - static_cast<double>(xi), yr - static_cast<double>(yi), pp[4] - static_cast<double>(zi));
		};
		bool stop = false;
		int it = 0;
		while (!stop) {
			++it;
			const double oldErr = err, oldLambda = lambda;
			double oldP[5], oldUpd[5];
			#pragma unroll
			for (int a = 0; a < 5; ++a) { oldP[a] = p[a]; oldUpd[a] = upd[a]; upd[a] = 0; }
			long long xi, yi, zi;
			cell(p, xi, yi, zi);
			double dev = 0, jac[5] = {0, 0, 0, 0, 0}, hs[15] = {};
			for (int idx0 = lane; idx0 < npx; idx0 += 32 * kSide) {
				double dudt[kSide][5], model[kSide];
				Eval(fp, P, idx0, npx, roi, xi, yi, zi, p, model, dudt);
				#pragma unroll
				for (int t = 0; t < kSide; ++t) {
					const int idx = idx0 + 32 * t;
					if (idx >= npx) { break; }
					const int i = idx / roi, j = idx - i * roi;
					const double d = static_cast<double>(__ldg(base + static_cast<long long>(i) * W + j));
					dev += d > 0 ? 2 * (model[t] - d - (d * log(model[t] / d))) : 2 * model[t];
					const double t1 = 1 - (d / model[t]), t2 = d / (model[t] * model[t]);
					int q = 0;
					#pragma unroll
					for (int a = 0; a < 5; ++a) {
						jac[a] += t1 * dudt[t][a];
						#pragma unroll
						for (int b = a; b < 5; ++b) { hs[q++] += t2 * dudt[t][a] * dudt[t][b]; }
					}
				}
			}
			err = err + WarpSumD(dev);
			double hess[5][5];
			{
				int q = 0;
				#pragma unroll
				for (int a = 0; a < 5; ++a) {
					jac[a] = WarpSumD(jac[a]);
					#pragma unroll
					for (int b = a; b < 5; ++b) {
						hess[a][b] = WarpSumD(hs[q++]);
						hess[b][a] = hess[a][b];
					}
				}
			}
			#pragma unroll
			for (int a = 0; a < 5; ++a) { hess[a][a] = hess[a][a] * mu; }
			// Cholesky, lower factor u (Matrix.cpp:272-294)
			double u[5][5] = {};
			bool chol = true;
			#pragma unroll
			for (int a = 0; a < 5; ++a) {
				#pragma unroll
				for (int b = 0; b <= a; ++b) {
					double s = 0;
					#pragma unroll
					for (int c = 0; c < b; ++c) { s += u[a][c] * u[b][c]; }
					if (a == b) {
						if (hess[a][a] - s >= 0) { u[a][b] = sqrt(hess[a][a] - s); }
						else { chol = false; }
					}
					else { u[a][b] = 1.0 / u[b][b] * (hess[a][b] - s); }
				}
			}
			if (chol) {
				double yv[5];
				#pragma unroll
				for (int a = 0; a < 5; ++a) {
					yv[a] = jac[a];
					#pragma unroll
					for (int b = 0; b < a; ++b) { yv[a] -= u[a][b] * yv[b]; }
					yv[a] /= u[a][a];
				}
				#pragma unroll
				for (int a = 4; a >= 0; --a) {
					upd[a] = yv[a];
					#pragma unroll
					for (int b = a + 1; b < 5; ++b) { upd[a] -= u[b][a] * upd[b]; }
					upd[a] /= u[a][a];
				}
				#pragma unroll
				for (int a = 0; a < 5; ++a) {
					if (fabs(oldUpd[a]) > kEps && upd[a] / oldUpd[a] < -0.5) { jump[a] *= 0.5; }
					const double scale = upd[a] / (1.0 + (fabs(upd[a]) / jump[a]));
					p[a] -= scale;
					p[a] = fmin(fmax(p[a], lo[a]), hi[a]);
					upd[a] = scale;
				}
			}
			if (!chol || err > oldErr) {
				err = oldErr;
				#pragma unroll
				for (int a = 0; a < 5; ++a) { p[a] = oldP[a]; upd[a] = oldUpd[a]; }
				lambda = oldLambda;
				mu = fmax((1 + (lambda * 10)) / (1 + lambda), 1.3);
				lambda = 10 * lambda;
			}
			else {
				lambda = 0.1 * lambda;
				mu = 1 + lambda;
			}
			if (it >= kMaxIter) { stop = true; }
			if (it > 2 && (err < 1e-6 || fabs(err - oldErr) / err < 1e-6)) { stop = true; }
		}
		// CRLB from the Fisher information at the final parameters (SplineFit.cpp:164-205)
		long long xi, yi, zi;
		cell(p, xi, yi, zi);
		double fs[15] = {};
		for (int idx0 = lane; idx0 < npx; idx0 += 32 * kSide) {
			double dudt[kSide][5], model[kSide];
			Eval(fp, P, idx0, npx, roi, xi, yi, zi, p, model, dudt);
			#pragma unroll
			for (int t = 0; t < kSide; ++t) {
				if (idx0 + 32 * t >= npx) { break; }
				int q = 0;
				#pragma unroll
				for (int a = 0; a < 5; ++a) {
					#pragma unroll
					for (int b = a; b < 5; ++b) { fs[q++] += dudt[t][b] * dudt[t][a] / model[t]; }
				}
			}
		}
		double m[25];
		{
			int q = 0;
			#pragma unroll
			for (int a = 0; a < 5; ++a) {
				#pragma unroll
				for (int b = a; b < 5; ++b) {
					const double v = WarpSumD(fs[q++]);
					m[a * 5 + b] = v;
					m[b * 5 + a] = v;
				}
			}
		}
		#pragma unroll
		for (int a = 0; a < 5; ++a) {
			if (fabs(m[a * 5 + a]) < 2.220446049250313e-16) { m[a * 5 + a] = 1e-10; }
		}
		// LU inverse without pivoting, column-major as Matrix.cpp:358-410 (only the diagonal of the inverse is kept)
		double crlb[5];
		{
			double acc = 0;
			#pragma unroll
			for (int j = 0; j < 5; ++j) {
				#pragma unroll
				for (int i = 1; i <= j; ++i) {
					#pragma unroll
					for (int q = 0; q <= i - 1; ++q) { acc += m[i + q * 5] * m[q + j * 5]; }
					m[i + j * 5] -= acc;
					acc = 0;
				}
				#pragma unroll
				for (int i = j + 1; i < 5; ++i) {
					if (j > 0) {
						#pragma unroll
						for (int q = 0; q <= j - 1; ++q) { acc += m[i + q * 5] * m[q + j * 5]; }
						m[i + j * 5] = (1 / m[j + j * 5]) * (m[i + j * 5] - acc);
						acc = 0;
					}
					else { m[i + j * 5] = (1 / m[j + j * 5]) * m[i + j * 5]; }
				}
			}
			#pragma unroll
			for (int num = 0; num < 5; ++num) {
				double yv[5], out[5];
				yv[0] = num == 0 ? 1 : 0;
				#pragma unroll
				for (int i = 1; i < 5; ++i) {
					#pragma unroll
					for (int j = 0; j <= i - 1; ++j) { acc += m[i + j * 5] * yv[j]; }
					yv[i] = (i == num ? 1.0 : 0.0) - acc;
					acc = 0;
				}
				out[4] = yv[4] / m[4 + 4 * 5];
				#pragma unroll
				for (int i = 3; i >= 0; --i) {
					#pragma unroll
					for (int j = i + 1; j < 5; ++j) { acc += m[i + j * 5] * out[j]; }
					out[i] = (1 / m[i + i * 5]) * (yv[i] - acc);
					acc = 0;
				}
				const double v = out[num];
				crlb[num] = isnan(v) ? v : (v >= 0 ? sqrt(v) : 0.0);  // real part of the complex square root
			}
		}
		const double xo = p[2] - static_cast<double>(hh) + cd.x;
		const double yo = p[3] - static_cast<double>(hh) + cd.y;
		const double zo = fp.deltaZ * (p[4] - fp.initZ);
		StoreRow(row, cd.intensity, cd.surf, xo, yo, zo, crlb[0], crlb[1], (crlb[2] + crlb[3]) / 2, fp.deltaZ * crlb[4], false);
	}
}

// The table as given, [64][cells], in the layouts the maximum-likelihood spline fit reads: [cells][64] in FP32 and
// [16][cells][4] in FP32 and FP64. A tile of 32 cells per CTA, read along the cells and written along the coefficients.
constexpr int kTableCells = 32;
__global__ void __launch_bounds__(256) CellTable(const double* __restrict__ given, double2* __restrict__ quads64,
                                                 float* __restrict__ cells32, float4* __restrict__ quads32, size_t cells)
{
	__shared__ double tile[64][kTableCells + 1];
	const size_t c0 = static_cast<size_t>(blockIdx.x) * kTableCells;
	for (int i = threadIdx.x; i < 64 * kTableCells; i += 256) {
		const int k = i / kTableCells, c = i % kTableCells;
		if (c0 + c < cells) { tile[k][c] = __ldg(given + k * cells + c0 + c); }
	}
	__syncthreads();
	for (int i = threadIdx.x; i < 64 * kTableCells; i += 256) {
		const int c = i / 64, k = i % 64;
		if (c0 + c < cells) { cells32[(c0 + c) * 64 + k] = static_cast<float>(tile[k][c]); }
	}
	for (int i = threadIdx.x; i < 16 * kTableCells; i += 256) {
		const int q = i / kTableCells, c = i % kTableCells;
		if (c0 + c < cells) {
			const double v[4] = {tile[4 * q][c], tile[4 * q + 1][c], tile[4 * q + 2][c], tile[4 * q + 3][c]};
			double2* at = quads64 + (q * cells + c0 + c) * 2;
			at[0] = make_double2(v[0], v[1]);
			at[1] = make_double2(v[2], v[3]);
			quads32[q * cells + c0 + c] = make_float4(static_cast<float>(v[0]), static_cast<float>(v[1]), static_cast<float>(v[2]),
			                                          static_cast<float>(v[3]));
		}
	}
}

__global__ void SwapTable(const double* __restrict__ given, double* __restrict__ swapped, int sx, int sy, long long n)
{
	const long long slab = static_cast<long long>(sx) * sy;
	for (long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; k < n; k += gridDim.x * static_cast<long long>(blockDim.x)) {
		const long long s = k / slab, r = k - s * slab;
		const int x = static_cast<int>(r / sy), y = static_cast<int>(r - static_cast<long long>(x) * sy);
		swapped[k] = __ldg(given + s * slab + static_cast<long long>(y) * sx + x);
	}
}

}  // namespace

bool LaunchCellTable(const double* given, double* quads64, float* cells32, float* quads32, size_t cells, cudaStream_t st)
{
	CellTable<<<static_cast<unsigned>((cells + kTableCells - 1) / kTableCells), 256, 0, st>>>(
		given, reinterpret_cast<double2*>(quads64), cells32, reinterpret_cast<float4*>(quads32), cells);
	CountLaunch();
	return PTB_LAUNCHED();
}

// The reference's table [slabs = 64 sz][sy][sx] as [slabs][sx][sy].
bool LaunchSwapTable(const double* given, double* swapped, int sx, int sy, long long slabs, cudaStream_t st)
{
	const long long n = slabs * sx * sy;
	SwapTable<<<static_cast<unsigned>(std::min<long long>((n + 255) / 256, 148 * 8)), 256, 0, st>>>(given, swapped, sx, sy, n);
	CountLaunch();
	return PTB_LAUNCHED();
}

bool LaunchSpline(const uint16_t* img, int H, int W, long long N, const Cand* cands, const uint32_t* nptr, uint32_t nconst,
                  uint32_t cap, const FitParams& fp, double* rows, cudaStream_t st)
{
	const uint32_t blocks = std::min<uint32_t>((std::max<uint32_t>(cap, 1) + kWarps - 1) / kWarps, 148u * 16u);
	SplineFitKernel<<<blocks, 32 * kWarps, 0, st>>>(img, H, W, N, cands, nptr, nconst, fp, rows);
	CountLaunch();
	return PTB_LAUNCHED();
}

}  // namespace ptb
