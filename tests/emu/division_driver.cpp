// The least-squares fits' division by a shared divisor and their model, the code of csrc/fit_exact.cu itself, on the CPU:
// the quick quotient against IEEE division over its stated operands, the range predicates at their edges, and the model
// formed with quick quotients against plain ones wherever it calls its parameters quick. Test harness only.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

inline int __double2hiint(double d)
{
	uint64_t b;
	std::memcpy(&b, &d, 8);
	return static_cast<int>(b >> 32);
}
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
enum Modes { kG2Fixed = 1, kG2Sigma = 2, kG3Fixed = 3, kG3Theta = 4 };

#include "division.inc"

namespace {

std::mt19937_64 rng(1);
uint64_t bad = 0;

double Pow2(int e) { return std::ldexp(1.0, e); }

// A double of exponent lo..hi with a random, a short or an almost full mantissa.
double Draw(int lo, int hi)
{
	uint64_t m = rng() & 0xfffffffffffffull;
	const int kind = rng() & 3;
	if (kind == 1) { m &= 0xff; }
	if (kind == 2) { m |= 0xfffffffffff00ull; }
	if (kind == 3 && (rng() & 1)) { m = rng() & 1 ? 0 : 0xfffffffffffffull; }
	const uint64_t b = (static_cast<uint64_t>(1023 + lo + static_cast<int>(rng() % static_cast<unsigned>(hi - lo + 1))) << 52) | m;
	double d;
	std::memcpy(&d, &b, 8);
	return d;
}

void Check(bool ok, const char* what, double a, double b)
{
	if (!ok && ++bad < 10) { std::printf("%s %a %a\n", what, a, b); }
}

template <int MODE> void Model(int n)
{
	constexpr int NP = NpOf<MODE>::v;
	std::uniform_real_distribution<double> u(0.0, 1.0);
	uint64_t quick = 0;
	for (int i = 0; i < n; ++i) {
		double p[7] = {1000 * u(rng), 0, 20 + 5 * u(rng), 30 + 5 * u(rng), 0, 0, 0};
		p[1] = i % 5 == 0 ? std::exp(-60 * u(rng)) : 60000 * u(rng);   // from 1e-26
		if (i % 7 == 0) { p[2] = std::floor(p[2]) + Draw(-59, -20) * (rng() & 1 ? 1 : -1); }
		if (i % 11 == 0) { p[2] = std::floor(p[2]); p[3] = std::floor(p[3]); }  // distances of zero
		double sigma = i % 3 ? 0.1 + 19.9 * u(rng) : 0.1;
		if (i % 13 == 0) { sigma = Draw(-62, 62); }
		const double theta = i % 4 == 0 ? 0.0 : i % 4 == 1 ? 1.5707963267948966 * static_cast<double>(rng() % 100) : 300 * u(rng) - 150;
		if (MODE == kG2Sigma) { p[4] = sigma; }
		if (MODE >= kG3Fixed) { p[4] = sigma; p[5] = i % 6 ? 0.1 + 19.9 * u(rng) : sigma; }
		if (MODE == kG3Theta) { p[6] = theta; }
		GModel<MODE> m;
		m.Make(p, sigma, theta);
		quick += m.quick;
		for (int k = 0; k < 9; ++k) {
			const double x[1] = {static_cast<double>(18 + rng() % 12) - p[2]}, y[1] = {static_cast<double>(28 + rng() % 12) - p[3]};
			double v[1], g[1][NP], plain[NP], e = 0;
			m.template Eval<true, 1>(x, y, v, g);
			const double w = m.template Form<true, false>(x[0], y[0], plain, e);
			Check(v[0] == w || (std::isnan(v[0]) && std::isnan(w)), "model value", v[0], w);
			for (int a = 0; a < NP; ++a) { Check(g[0][a] == plain[a] || (std::isnan(g[0][a]) && std::isnan(plain[a])), "gradient", g[0][a], plain[a]); }
		}
	}
	std::printf("mode %d: quick %.3f of %d\n", MODE, static_cast<double>(quick) / n, n);
	if (quick * 2 < static_cast<uint64_t>(n)) { ++bad; }
}

}  // namespace

int main()
{
	const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
	const double lo = Pow2(-60), hi = Pow2(60);
	for (double s : {1.0, -1.0}) {
		Check(Safe(s * lo) && !Safe(s * std::nextafter(lo, 0.0)) && !Safe(s * hi) && Safe(s * std::nextafter(hi, 0.0)), "Safe", s, 0);
		Check(!Safe(s * 0.0) && !Safe(s * inf) && !Safe(s * nan) && !Safe(s * std::numeric_limits<double>::denorm_min()), "Safe", s, 1);
		Check(ZeroOrAbove<-960>(s * 0.0) && ZeroOrAbove<-960>(s * Pow2(-960)) && !ZeroOrAbove<-960>(s * std::nextafter(Pow2(-960), 0.0)), "ZeroOrAbove", s, 0);
		Check(ZeroOrAbove<-60>(s * lo) && !ZeroOrAbove<-60>(s * std::nextafter(lo, 0.0)), "ZeroOrAbove", s, 1);
	}
	for (int i = 0; i < 8000000; ++i) {
		double b = i & 1 ? Draw(-60, 59) : i & 2 ? (rng() & 1 ? lo : std::nextafter(hi, 0.0)) * (1 + (rng() & 3) * 0x1p-52) : Draw(-2, 4);
		if (!Safe(b)) { b = lo; }
		if (rng() & 1) { b = -b; }
		double a = i % 3 == 0 ? Draw(-960, 299) : i % 3 == 1 ? Draw(-960, -950) : b * Draw(0, 1) * (1 + 0x1p-53);
		if (i % 17 == 0) { a = rng() & 1 ? Pow2(-960) : std::nextafter(Pow2(300), 0.0); }
		if (i % 1001 == 0) { a = 0.0; }
		if (rng() & 1) { a = -a; }
		Divisor d;
		d.Set(b);
		Check(d.Quick(a) == a / b, "quotient", a, b);
	}
	Model<kG2Fixed>(200000);
	Model<kG2Sigma>(200000);
	Model<kG3Fixed>(200000);
	Model<kG3Theta>(200000);
	std::printf("%llu differences\n", static_cast<unsigned long long>(bad));
	return bad ? 1 : 0;
}
