"""Least-squares fits (modes 1-4): the ROI mappings chosen by the number of ROIs give the same bits, and the few-ROI
mapping agrees with the oracle. The ROIs include hot pixels (widths at their bound, where exp underflows and the plain
divisions run), flat ROIs, border positions and sizes around the staged block of 88 pixels."""
import os
import subprocess
import tempfile

import numpy as np
import pytest

XY_TOL, REL_TOL = 1e-3, 1e-4


def _stack_and_positions(roi):
    import synth
    stack, em = synth.stack("c1", frames=4, seed=77)
    rng = np.random.default_rng(roi)
    stack[2:] = 140  # flat frames with hot pixels of one pixel and of two pixels
    ys, xs = rng.integers(20, 236, 40), rng.integers(20, 236, 40)
    stack[2, ys, xs] = 60000
    stack[3, ys, xs] = 4000
    stack[3, ys, xs + 1] = 3000
    rows = []
    for f, x, y in em[em[:, 0] < 2][:, :3]:
        rows.append([f + 1, x + rng.normal(0, 0.3), y + rng.normal(0, 0.3)])
    for f in (3, 4):
        rows += [[f, x + rng.uniform(-0.4, 0.4), y + rng.uniform(-0.4, 0.4)] for x, y in zip(xs, ys)]
    rows += [[3, 128.0, 10.5], [1, 1.0, 1.0], [2, 255.5, 128.0], [1, -1.0, 5.0], [9, 50.0, 50.0], [1, roi // 2, roi // 2]]
    rows = np.array(rows)
    pos = np.empty((len(rows), 6))
    pos[:, 0], pos[:, 1:4], pos[:, 4], pos[:, 5] = np.arange(len(rows)) + 1, rows, 1000.0, 9.0
    return stack, pos


# one count in each mapping's range: a warp per ROI up to 5000, 8 lanes up to 32 000-110 000 by mode, a thread above
@pytest.mark.gpu
@pytest.mark.parametrize("fit,many", [(1, 111000), (2, 57000), (3, 43000), (4, 33000)])
@pytest.mark.parametrize("roi", [1, 3, 7, 9, 11, 15])
def test_mappings_give_the_same_rows(lib, orc, fit, many, roi):
    stack, pos = _stack_and_positions(roi)
    params = np.array([float(roi), 1.3, 1.1, 0.3 if fit == 4 else 0.0])
    few = lib.fitting(stack, pos, fit, params)
    for n in (5001, many):
        at = np.arange(n) % len(pos)
        rows = lib.fitting(stack, pos[at], fit, params)
        assert np.array_equal(rows[:, 3:], few[at][:, 3:], equal_nan=True)
    if roi < 7:
        return  # under-determined: the reference's own path depends on the last bits of exp
    # against the oracle: the emitters' planes (a hot pixel's fit hangs on the last bits of exp, and a plane outside the
    # stack gives a border row here, while the oracle reads beyond the stack as the reference does)
    few, inside = few[pos[:, 1] <= 2], pos[pos[:, 1] <= 2]
    want = orc.fitting(stack, inside, fit, params)
    good = want[:, 11] > 0.9
    assert good.sum() > 40
    assert np.array_equal(few[:, 11] > 0, want[:, 11] > 0)
    assert np.abs(few[good, 4:6] - want[good, 4:6]).max() < XY_TOL
    assert (np.abs(few[good, 13] - want[good, 13]) <= REL_TOL * np.abs(want[good, 13])).all()


_DIVISION = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
static double Make(std::mt19937_64& r, int lo, int hi)
{
	uint64_t m = r() & 0xfffffffffffffull;
	const int kind = r() & 3;
	if (kind == 1) { m &= 0xff; }
	if (kind == 2) { m |= 0xfffffffffff00ull; }
	const uint64_t b = (static_cast<uint64_t>(1023 + lo + static_cast<int>(r() % static_cast<unsigned>(hi - lo + 1))) << 52) | m;
	double d;
	std::memcpy(&d, &b, 8);
	return d;
}
int main()
{
	std::mt19937_64 r(1);
	uint64_t bad = 0;
	for (int i = 0; i < 6000000; ++i) {
		const double b = Make(r, -60, 59), y = 1.0 / b;
		double a = i % 3 == 0 ? Make(r, -960, 299) : i % 3 == 1 ? Make(r, -960, -950) : b * Make(r, 0, 1) * (1 + 0x1p-53);
		if (r() & 1) { a = -a; }
		const double q = a * y;
		const double q1 = std::fma(std::fma(-q, b, a), y, q);
		bad += std::fma(std::fma(-q1, b, a), y, q1) != a / b;
	}
	std::printf("%llu\n", static_cast<unsigned long long>(bad));
}
"""


def test_quick_division_is_the_correctly_rounded_one():
    """The five-operation division of the fits equals IEEE division over its stated range of operands."""
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "div.cpp"), os.path.join(d, "div")
        with open(src, "w") as f:
            f.write(_DIVISION)
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", src, "-o", exe])
        assert subprocess.check_output([exe]).split() == [b"0"]
