// The border test of the fits (RoiInside, csrc/pt_common.cuh) against its definition: every pixel of the ROI lies in the
// frame. Frames narrower than half a ROI are among them. Test harness only.
#include <cuda_runtime.h>

#include <cstdio>

#include "../../palmtracer-cpp_b200/csrc/pt_common.cuh"

int main()
{
	const unsigned long long far[] = {100, 1ull << 31, 1ull << 63, ~0ull - 7, ~0ull};
	int bad = 0, inside = 0;
	for (int W = 1; W <= 20; ++W) {
		for (int H = 1; H <= 20; ++H) {
			for (int h = 0; h <= 15; ++h) {
				for (int i = 0; i < 30; ++i) {
					for (int j = 0; j < 30; ++j) {
						const unsigned long long x = i < 25 ? i : far[i - 25], y = j < 25 ? j : far[j - 25];
						const unsigned long long hh = static_cast<unsigned long long>(h);
						const bool want = x >= hh && y >= hh && x < static_cast<unsigned long long>(W) && y < static_cast<unsigned long long>(H) &&
						                  x + hh < static_cast<unsigned long long>(W) && y + hh < static_cast<unsigned long long>(H);
						bad += ptb::RoiInside(x, y, h, H, W) != want;
						inside += want;
					}
				}
			}
		}
	}
	std::printf("%d wrong, %d inside\n", bad, inside);
	return bad || !inside ? 1 : 0;
}
