"""Prefix sums across several tiles (4096 entries each) in one launch, seen through the entry points that use them:
tracking tables and detection stacks whose planes, points, rows and regions fall just below, on and above whole tiles."""
import numpy as np
import pytest

from conftest import GAUSS_PARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 8192, 140001])
def test_tracking_point_counts(lib, orc, n):
    rng = np.random.default_rng(n)
    planes = max(1, n // 7)
    pts = np.c_[np.arange(1, n + 1), rng.integers(1, planes + 1, n), rng.uniform(0, 30, (n, 2))]
    assert np.array_equal(lib.tracking(pts, 3.0), orc.tracking(pts, 3.0))


@pytest.mark.parametrize("frames,h,w", [(1, 4096, 17), (2, 2048, 40), (63, 65, 33), (64, 64, 48), (65, 65, 31), (4097, 9, 11)])
def test_rows_regions_and_frames(lib, orc, frames, h, w):
    rng = np.random.default_rng(frames)
    stack = rng.integers(0, 4000, (frames, h, w)).astype(np.uint16)  # noise: many regions
    a = lib.localization(stack, 100.0, 0.0, 0, GAUSS_PARAMS)
    b = orc.localization(stack, 100.0, 0.0, 0, GAUSS_PARAMS)
    assert np.array_equal(a, b)
