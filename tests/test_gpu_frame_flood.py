"""Frame-wide floods by a warp against the oracle, bit for bit: strict mode and routed frames, with and without basin
fusion, on frames with equal keys (the binary heap's ties), more open entries than shared memory holds, and sizes around
the heap's levels."""
import numpy as np
import pytest

from conftest import GAUSS_PARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,levels", [(1, 40, 1), (7, 9, 1), (40, 33, 1), (64, 64, 900), (210, 230, 1), (210, 230, 500), (400, 410, 1)])
@pytest.mark.parametrize("ratio", [0.0, 10.0])
def test_strict_mode_matches_the_oracle(lib, orc, h, w, levels, ratio):
    rng = np.random.default_rng(h + levels)
    stack = (rng.integers(0, 60000 // levels, (2, h, w)) * levels).astype(np.uint16)  # noise: half the pixels join the domain
    before = lib.set_segmentation_mode(1)
    try:
        a = lib.localization(stack, 1.0, ratio, 0, GAUSS_PARAMS)
    finally:
        lib.set_segmentation_mode(before)
    assert np.array_equal(a, orc.localization(stack, 1.0, ratio, 0, GAUSS_PARAMS))


@pytest.mark.parametrize("frames", [3, 40])
@pytest.mark.parametrize("ratio", [0.0, 10.0])
def test_more_failing_frames_than_before_are_reflooded(lib, orc, frames, ratio):
    import synth
    one, _ = synth.stack("c2", frames=1, seed=21, size=(512, 512))
    thr = 0.15 * synth.mad_threshold(orc.planes(one[0])[1])  # fails the rank test (as in the parity tests)
    stack = np.repeat(one, frames, axis=0)
    want = orc.localization(one, thr, ratio, 0, GAUSS_PARAMS)
    lib.segmentation_stats()
    got = lib.localization(stack, thr, ratio, 0, GAUSS_PARAMS)
    stats = lib.segmentation_stats()
    assert stats["reflooded"] == frames and stats["routed_why"].get("no_reflood_slot", 0) == max(0, frames - 32), stats
    for f in range(frames):
        rows = got[got[:, 1] == f + 1]
        assert np.array_equal(rows[:, 2:], want[:, 2:])
