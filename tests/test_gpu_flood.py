"""Warp-wide floods and basin fusions against the oracle, bit for bit, where they can go wrong: equal potentials (the
heap settles ties), plateaus, more open entries than the warp's list holds, boxes around the shared-memory limit, more
basins than a warp has lanes, groups at the frame's border."""
import numpy as np
import pytest

from conftest import GAUSS_PARAMS

pytestmark = pytest.mark.gpu


def _blobs(rng, h, w, centres, sigma, amp, levels):
    y, x = np.mgrid[0:h, 0:w]
    f = np.full((h, w), 200.0)
    for cy, cx in centres:
        f += amp * rng.uniform(0.5, 1.0) * np.exp(-((y - cy) ** 2 + (x - cx) ** 2) / (2 * sigma ** 2))
    f += rng.normal(0, 3, (h, w))
    if levels:  # few grey levels: equal W1 values everywhere
        f = np.round(f / levels) * levels
    return np.clip(f, 0, 65535).astype(np.uint16)


def _frame(kind, seed):
    rng = np.random.default_rng(seed)
    h, w = 90 + seed, 121 + 2 * seed
    if kind == "noise":
        return rng.integers(0, 65536, (h, w)).astype(np.uint16)
    if kind == "ties":
        return rng.integers(0, 3, (h, w)).astype(np.uint16) * 1000
    if kind == "plateaus":
        return np.kron(rng.integers(0, 4, (h // 3 + 1, w // 3 + 1)), np.ones((3, 3)))[:h, :w].astype(np.uint16) * 700
    if kind == "pairs":  # groups of two and three close emitters, some on the border
        c = [(rng.uniform(0, h), rng.uniform(0, w)) for _ in range(25)]
        return _blobs(rng, h, w, c + [(a + rng.uniform(2, 4), b + rng.uniform(-3, 3)) for a, b in c], 1.3, 2000, 0)
    if kind == "levels":
        c = [(rng.uniform(0, h), rng.uniform(0, w)) for _ in range(60)]
        return _blobs(rng, h, w, c, 1.6, 1500, 64)
    # one dense cluster: a group of many basins in a box around and above 320 pixels
    n = 12 + 8 * (seed % 6)
    c = [(h / 2 + rng.normal(0, 2 + seed), w / 2 + rng.normal(0, 2 + seed)) for _ in range(n)]
    return _blobs(rng, h, w, c, 1.2, 1500, 0)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("kind", ["noise", "ties", "plateaus", "pairs", "levels", "cluster"])
def test_flood_and_fusion_match_the_oracle(lib, orc, kind, seed):
    stack = np.stack([_frame(kind, seed), _frame(kind, seed)[::-1]])
    w1 = orc.planes(stack[0])[1]
    top = float(w1.max())
    for thr in (float(np.quantile(w1[w1 > 0], 0.6)), 0.02 * top):
        for ratio in (0.0, 0.5, 1.5, 10.0):
            a = lib.localization(stack, thr, ratio, 0, GAUSS_PARAMS)
            b = orc.localization(stack, thr, ratio, 0, GAUSS_PARAMS)
            assert np.array_equal(a, b), (thr, ratio)
