"""Cubic-spline EMCCD fit (mode 5) of bright spots against the oracle, on inputs that the oracle's own arithmetic holds:
almost every row is compared, at ROIs below, at and above the pixel groups' 96 pixels and tables of unequal sides."""
import numpy as np
import pytest

FREE = 7  # columns before the intensity: what one pixel determines


def _inputs(roi, table):
    import spline_table
    rng = np.random.default_rng(roi)
    n = 60
    pos = np.empty((n, 6))
    pos[:, 0], pos[:, 1] = np.arange(n) + 1, rng.integers(1, 3, n)
    gx, gy = np.meshgrid(np.arange(10), np.arange(6))
    x, y = 9 + 10 * gx.ravel() + rng.uniform(-0.4, 0.4, n), 9 + 15 * gy.ravel() + rng.uniform(-0.4, 0.4, n)
    yy, xx = np.mgrid[0:96, 0:112]
    mu = np.full((2, 96, 112), 20.0)
    for k in range(n):
        mu[int(pos[k, 1]) - 1] += 20000 * np.exp(-((xx - x[k]) ** 2 + (yy - y[k]) ** 2) / (2 * 1.3 ** 2)) / (2 * np.pi * 1.69)
    stack = rng.poisson(mu).astype(np.uint16)
    pos[:, 2], pos[:, 3], pos[:, 4], pos[:, 5] = np.round(x) + 0.2, np.round(y) - 0.1, 500.0, 9.0
    return stack, pos, spline_table.fit_params(roi=roi, sx=table[0], sy=table[1], sz=table[2])


def _held(orc, stack, pos, params, want):
    """Entries that the oracle itself moves by less than 1e-9 when its table moves by a rounding error, three ways."""
    held = np.ones(want.shape, bool)
    rng = np.random.default_rng(3)
    size = params.size - 5
    for step in (np.ones(size), -np.ones(size), rng.choice([-1.0, 1.0], size)):
        moved = params.copy()
        moved[5:] *= 1 + step * 2.0 ** -52
        held &= np.isclose(orc.fitting(stack, pos, 5, moved), want, rtol=1e-9, atol=1e-9, equal_nan=True)
    return held


SIZES = [(1, (5, 6, 3)), (3, (7, 5, 4)), (5, (9, 13, 6)), (7, (13, 11, 9)), (9, (17, 19, 7)), (11, (15, 21, 5)),
         (13, (25, 17, 8)), (15, (19, 23, 4))]


@pytest.mark.parametrize("roi, table", SIZES)
def test_the_oracle_holds_its_rows(orc, roi, table):
    """What the GPU comparison below relies on: at least 50 of the 60 rows are held, and are fits of a spot."""
    stack, pos, params = _inputs(roi, table)
    want = orc.fitting(stack, pos, 5, params)
    held = _held(orc, stack, pos, params, want)
    if roi == 1:  # five parameters from one pixel: position and z are the start's, the rest is a singular solve's
        assert held[:, :FREE].all()
        return
    assert held.all(1).sum() >= 50
    assert np.unique(want[held.all(1), 6]).size >= 40  # z of a fit


@pytest.mark.gpu
@pytest.mark.parametrize("roi, table", SIZES)
def test_spots_match_the_oracle(lib, orc, roi, table):
    stack, pos, params = _inputs(roi, table)
    got, want = lib.fitting(stack, pos, 5, params), orc.fitting(stack, pos, 5, params)
    held = _held(orc, stack, pos, params, want)
    # the same operations with FMA contraction allowed: 1e-6, as for the other mode-5 comparisons
    close = np.isclose(got, want, rtol=1e-6, atol=1e-6, equal_nan=True)
    if roi == 1:
        assert close[:, :FREE].all()
        return
    rows = held.all(1)
    assert rows.sum() >= 50 and close[rows].all()
