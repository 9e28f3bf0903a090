"""Cubic-spline EMCCD fit (mode 5) against the oracle at the sizes where its pixel groups and table layout can go wrong:
ROIs below, at and above 96 pixels (three per lane), tables of unequal sides, positions at the border."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("roi,table", [(1, (5, 6, 3)), (3, (7, 5, 4)), (5, (9, 13, 6)), (7, (13, 11, 9)), (9, (17, 19, 7)),
                                       (11, (15, 21, 5)), (13, (25, 17, 8)), (15, (19, 23, 4))])
def test_fit_matches_the_oracle(lib, orc, roi, table):
    import spline_table
    rng = np.random.default_rng(roi)
    stack = (rng.poisson(20, (2, 96, 112)) + 1).astype(np.uint16)
    params = spline_table.fit_params(roi=roi, sx=table[0], sy=table[1], sz=table[2])
    n = 60
    pos = np.empty((n, 6))
    pos[:, 0], pos[:, 1] = np.arange(n) + 1, rng.integers(1, 3, n)
    pos[:, 2], pos[:, 3], pos[:, 4], pos[:, 5] = rng.uniform(0, 112, n), rng.uniform(0, 96, n), 500.0, 9.0
    got, want = lib.fitting(stack, pos, 5, params), orc.fitting(stack, pos, 5, params)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    # the same operations with FMA contraction allowed: 1e-6, as for the other mode-5 comparisons, on the rows that the
    # oracle itself holds that well when its table moves by one rounding error
    moved = params.copy()
    moved[5:] *= 1 + 2.0 ** -52
    held = np.isclose(orc.fitting(stack, pos, 5, moved), want, rtol=1e-9, atol=1e-9, equal_nan=True).all(1)
    close = np.isclose(got, want, rtol=1e-6, atol=1e-6, equal_nan=True).all(1)
    assert (close | ~held).all()
