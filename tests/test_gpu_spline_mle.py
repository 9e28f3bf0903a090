"""Cubic-spline maximum-likelihood fit (mode 8) against the oracle for every number of lanes per ROI, at the sizes where
its table layouts, pixel shares and pre-scan blocks can go wrong: tables of unequal sides (also even ones), ROIs smaller
than a lane group, counts that fill neither a block nor a group, positions whose ROI crosses the border."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(roi, table, n, seed):
    """n emitters of the table's own model, one per cell of a grid, and two positions at the border."""
    import spline_table
    rng = np.random.default_rng(seed)
    sx, sy, sz = table
    p = spline_table.fit_params(roi=roi, sx=sx, sy=sy, sz=sz, dz_nm=40.0)
    coef = p[5:].reshape(4, 4, 4, sz, sy, sx)
    params = np.concatenate([p[:5], [100.0, 2.0, 30, 0.0], p[5:]])
    pitch, per, h = roi + 2, 8, roi // 2
    img = np.full((pitch * -(-n // per) + 1, pitch * per + 1), 20.0)
    pos = np.zeros((n + 2, 6))
    for e in range(n):
        cy, cx = e // per * pitch + pitch // 2, e % per * pitch + pitch // 2
        x, y = rng.uniform(0.1, 0.9, 2)
        z = sz / 2 + rng.uniform(-0.25, 0.25) * sz
        for i in range(-h, h + 1):
            for j in range(-h, h + 1):
                at = np.array([z, (sy - 1) / 2 + i - y, (sx - 1) / 2 + j - x])
                c = np.clip(np.floor(at).astype(int), 0, [sz - 1, sy - 1, sx - 1])
                f = (at - c)[:, None] ** np.arange(4)
                img[cy + i, cx + j] += 6000 * np.einsum("i,j,k,ijk", f[0], f[1], f[2], coef[:, :, :, c[0], c[1], c[2]])
        pos[e] = e + 1, 1, cx + x, cy + y, 500.0, 9.0
    pos[n:, 0], pos[n:, 1], pos[n:, 4], pos[n:, 5] = n + 1, 1, 500.0, 9.0
    pos[n, 2:4], pos[n + 1, 2:4] = (0.5, 0.5), (img.shape[1] - 0.5, img.shape[0] / 2)
    stack = (rng.poisson(img) * 2 + 100).astype(np.uint16)[None]
    return stack, pos, params


@pytest.mark.parametrize("lanes", ["1", "2", "4", "8", "16", "32"])
@pytest.mark.parametrize("roi,table,n", [(7, (13, 17, 9), 1), (7, (16, 13, 12), 33), (11, (17, 20, 7), 63), (15, (21, 25, 10), 65)])
def test_fit_matches_the_oracle(lib, orc, roi, table, n, lanes, monkeypatch):
    monkeypatch.setenv("PTB_MLE_LANES", lanes)
    stack, pos, params = _case(roi, table, n, roi + n)
    got, want = lib.fitting(stack, pos, 8, params), orc.fitting(stack, pos, 8, params)
    assert got.shape == want.shape == (n + 2, 18)
    # the stated tolerances of the fit against its FP64 oracle
    for col, atol, rtol in ((4, 1e-3, 0), (5, 1e-3, 0), (6, 0.05, 0), (7, 0, 1e-4), (14, 0, 1e-4)):
        np.testing.assert_allclose(got[:, col], want[:, col], atol=atol, rtol=rtol, err_msg="column %d" % col)
    assert (got[n:, 10] == -1).all() and (got[:n, 10] > 0).all()


@pytest.mark.parametrize("roi,n", [(5, 33), (15, 65)])
def test_astigmatic_pre_scan(lib, orc, roi, n, monkeypatch):
    """Mode 7, whose pre-scan runs in the same blocks, at a small and the largest ROI; the spots are those of its own
    calibration (the table samples that Gaussian)."""
    monkeypatch.setenv("PTB_MLE_LANES", "4")
    stack, pos, _ = _case(15, (21, 25, 10), n, roi + n)
    astig = [150.0, 400.0, 0.05, 0.0, 1.3 * 160, -150.0, 400.0, -0.05, 0.0, 1.3 * 160]
    params = np.array([float(roi), 160.0] + astig + [100.0, 2.0, 30, -600.0, 600.0, 0.0])
    got, want = lib.fitting(stack, pos, 7, params), orc.fitting(stack, pos, 7, params)
    for col, atol, rtol in ((4, 1e-3, 0), (5, 1e-3, 0), (6, 0.05, 0), (7, 0, 1e-4), (14, 0, 1e-4)):
        np.testing.assert_allclose(got[:, col], want[:, col], atol=atol, rtol=rtol, err_msg="column %d" % col)
