"""The round-by-round matching of Tracking against the oracle where it can go wrong: more rounds of equal distances than
it takes before the sequential pass (a row links one pair a round), many candidates per point, equal positions, planes
whose points are interleaved in the table, chains longer than one launch of pointer jumping covers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _row(n, planes=2):
    """Points 2 apart on odd planes, midway between them on even ones: every neighbour at distance 1."""
    rows = []
    for p in range(planes):
        rows += [[len(rows) + i + 1, p + 1, 2.0 * i + (p & 1), 0.0] for i in range(n)]
    return np.array(rows, dtype=np.float64)


@pytest.mark.parametrize("n", [1, 2, 23, 24, 25, 60, 700])
@pytest.mark.parametrize("planes", [2, 5])
def test_rows_of_equal_distances(lib, orc, n, planes):
    pts = _row(n, planes)
    for p in (pts, pts[::-1].copy()):
        assert np.array_equal(lib.tracking(p, 1.0), orc.tracking(p, 1.0))


@pytest.mark.parametrize("seed", range(4))
def test_dense_and_equal_positions(lib, orc, seed):
    rng = np.random.default_rng(seed)
    n = 900
    pts = np.c_[np.arange(1, n + 1), rng.integers(1, 4, n), rng.integers(0, 12, (n, 2)).astype(float)]  # a coarse grid
    assert np.array_equal(lib.tracking(pts, 2.0), orc.tracking(pts, 2.0))


@pytest.mark.parametrize("planes", [31, 32, 33, 34, 1100])
def test_long_chains_and_interleaved_planes(lib, orc, planes):
    rng = np.random.default_rng(planes)
    rows = [[0, p + 1, 40.0 * k + 0.3 * rng.normal(), 5.0] for p in range(planes) for k in range(3)]
    pts = np.array(rows)[rng.permutation(len(rows))]
    pts[:, 0] = np.arange(1, len(pts) + 1)
    assert np.array_equal(lib.tracking(pts, 5.0), orc.tracking(pts, 5.0))
