"""(Y, X) order of each frame's rows at the sizes where its bands of Y can go wrong: no row, one row, many rows on one
line (equal Y; more than a band holds), counts on both sides of the shared-memory limit, one frame (written by several
CTAs) and many. The rows without a fit are the oracle's bit for bit, so their order is, too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(h, w, ys, xs):
    """Equal spots (a 5 x 5 pyramid) centred at every (y, x)."""
    img = np.full((h, w), 100, dtype=np.uint16)
    k = np.minimum(*np.meshgrid([1, 2, 3, 2, 1], [1, 2, 3, 2, 1])) * 400
    for y in ys:
        for x in xs:
            img[y - 2:y + 3, x - 2:x + 3] += k.astype(np.uint16)
    return img


@pytest.mark.parametrize("frames", [1, 3, 160])
@pytest.mark.parametrize("rows_of,cols_of", [(0, 0), (1, 1), (1, 20), (1, 64), (1, 65), (2, 90), (9, 40)])
def test_rows_on_lines(lib, orc, rows_of, cols_of, frames):
    h, w = 16 + 12 * max(rows_of, 1), 24 + 12 * max(cols_of, 1)
    img = _frame(h, w, [12 + 12 * r for r in range(rows_of)], [16 + 12 * c for c in range(cols_of)])
    stack = np.repeat(img[None], frames, 0)
    stack[1::2] = stack[1::2, :, ::-1]
    got, want = lib.localization(stack, 50.0, 0.0, 0, np.zeros(6)), orc.localization(stack, 50.0, 0.0, 0, np.zeros(6))
    assert want.shape[0] == rows_of * cols_of * frames
    assert got.shape == want.shape and np.array_equal(got, want)


@pytest.mark.parametrize("size", [(600, 900), (760, 900)])
@pytest.mark.parametrize("frames", [1, 2])
def test_counts_around_the_shared_memory_limit(lib, orc, size, frames):
    rng = np.random.default_rng(size[0])
    img = _frame(*size, range(8, size[0] - 8, 12), range(8, size[1] - 8, 12))
    stack = rng.poisson(np.repeat(img[None], frames, 0)).astype(np.uint16)
    got = lib.localization(stack, 50.0, 0.0, 0, np.zeros(6), capacity_doubles=6000 * frames * 18)
    want = orc.localization(stack, 50.0, 0.0, 0, np.zeros(6), capacity_doubles=6000 * frames * 18)
    per_frame = want.shape[0] // frames
    assert (per_frame <= 4096) == (size[0] == 600)
    assert got.shape == want.shape and np.array_equal(got, want)
