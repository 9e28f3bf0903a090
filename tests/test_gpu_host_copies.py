"""Pageable host buffers through the pinned ring: sizes around its pieces (1 MB to 4 MB, four slots), odd offsets of the
buffers, the same rows as from pinned memory, and several threads copying at once."""
import threading

import numpy as np
import pytest

from conftest import GAUSS_PARAMS

pytestmark = pytest.mark.gpu


def _stack(frames, h, w, seed):
    return np.random.default_rng(seed).integers(90, 130, (frames, h, w)).astype(np.uint16)


@pytest.mark.parametrize("frames,h,w", [(1, 1, 1), (1, 512, 511), (4, 512, 256), (5, 512, 256), (17, 700, 701), (9, 1024, 1024)])
def test_pageable_and_pinned_buffers_give_the_same_rows(lib, orc, frames, h, w):
    import torch
    raw = np.empty(frames * h * w + 3, dtype=np.uint16)
    stack = raw[3:].reshape(frames, h, w)  # not aligned to anything but its own type
    stack[:] = _stack(frames, h, w, h)
    pinned = torch.empty((frames, h, w), dtype=torch.int16, pin_memory=True)
    pinned.numpy().view(np.uint16)[:] = stack
    for k in (1, 3):
        assert np.array_equal(lib.wavelett(stack, k), lib.wavelett(pinned.numpy().view(np.uint16), k))
    assert np.array_equal(lib.wavelett(stack[-1:], 2), orc.wavelett(stack[-1:], 2))
    a = lib.localization(stack, 3.0, 0.0, 0, GAUSS_PARAMS)
    b = lib.localization(pinned.numpy().view(np.uint16), 3.0, 0.0, 0, GAUSS_PARAMS)
    assert np.array_equal(a, b)


def test_threads_share_the_copy_helpers(lib):
    stacks = [_stack(6, 512, 512 + 8 * k, k) for k in range(4)]
    want = [lib.wavelett(s, 2) for s in stacks]
    got = [[None] * 3 for _ in stacks]

    def work(k):
        for r in range(3):
            got[k][r] = lib.wavelett(stacks[k], 2)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        assert all(np.array_equal(g, want[k]) for g in got[k])
