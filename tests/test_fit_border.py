"""The fits' border test: a ROI that leaves the frame is never read, also where the frame is narrower than half of it."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "palmtracer-cpp_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"


def test_roi_inside_the_frame(tmp_path):
    """Every frame size up to 20 x 20, half ROIs up to 15 and positions inside, beside and far beyond the frame."""
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    exe = tmp_path / "border"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wno-attributes", "-I" + CUDA_INCLUDE, os.path.join(HERE, "emu", "border_driver.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    for f in ("fit_exact.cu", "fit_gauss.cu", "fit_mle.cu", "fit_spline.cu"):
        src = open(os.path.join(CSRC, f)).read()
        assert len(re.findall(r"RoiInside\(", src)) == 1 and ">(W) - h" not in src, f


@pytest.mark.gpu
@pytest.mark.parametrize("fit", [1, 2, 3, 4, 5, 6, 7, 8])
def test_frames_narrower_than_half_a_roi(lib, fit):
    """Positions beside and beyond a 5 x 40 and a 40 x 5 frame with a ROI of 15: border rows, as for every ROI that does not
    fit, and the same frame's other rows unaffected."""
    import spline_table
    roi = 15
    spline = spline_table.fit_params(roi=roi, sx=21, sy=21, sz=9)
    astig = [150.0, 400.0, 0.05, 0.0, 208.0, -150.0, 400.0, -0.05, 0.0, 208.0]
    params = {5: spline, 6: np.array([roi, 1.3, 100.0, 2.0, 20.0, 0.0]),
              7: np.array([roi, 160.0] + astig + [100.0, 2.0, 20.0, -600.0, 600.0, 0.0]),
              8: np.concatenate([[float(roi)], spline[1:5], [100.0, 2.0, 20.0, 0.0], spline[5:]])}.get(fit, np.array([roi, 1.3, 1.3, 0.0]))
    for h, w in ((5, 40), (40, 5)):
        stack = np.full((2, h, w), 300, dtype=np.uint16)
        xy = [(2.0, 2.0), (6.0, 20.0), (20.0, 6.0), (7.0, 7.0), (100.0, 20.0), (20.0, 100.0), (1e6, 1e6), (1e300, 20.0), (20.0, 1e300)]
        pos = np.array([[i + 1, 1 + i % 2, x, y, 500.0, 9.0] for i, (x, y) in enumerate(xy)])
        rows = lib.fitting(stack, pos, fit, params)
        assert np.array_equal(rows[:, 4:6], pos[:, 2:4])
        assert np.array_equal(rows[:, 13], np.full(len(xy), -1.0))  # amplitude of a border row
