"""The least-squares fits' quick division: the code of csrc/fit_exact.cu (the divisor, its range predicates and the model
that chooses between quick and plain quotients) compiled for the CPU and compared with IEEE division."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "palmtracer-cpp_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"


def test_quick_quotients_are_the_plain_ones(tmp_path):
    """Quotients over the whole stated range and at its edges; model values and gradients formed with quick quotients equal
    those formed with plain ones for every set of parameters the model takes as quick (widths from 2^-62 to 2^62,
    amplitudes from 1e-26, positions on and beside pixel centres, angles at multiples of a right angle)."""
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    src = open(os.path.join(CSRC, "fit_exact.cu")).read()
    a, b = src.index("template <int MODE> struct NpOf;"), src.index("// Exact conversion of a pixel value")
    (tmp_path / "division.inc").write_text(src[a:b])
    exe = tmp_path / "division"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-attributes", "-I" + CUDA_INCLUDE, "-I" + str(tmp_path),
           os.path.join(HERE, "emu", "division_driver.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
