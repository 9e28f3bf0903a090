"""Builds the host-code drivers of tests/emu: the library's own objects linked with a stand-in for the CUDA runtime."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda"


def link(exe, sources, runtime="fake"):
    """exe from tests/emu sources and the library's objects, on the stand-in runtime or (runtime="cuda") on the CUDA one."""
    import build  # palmtracer-cpp_b200/build.py
    if shutil.which("g++") is None or not os.path.exists(build.NVCC):
        pytest.skip("g++ or nvcc is missing")
    build.build()
    objs = sorted(os.path.join(build.OBJ, os.path.basename(s) + ".o") for s in build.sources())
    emu = os.path.join(HERE, "emu")
    libs = [os.path.join(emu, "fake_cudart.cpp")] if runtime == "fake" else ["-L" + CUDA + "/lib64", "-lcudart_static", "-lrt"]
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I" + CUDA + "/include"] + [os.path.join(emu, s) for s in sources] + \
        objs + libs + ["-ldl", "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return str(exe)


def run(exe, *args, timeout=120):
    r = subprocess.run([exe] + list(args), capture_output=True, text=True, timeout=timeout)
    print(r.stdout, r.stderr)
    return r.returncode
