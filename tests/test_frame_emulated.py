"""A chunk's whole segmentation on the CPU (tests/emu/frame_driver.cpp: the library's kernels in the library's launch
order, each CUDA thread a host thread) under ThreadSanitizer and AddressSanitizer, against the oracle's labels.

tests/emu/warp_shim.h gives the warp's ballots and shuffles the ordering that the hardware promises, none: only
__syncwarp and __syncthreads order a lane's loads before another lane's stores. ThreadSanitizer therefore reports every
pair of accesses that a flood leaves to the compiler's schedule.
"""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "palmtracer-cpp_b200", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"
STATS = ("routed", "rank_tested", "reflooded", "fused_global", "fits", "fault", "groups")


def _source(name, host, out, small=()):
    """The kernels of csrc/<name> as a host include: the launch functions from `host` on are left out, dynamic shared
    memory becomes a static buffer of its own size, and the constants in `small` take the values given."""
    src = open(os.path.join(CSRC, name)).read()
    src = src[:src.index(host)] + src[src.rindex("}  // namespace ptb"):]
    src = src.replace('#include "pt_common.cuh"', '#include "%s"' % os.path.join(CSRC, "pt_common.cuh"))
    for const, value in small:
        src, n = re.subn(r"(constexpr \w+ %s = )\w+;" % const, r"\g<1>%s;" % value, src)
        assert n == 1, const
    src = src.replace("extern __shared__ uint32_t frameHeap[];", "static __attribute__((aligned(16))) uint32_t frameHeap[3 * kFrameHeap];")
    src = src.replace("extern __shared__ uint32_t hist[];", "static uint32_t hist[kRefloodBuckets];")
    open(out, "w").write(src)


def _build(d, sanitizer, small=()):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    _source("segment.cu", "bool LaunchSegment(", d / "frame_emu.inc", small)
    _source("scan.cu", "// state: the jobs' words", d / "scan_emu.inc")
    exe = d / "frame_emu"
    cmd = ["g++", "-std=c++20", "-O1", "-g", "-fsanitize=" + sanitizer, "-pthread", "-Wno-attributes", "-I" + CUDA_INCLUDE,
           "-I" + str(d), "-I" + os.path.join(HERE, "emu"), os.path.join(HERE, "emu", "frame_driver.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.fixture(scope="module")
def racecheck(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("frame_tsan"), "thread")


def _run(exe, orc, frames, thr, ratio=0.0, mode=0, warps=0):
    """(label differences from the oracle, statistics, the sanitizer's reports)."""
    d = exe.parent
    b, h, w = frames.shape
    w1 = np.stack([orc.planes(f)[1] for f in frames])
    fixed = np.round(w1 * 65536).astype(np.int64)
    assert np.array_equal(fixed, w1 * 65536)  # W1 is an exact multiple of 2^-16
    with open(d / "in.bin", "wb") as f:
        np.array([h, w, b, mode], dtype=np.int32).tofile(f)
        np.array([int(np.floor(thr * 65536))], dtype=np.int64).tofile(f)
        np.array([ratio]).tofile(f)
        fixed.tofile(f)
    r = subprocess.run([str(exe), str(d / "in.bin"), str(d / "out.bin"), str(warps)], capture_output=True, text=True,
                       env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0", TSAN_OPTIONS="exitcode=0"), timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    raw = np.fromfile(d / "out.bin", dtype=np.uint8)
    p = b * h * w
    lab, code, rest = raw[:4 * p].view(np.uint32), raw[4 * p:5 * p], raw[5 * p:].view(np.uint32)
    out_base, stats = rest[:b + 1], dict(zip(STATS, map(int, rest[b + 1:])))
    assert stats["fault"] == 0 and out_base[-1] == stats["fits"] and out_base[0] == 0 and (np.diff(out_base.astype(np.int64)) >= 0).all()
    diff = 0
    for k, f in enumerate(frames):
        at = slice(k * h * w, (k + 1) * h * w)
        dom = (code[at] & 1) != 0
        got, want = lab[at][dom].astype(np.int64), orc.labels(f, thr, ratio).reshape(-1)[dom].astype(np.int64)
        if ratio < 1 and (want > 0).any():  # regions are numbered over the chunk
            got = np.where(got > 0, got - got[want > 0].min() + want[want > 0].min(), 0)
        elif ratio >= 1:  # a fusion keeps one of its basins' numbers: compared as partitions
            pairs, count = np.unique(np.stack([got, want]), axis=1, return_counts=True)
            keep = np.zeros(pairs.shape[1], bool)
            keep[[np.flatnonzero(pairs[0] == v)[np.argmax(count[pairs[0] == v])] for v in np.unique(pairs[0])]] = True
            diff += int(count[~keep].sum()) + keep.sum() - np.unique(pairs[1, keep]).size
            continue
        diff += int(np.sum(got != want))
    return diff, stats, r.stderr


def _reports(err, function):
    """ThreadSanitizer's reports with an access made in `function`."""
    return [x for x in err.split("WARNING: ThreadSanitizer")[1:] if function in x]


def _dense(size, seed, count=1):
    import synth
    s, _ = synth.stack("c2", frames=count, seed=seed, size=size)
    return s, synth.mad_threshold


def test_box_flood_orders_its_accesses(racecheck, orc):
    """The flood of a staged box by a warp: what a lane reads before a pop's stores is read before them by more than the
    compiler's schedule (the last open entry, which the first pushing lane overwrites)."""
    s, mad = _dense((64, 64), 21)
    diff, stats, err = _run(racecheck, orc, s, 0.3 * mad(orc.planes(s[0])[1]), warps=1)
    print(stats, "label differences", diff)
    assert diff == 0 and stats["groups"] >= 3, stats
    assert _reports(err, "FloodWarp") == [], _reports(err, "FloodWarp")[0][:3000]


@pytest.fixture(scope="module")
def boundscheck(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("frame_asan"), "address")


def _order(exe, n, pixels, base):
    r = subprocess.run([str(exe), "order", str(n), str(pixels), str(base)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (n, pixels, base, r.stderr[-2000:])
    return float(r.stdout)


@pytest.mark.parametrize("n, pixels, base", [(0, 100, 0), (1, 1, 7), (31, 31, 5), (33, 100, 200), (4000, 4000, 12345), (9000, 32768, 0),
                                             (5000, 32769, 2 * 32769), (20000, 1 << 20, 1 << 30), (3000, 2147483647, 0)])
def test_seed_order(boundscheck, n, pixels, base):
    """A frame's seeds in raster order: fewer pixels than bands, as many, one more, and the largest frame."""
    _order(boundscheck, n, pixels, base)


def test_seed_order_grows_with_the_seeds(boundscheck):
    """Sixteen times the seeds take about sixteen times as long (comparing all with all took 256 times)."""
    small, large = (min(_order(boundscheck, n, 1 << 22, 0) for _ in range(3)) for n in (1 << 15, 1 << 19))
    print("ms", small, large)
    assert large < 64 * small
