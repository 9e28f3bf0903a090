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
        src, n = re.subn(r"(constexpr \w+ %s = )[^;]+;" % const, r"\g<1>%s;" % value, src)
        assert n == 1, const
    src = src.replace("extern __shared__ uint32_t frameHeap[];", "static __attribute__((aligned(16))) uint32_t frameHeap[3 * kFrameHeap];")
    src = src.replace("extern __shared__ uint32_t hist[];", "static uint32_t hist[kRefloodBuckets];")
    open(out, "w").write(src)


def _build(d, sanitizer, small=()):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    _source("segment.cu", "bool LaunchSegment(", d / "frame_emu.inc", small)
    _source("scan.cu", "// state: the jobs' words", d / "scan_emu.inc", [("kScanPolls", "200")] if sanitizer == "address" else ())
    exe = d / "frame_emu"
    cmd = ["g++", "-std=c++20", "-O1", "-g", "-fsanitize=" + sanitizer, "-pthread", "-Wno-attributes", "-I" + CUDA_INCLUDE,
           "-I" + str(d), "-I" + os.path.join(HERE, "emu"), os.path.join(HERE, "emu", "frame_driver.cpp"), "-o", str(exe)]
    cmd += ["-DPTB_UNORDERED"] if sanitizer == "thread" else []
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.fixture(scope="module")
def racecheck(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("frame_tsan"), "thread")


def _run(exe, orc, frames, thr, ratio=0.0, mode=0, warps=0, points=0xffffffff):
    """(label differences from the oracle, statistics, the sanitizer's reports). The frames' output offsets are checked
    against the labelled regions' sizes."""
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
    if os.path.exists(d / "out.bin"):
        os.remove(d / "out.bin")
    r = subprocess.run([str(exe), str(d / "in.bin"), str(d / "out.bin"), str(warps), str(points)], capture_output=True, text=True,
                       env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0", TSAN_OPTIONS="exitcode=66"), timeout=900)
    if "unexpected memory mapping" in r.stderr:
        pytest.skip("ThreadSanitizer does not start under this kernel's address layout")
    assert r.returncode in (0, 66) and os.path.exists(d / "out.bin"), r.stderr[-3000:]
    raw = np.fromfile(d / "out.bin", dtype=np.uint8)
    p = b * h * w
    lab, code, rest = raw[:4 * p].view(np.uint32), raw[4 * p:5 * p], raw[5 * p:].view(np.uint32)
    out_base, stats = rest[:b + 1], dict(zip(STATS, map(int, rest[b + 1:])))
    assert stats["fault"] == 0 and out_base[-1] == stats["fits"] and out_base[0] == 0 and (np.diff(out_base.astype(np.int64)) >= 0).all()
    diff = 0
    for k, f in enumerate(frames):
        at = slice(k * h * w, (k + 1) * h * w)
        regions, area = np.unique(lab[at][(code[at] & 1) != 0], return_counts=True)
        assert out_base[k + 1] - out_base[k] == min(points, int(np.sum(area[regions > 0] > 4))), k
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


def _check(exe, *args):
    return subprocess.run([str(exe)] + [str(a) for a in args], capture_output=True, text=True, timeout=600,
                          env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0"))


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


@pytest.fixture(scope="module")
def smallheap(tmp_path_factory):
    """The frame-wide flood's heaps with 48 entries in shared memory: nearly all of them lie in global memory."""
    return _build(tmp_path_factory.mktemp("frame_heap"), "address", [("kFrameHeap", "48u")])


def _frames(kind, orc):
    """(frames, threshold)"""
    def w1(frame):
        return orc.planes(frame)[1]

    rng = np.random.default_rng(5)
    if kind in ("noise", "low"):  # large groups without ties; counts of 0-5, where most keys tie
        s = rng.integers(0, 65536, size=(2, 90, 110), dtype=np.uint16)
        s, q = (s, 0.5) if kind == "noise" else (rng.poisson(1.0, size=(2, 90, 110)).astype(np.uint16), 0.3)
        plane = w1(s[0])
        return s, float(np.quantile(plane[plane > 0], q))
    s, mad = _dense((130, 140), 21, 2)  # emitters at a threshold far below theirs
    return s, 0.1 * mad(w1(s[0]))


# what each row reaches: ties settled by the binary heap, the rank test and the re-flood, fusions in boxes and of groups
# too large for one, frames routed after a fusion, every frame flooded frame-wide
CHUNKS = [("noise", 10.0, 0), ("noise", 0.0, 1), ("low", 0.0, 0), ("low", 0.0, 1), ("low", 10.0, 2),
          ("dense", 10.0, 0), ("dense", 0.0, 1)]


@pytest.mark.parametrize("kind, ratio, mode", CHUNKS)
def test_chunk_in_bounds(smallheap, orc, kind, ratio, mode):
    frames, thr = _frames(kind, orc)
    diff, stats, _ = _run(smallheap, orc, frames, thr, ratio, mode, warps=2)
    print(stats, "label differences", diff)
    assert diff == 0, stats
    if ratio and mode != 1:
        assert stats["fused_global"] >= 1 and stats["routed"] >= 1, stats
    if kind == "low" and mode == 0:
        assert stats["rank_tested"] >= 1 and stats["reflooded"] >= 1, stats


@pytest.mark.parametrize("kind, ratio, mode", [("low", 0.0, 0), ("low", 10.0, 2)])
def test_chunk_orders_its_accesses(racecheck, orc, kind, ratio, mode):
    """No flood or fusion by a warp leaves two lanes' accesses to the compiler's schedule."""
    frames, thr = _frames(kind, orc)
    diff, stats, err = _run(racecheck, orc, frames, thr, ratio, mode, warps=1)
    assert diff == 0, stats
    for f in ("FloodWarp", "FloodBox", "GroupFloodBox", "GroupFuse", "FrameFlood", "FloodWide", "FloodBinary", "RefloodBox"):
        bad = [r for r in _reports(err, f) if "SuspectPair" not in r]  # marks a frame: every writer writes 1
        assert bad == [], bad[0][:3000]


def test_offsets_of_many_frames(boundscheck, orc):
    """More frames than the offsets' one CTA has threads, their regions cut to two per frame."""
    frames = np.random.default_rng(2).integers(0, 4000, size=(1030, 12, 12), dtype=np.uint16)
    diff, stats, _ = _run(boundscheck, orc, frames, 100.0, mode=2, points=2)
    assert diff == 0 and stats["fits"] > 500, stats


@pytest.mark.parametrize("n, cap", [(0, 10), (1, 1), (5, 3), (4095, 5000), (4096, 4096), (4097, 4097), (9001, 20000), (50001, 50001)])
def test_prefix_sums(boundscheck, n, cap):
    """Tiles of 4096 entries and their remainders; a device-side count above the capacity is cut to it."""
    for blocks in (1, 3):
        assert _check(boundscheck, "scan", n, cap, blocks).returncode == 0


@pytest.mark.parametrize("tile, prefix, missing", [(1, 0, -1), (1, -1, -1), (31, 3, -1), (32, -1, -1), (33, 0, -1), (33, 32, -1), (64, 31, -1),
                                                   (100, -1, -1), (100, 67, -1), (100, 5, 50), (2, -1, 0)])
def test_prefix_sum_look_back(boundscheck, tile, prefix, missing):
    """A tile whose predecessors have published sums only, or a whole prefix somewhere; one that never publishes runs the
    bounded wait out and is reported."""
    assert _check(boundscheck, "lookback", tile, prefix, missing).returncode == 0


def _order(exe, n, pixels, base):
    r = _check(exe, "order", n, pixels, base)
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
