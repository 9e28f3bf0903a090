"""The work that users of the localization library have it do, as timed cases through its public entry points.

A case is a plain dict; `kind` names the entry point:
  localize   Localization: detection, segmentation and per-candidate fits of a stack (host or device buffers)
  fit        Fitting: fits at caller-given positions
  track      Tracking of a localization table
  threshold  AutoThreshold of a frame
Frames follow one camera model: ADU = 100 + 2 x Poisson(background + emitters), emitters rendered as pixel-integrated
Gaussians, 2D or astigmatic. The cases draw their sizes from the benchmark's workloads (200 x 256^2, 2000 x 1024^2,
1000 x 512^2 astigmatic, 1500 x 512^2 cubic spline, tracking of the resulting table) with the frame counts reduced,
from the per-frame form (one frame per call) and from odd, ragged frames.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "palmtracer-cpp_b200"))
import ptb  # noqa: E402

OFFSET, GAIN = 100.0, 2.0
COLS = 18
PIXEL_NM = 160.0
MAX_DISTANCE = 5.0
ASTIG = [150.0, 400.0, 0.05, 0.0, 1.3 * PIXEL_NM, -150.0, 400.0, -0.05, 0.0, 1.3 * PIXEL_NM]
TABLE_MLE = (25, 25, 121, 10.0)    # cells in x, y, z and z step (nm) of the cubic-spline tables
TABLE_EMCCD = (17, 17, 41, 25.0)

# emitters per pixel: 40 on 256^2, 0.1 / um^2 at 160 nm pixels, 800 on 512^2
SPARSE, DENSE, ASTIG_DENSITY = 40 / 256.0 ** 2, 0.1 * 0.16 ** 2, 800 / 512.0 ** 2


def localize(frames, height, width, fit, roi, density, where, psf="gauss", ratio=0.0, lanes=0, uneven=False):
    """lanes: ROI mapping of the maximum-likelihood fits (modes 6-8), pinned with PTB_MLE_LANES so that a program's
    rows are the same bits in every process (the library's own choice is timed per process)."""
    return {"kind": "localize", "frames": frames, "height": height, "width": width, "fit": fit, "roi": roi,
            "density": density, "where": where, "psf": psf, "ratio": ratio, "lanes": lanes, "uneven": uneven}


def listed():
    def named(name, case):
        return dict(case, name=name)
    return [
        # a live preview: each camera frame localized as it arrives, host buffers, the reference's own Gaussian fit
        named("preview 256 lsq", localize(1, 256, 256, 2, 7, SPARSE, "host")),
        # the same per-frame form on a full sensor with the maximum-likelihood fit
        named("frame 1024 mle", localize(1, 1024, 1024, 6, 7, DENSE, "host", lanes=32)),
        # a short 2D acquisition handed over whole, host buffers
        named("stack 256 mle", localize(200, 256, 256, 6, 7, SPARSE, "host", lanes=8)),
        # batched 2D throughput, frames resident in device memory
        named("batch 1024 mle", localize(500, 1024, 1024, 6, 7, DENSE, "device", lanes=1)),
        # the same frames with the reference's Gaussian least-squares fit
        named("batch 1024 lsq", localize(150, 1024, 1024, 2, 7, DENSE, "device")),
        # astigmatic 3D, maximum likelihood
        named("batch 512 astig", localize(300, 512, 512, 7, 11, ASTIG_DENSITY, "device", psf="astig", lanes=4)),
        # cubic-spline PSF 3D, maximum likelihood, strongly uneven emitter counts per frame
        named("batch 512 spline", localize(150, 512, 512, 8, 13, 750 / 512.0 ** 2, "device", psf="astig",
                                           lanes=16, uneven=True)),
        # a cropped region of odd size with basin fusion and the rotated elliptic fit, host buffers
        named("crop 317x203 fused", localize(37, 203, 317, 4, 9, DENSE, "host", psf="astig", ratio=10.0)),
        # the reference's cubic-spline EMCCD fit
        named("stack 256 emccd", localize(60, 256, 256, 5, 9, SPARSE, "host", psf="astig")),
        # elliptic fits at positions from another detector (widths for a z lookup)
        {"name": "fit positions", "kind": "fit", "frames": 40, "height": 512, "width": 512, "fit": 3, "roi": 9,
         "density": ASTIG_DENSITY / 4, "psf": "astig"},
        # trajectories of a localization table
        {"name": "track 400k", "kind": "track", "planes": 400, "per_plane": 1100, "size": 512.0, "step": 0.8},
        # the detection threshold of a new acquisition, estimated from its first frame
        {"name": "threshold 512", "kind": "threshold", "height": 512, "width": 512, "density": SPARSE},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["localize"] * 6 + ["fit", "fit", "track", "threshold"])
    if kind == "track":
        planes = int(_log(rng, 20, 600))
        return {"kind": "track", "planes": planes, "per_plane": int(min(_log(rng, 30, 3000), 440000 / planes)),
                "size": rng.choice([256.0, 512.0, 1024.0]), "step": round(rng.uniform(0.3, 1.5), 3)}
    height, width = int(_log(rng, 100, 1100)), int(_log(rng, 100, 1100))
    if rng.random() < 0.4:  # sensors and their crops mostly have widths that are multiples of 16
        width = max(112, width // 16 * 16)
    if kind == "threshold":
        return {"kind": "threshold", "height": height, "width": width, "density": _log(rng, SPARSE / 2, DENSE)}
    if kind == "fit":
        density = _log(rng, SPARSE / 2, ASTIG_DENSITY / 4)
        most = min(200.0, 20000 / (density * height * width))
        return {"kind": "fit", "frames": max(1, int(_log(rng, 1, max(1.01, most)))), "height": height, "width": width,
                "fit": rng.choice([1, 2, 3, 4]), "roi": rng.choice([7, 9, 11]), "density": density,
                "psf": rng.choice(["gauss", "astig"])}
    fit = rng.choice([1, 2, 2, 3, 4, 5, 6, 6, 6, 7, 7, 8])
    density = ASTIG_DENSITY if fit == 7 else _log(rng, SPARSE / 2, DENSE if fit != 8 else 750 / 512.0 ** 2)
    roi = {1: 7, 2: 7, 3: 9, 4: 9, 5: 9, 6: 7, 7: 11, 8: 13}[fit]
    pixels = {5: 4e6, 8: 2.5e7}.get(fit, 8e7)
    frames = max(1, int(_log(rng, 1, max(1.01, min(250.0, pixels / (height * width))))))
    count = frames * density * height * width
    return localize(frames, height, width, fit, roi, density, rng.choice(["host", "device"]),
                    psf="gauss" if fit in (1, 2, 6) else "astig", ratio=rng.choice([0.0, 0.0, 0.0, 10.0]),
                    lanes=0 if fit < 6 else ({6: 1, 7: 4, 8: 16}[fit] if count > 20000 else 32), uneven=fit == 8)


# ---- synthetic frames ---------------------------------------------------------------------------------------------
def _frames(seed, frames, height, width, density, psf, uneven=False):
    """([frames, height, width] int16 CUDA tensor of uint16 bit patterns, emitters [n, 4]: frame, x, y, photons)."""
    rng = np.random.default_rng(seed)
    mean = density * height * width
    # emitters per frame: uniform on 0 .. 2 mean, or Poisson with the stack's total given
    counts = rng.integers(0, int(2 * mean) + 1, frames) if uneven else rng.multinomial(round(frames * mean), np.full(frames, 1.0 / frames))
    n = int(counts.sum())
    em = np.empty((n, 6))
    em[:, 0] = np.repeat(np.arange(frames), counts)
    em[:, 1], em[:, 2] = rng.uniform(5.0, width - 5.0, n), rng.uniform(5.0, height - 5.0, n)
    if psf == "astig":
        em[:, 3] = np.exp(rng.uniform(math.log(1000), math.log(10000), n))
        z = rng.uniform(-600.0, 600.0, n)
        u, v = (z - 150.0) / 400.0, (z + 150.0) / 400.0
        em[:, 4] = 1.3 * np.sqrt(1 + u ** 2 + 0.05 * u ** 3)
        em[:, 5] = 1.3 * np.sqrt(1 + v ** 2 - 0.05 * v ** 3)
        bg = torch.full((height, width), 30.0, device="cuda")
    else:
        em[:, 3] = np.exp(rng.uniform(math.log(300), math.log(8000), n))
        em[:, 4] = em[:, 5] = rng.uniform(1.0, 1.6, n)
        cx = torch.cos(2 * math.pi * torch.arange(width, device="cuda") / width)
        cy = torch.cos(2 * math.pi * torch.arange(height, device="cuda") / height)
        bg = 10.0 + 35.0 * (cy[:, None] * cx[None, :] + 1.0)  # 10..80 photons, a smooth cosine field
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    out = torch.empty((frames, height, width), dtype=torch.int16, device="cuda")
    offs = torch.arange(-8, 9, device="cuda", dtype=torch.float64)
    chunk = max(1, min(frames, int(6e7 / (height * width))))
    bounds = np.searchsorted(em[:, 0], np.arange(0, frames + chunk, chunk))

    def axis(centre, pixels, sigma):
        k = 1.0 / (math.sqrt(2.0) * sigma[:, None])
        d = pixels - centre[:, None]
        return 0.5 * (torch.erf((d + 0.5) * k) - torch.erf((d - 0.5) * k))

    for b, c0 in enumerate(range(0, frames, chunk)):
        c1 = min(frames, c0 + chunk)
        e = torch.as_tensor(em[bounds[b]:bounds[b + 1]], device="cuda")
        mu = bg.unsqueeze(0).repeat(c1 - c0, 1, 1).reshape(-1)
        if e.shape[0]:
            xs, ys = e[:, 1].floor()[:, None] + offs, e[:, 2].floor()[:, None] + offs
            val = (e[:, 3, None, None] * axis(e[:, 2], ys, e[:, 5])[:, :, None] * axis(e[:, 1], xs, e[:, 4])[:, None, :])
            inside = ((ys >= 0) & (ys < height))[:, :, None] & ((xs >= 0) & (xs < width))[:, None, :]
            at = ((e[:, 0].long() - c0) * (height * width))[:, None, None] + ys.long()[:, :, None] * width + xs.long()[:, None, :]
            # summed in 2^-20 photon units: an integer sum does not depend on the order of the additions
            mu += torch.zeros(mu.numel(), dtype=torch.int64, device="cuda").index_add_(
                0, at[inside], (val[inside] * 2.0 ** 20).long()).double().mul_(2.0 ** -20).float()
        photons = torch.poisson(mu.reshape(c1 - c0, height, width), generator=gen)
        out[c0:c1] = torch.clamp(OFFSET + GAIN * photons, 0, 65535).to(torch.int32).to(torch.int16)
    return out, em[:, :4]


@functools.lru_cache(maxsize=2)
def _spline_table(nx, ny, nz, dz):
    """Coefficients of the astigmatic PSF's cubic spline, centred on grid point (nx - 1) / 2 as the fits expect."""
    z = (np.arange(nz + 1) - nz / 2.0) * dz
    u, v = (z - 150.0) / 400.0, (z + 150.0) / 400.0
    gx = 1.3 * np.sqrt(np.maximum(1 + u ** 2 + 0.05 * u ** 3, 1e-3))[:, None]
    gy = 1.3 * np.sqrt(np.maximum(1 + v ** 2 - 0.05 * v ** 3, 1e-3))[:, None]
    ex = np.exp(-0.5 * ((np.arange(nx + 1) - (nx - 1) / 2.0) / gx) ** 2) / (math.sqrt(2 * math.pi) * gx)
    ey = np.exp(-0.5 * ((np.arange(ny + 1) - (ny - 1) / 2.0) / gy) ** 2) / (math.sqrt(2 * math.pi) * gy)
    return ptb.spline_coefficients(ey[:, :, None] * ex[:, None, :]).ravel()


def _fit_params(fit, roi):
    if fit == 5:
        return np.concatenate([[float(roi)], TABLE_EMCCD, _spline_table(*TABLE_EMCCD)])
    if fit == 6:
        return np.array([roi, 1.3, OFFSET, GAIN, 20.0, 0.0])
    if fit == 7:
        return np.array([roi, PIXEL_NM] + ASTIG + [OFFSET, GAIN, 20.0, -600.0, 600.0, 0.0])
    if fit == 8:
        return np.concatenate([[float(roi)], TABLE_MLE, [OFFSET, GAIN, 20.0, 0.0], _spline_table(*TABLE_MLE)])
    return np.array([roi, 1.3, 1.3, 0.0])


def _host(frames):
    return frames.cpu().numpy().view(np.uint16)


def prepare(case, seed):
    if case["kind"] == "track":
        return {"case": case, "points": _points(case, seed)}
    if case["kind"] == "threshold":
        frame, _ = _frames(seed, 1, case["height"], case["width"], case["density"], "gauss")
        return {"case": case, "frame": _host(frame)[0], "params": np.array([7.0, 1.3, 1.3, 0.0])}
    shape = (case["frames"], case["height"], case["width"])
    frames, em = _frames(seed, *shape, case["density"], case["psf"], case.get("uneven", False))
    params = _fit_params(case["fit"], case["roi"])
    if case["kind"] == "fit":
        return {"case": case, "stack": _host(frames), "positions": _positions(em, seed), "params": params}
    # the usual detection threshold: 3 x 1.4826 x MAD of the first frame's second wavelet plane
    plane = ptb.wavelett(_host(frames[:1]), 2)[0]
    thr = float(3.0 * 1.4826 * np.median(np.abs(plane - np.median(plane))))
    if case["lanes"]:
        os.environ["PTB_MLE_LANES"] = str(case["lanes"])
    else:
        os.environ.pop("PTB_MLE_LANES", None)
    # rows per plane: room for twice the emitters
    capacity = shape[0] * int(64 + 2 * case["density"] * shape[1] * shape[2]) * COLS
    state = {"case": case, "shape": shape, "thr": thr, "params": params, "capacity": capacity}
    if case["where"] == "host":
        state["stack"], state["out"] = _host(frames), np.zeros(capacity)
    else:
        state["stack"], state["out"] = frames, torch.zeros(capacity, dtype=torch.float64, device="cuda")
    return state


def _positions(em, seed):
    """Positions rows (Id, Plane, X, Y, SegIntensity, Surface): the emitters, found to a third of a pixel."""
    rng = np.random.default_rng(seed + 2)
    pos = np.empty((em.shape[0], 6))
    pos[:, 0], pos[:, 1] = np.arange(1, em.shape[0] + 1), em[:, 0] + 1
    pos[:, 2:4] = em[:, 1:3] + rng.normal(0.0, 0.3, (em.shape[0], 2))
    pos[:, 4], pos[:, 5] = em[:, 3], 20.0
    return pos


def _points(case, seed):
    """Emitters drifting by about `step` px per plane, nine in ten of them seen on each: rows (Id, Plane, X, Y)."""
    rng = np.random.default_rng(seed)
    planes, per = case["planes"], case["per_plane"]
    xy = rng.uniform(0.0, case["size"], (per, 2)) + np.cumsum(rng.normal(0.0, case["step"], (planes, per, 2)), axis=0)
    which = np.sort(np.argsort(rng.random((planes, per)), axis=1)[:, :max(1, int(0.9 * per))], axis=1)
    plane, which = np.repeat(np.arange(planes), which.shape[1]), which.ravel()
    pts = np.empty((plane.size, 4))
    pts[:, 0], pts[:, 1], pts[:, 2:] = np.arange(1, plane.size + 1), plane + 1, xy[plane, which]
    return pts


def run(state):
    case = state["case"]
    if case["kind"] == "track":
        return ptb.tracking(state["points"], MAX_DISTANCE).view(np.int64)
    if case["kind"] == "threshold":
        return ptb.auto_threshold(state["frame"], state["params"])
    if case["kind"] == "fit":
        return ptb.fitting(state["stack"], state["positions"], case["fit"], state["params"])
    if case["where"] == "host":
        n = ptb.localization_raw(state["stack"], state["out"], state["thr"], case["ratio"], case["fit"], state["params"])
    else:
        n = ptb.localization_device(state["stack"].data_ptr(), state["out"].data_ptr(), state["capacity"], state["shape"],
                                    state["thr"], case["ratio"], case["fit"], state["params"],
                                    torch.cuda.current_stream().cuda_stream)
    return {"rows": state["out"], "doubles": n}  # the caller's row buffer, of which the first n doubles are written


def work(case):
    if case["kind"] == "track":
        n = 0.9 * case["planes"] * case["per_plane"]
        return {"bytes": n * 48, "flops": n * 6}
    pixels = case.get("frames", 1) * case["height"] * case["width"]
    if case["kind"] == "threshold":
        return {"bytes": pixels * 2, "flops": 5 * pixels * 40}
    n = pixels * case["density"]
    # model evaluations of a fit and operations per ROI pixel and evaluation: the model and its derivatives, the
    # gradient and the triangle of the curvature matrix
    params, model = {1: (4, 30), 2: (5, 35), 3: (6, 60), 4: (7, 75), 5: (5, 512), 6: (5, 25), 7: (5, 25), 8: (5, 512)}[case["fit"]]
    flops = n * case["roi"] ** 2 * 6 * (model + 2 * params + params * (params + 1))
    if case["kind"] == "fit":
        return {"bytes": n * (case["roi"] ** 2 * 2 + 48 + 144), "flops": flops}
    return {"bytes": pixels * 2 + n * 144, "flops": flops + pixels * 40}


# ---- the same results in plain 64-bit arithmetic ------------------------------------------------------------------
def exact(case, seed):
    """Fitting's rows: the damped least squares of the fit modes 1-4 in batched float64. The other kinds have no value
    here: the candidates of a stack come from a watershed whose frame-wide flood is one serial chain, and tracks and
    a threshold's detections are whole decisions that the comparison of two builds holds to equality."""
    if case["kind"] != "fit":
        return None
    state = prepare(case, seed)
    return _lsq_rows(state["stack"], state["positions"], case["fit"], state["params"])


def _model(mode, p, X, Y, s0, th0):
    """Model and gradient [m, n, np] of the Gaussian fits (lib/fit/GaussianModel.cpp:19-52)."""
    x, y = X - p[:, 2, None], Y - p[:, 3, None]
    one = torch.ones_like(x)
    if mode in (1, 2):
        s = torch.full_like(p[:, :1], s0[0]) if mode == 1 else p[:, 4, None]
        r2 = x * x + y * y
        e = torch.exp(-r2 / (2 * s * s))
        P = p[:, 1, None] * e
        g = [one, e, P * x / s ** 2, P * y / s ** 2] + ([P * r2 / s ** 3] if mode == 2 else [])
    else:
        th = torch.full_like(p[:, :1], th0) if mode == 3 else p[:, 6, None]
        sx, sy, c, s = p[:, 4, None], p[:, 5, None], torch.cos(th), torch.sin(th)
        a, b = x * c - y * s, x * s + y * c
        e = torch.exp(-(a / sx) ** 2 - (b / sy) ** 2)
        P = p[:, 1, None] * e
        # d/dx0 and d/dy0 of the exponent with the reference's signs
        gx = P * (2 * c * (c * x - s * y) / sx ** 2 + 2 * s * (s * x + c * y) / sy ** 2)
        gy = P * (2 * s * (s * y - c * x) / sx ** 2 + 2 * c * (c * y + s * x) / sy ** 2)
        g = [one, e, gx, gy, P * 2 * a * a / sx ** 3, P * 2 * b * b / sy ** 3]
        if mode == 4:
            f4 = 2 * x * y / sx ** 2 - 2 * x * y / sy ** 2
            g.append(P * (2 * c * s * ((x * x - y * y) / sx ** 2 + (y * y - x * x) / sy ** 2) - s * s * f4 + c * c * f4))
    return P + p[:, 0, None], torch.stack(g, -1)


def _lsq_rows(stack, pos, mode, params):
    dev = "cuda"
    roi = int(params[0])
    h, n = roi // 2, pos.shape[0]
    frames, height, width = stack.shape
    rows = torch.zeros((n, COLS), dtype=torch.float64, device=dev)
    q = torch.as_tensor(pos, device=dev)
    ux, uy, f = q[:, 2].long(), q[:, 3].long(), q[:, 1].long() - 1
    ok = (q[:, 2] >= 0) & (q[:, 3] >= 0) & (ux >= h) & (uy >= h) & (ux < width - h) & (uy < height - h)
    rows[:, 0:2], rows[:, 4:6] = q[:, 0:2], q[:, 2:4]
    rank = np.zeros(n)
    for k in range(frames):
        at = np.nonzero(pos[:, 1] == k + 1)[0]
        rank[at] = np.arange(1, at.size + 1)
    rows[:, 2] = torch.as_tensor(rank, device=dev)
    rows[:, 3], rows[:, 6], rows[:, 17] = -1, 0, 1
    rows[:, 7:15] = -1
    rows[:, 15:17] = q[:, 4:6]
    sel = ok.nonzero()[:, 0]
    d = torch.arange(-h, h + 1, device=dev)
    yi = (uy[sel, None, None] + d[:, None]).expand(-1, roi, roi).reshape(-1, roi * roi)
    xi = (ux[sel, None, None] + d[None, :]).expand(-1, roi, roi).reshape(-1, roi * roi)
    img = torch.as_tensor(stack.astype(np.int32), device=dev)
    v = img[f[sel, None], yi, xi].double()
    X, Y = xi.double(), yi.double()
    m, x0, y0 = sel.numel(), q[sel, 2], q[sel, 3]
    s0, th0 = params[1:3], float(params[3])
    start = [v.amin(1), v.amax(1) - v.amin(1), x0, y0]
    lo, hi = [0.0, 0.0, x0 - 1, y0 - 1], [65535.0, 65535.0, x0 + 1, y0 + 1]
    if mode == 2:
        start, lo, hi = start + [s0[0]], lo + [0.1], hi + [20.0]
    if mode >= 3:
        r2 = math.sqrt(2.0)
        start, lo, hi = start + [r2 * s0[0], r2 * s0[1]], lo + [0.1, 0.1], hi + [20.0, 20.0]
    if mode == 4:
        start, lo, hi = start + [th0], lo + [-150.0], hi + [150.0]

    def columns(c):
        return torch.stack([a if torch.is_tensor(a) else torch.full((m,), float(a), dtype=torch.float64, device=dev) for a in c], 1)

    p, lo, hi = columns(start), columns(lo), columns(hi)
    npar = p.shape[1]

    def normal(pp):
        hat, g = _model(mode, pp, X, Y, s0, th0)
        if mode == 4:
            g[(pp[:, 4] - pp[:, 5]).abs() <= 2.220446049250313e-16, :, 6] = 0.0
        r = v - hat
        return (r * r).sum(1), (g * r[..., None]).sum(1), g.transpose(1, 2) @ g

    err, beta, alpha = normal(p)
    lam = torch.full((m,), 1e-2, dtype=torch.float64, device=dev)
    dp = torch.zeros_like(p)
    live = beta.abs().amax(1) >= 1e-6
    diag = torch.arange(npar, device=dev)
    for it in range(75):
        if not bool(live.any()):
            break
        A = alpha.clone()
        dg = alpha[:, diag, diag]
        A[:, diag, diag] = torch.where(dg == 0, torch.ones_like(dg), (1 + lam[:, None]) * dg)
        step = torch.linalg.solve_ex(A, beta)[0]
        trial = torch.minimum(torch.maximum(p + step, lo), hi)
        move = torch.where(live[:, None], trial - p, dp)
        tiny = (move.abs() < 1e-15).all(1)
        gain = 2 * (move * beta).sum(1) - (move * (alpha @ move[..., None])[..., 0]).sum(1)
        uphill = gain <= 0
        e2, b2, a2 = normal(trial)
        rho = (err - e2) / (2 * (move * (lam[:, None] * move + beta)).sum(1))
        moved = live & ~tiny & ~uphill & (rho > 1e-2)
        dp = move
        end = live & ~moved & (lam >= 1e7)
        p = torch.where(moved[:, None], trial, p)
        err, beta, alpha = torch.where(moved, e2, err), torch.where(moved[:, None], b2, beta), torch.where(moved[:, None, None], a2, alpha)
        lam = torch.where(live, torch.where(moved, (lam / 9).clamp_min(1e-7), (lam * 11).clamp_max(1e7)), lam)
        if it >= 2:
            small = (dp.abs() / p.abs().clamp_min(1e-12)).amax(1) < 1e-6
            done = small | (~uphill & ((err / (roi * roi) < 1e-5) | (beta.abs().amax(1) < 1e-6)))
            end = end | (live & ~tiny & done)
        live = live & ~end
    hat, _ = _model(mode, p, X, Y, s0, th0)
    dv, dm = v - v.mean(1, keepdim=True), hat - hat.mean(1, keepdim=True)
    quality = ((dv * dm).sum(1) / torch.sqrt((dv * dv).sum(1) * (dm * dm).sum(1))).nan_to_num(0.0) ** 2
    good = quality >= 1e-7
    rows[sel, 4], rows[sel, 5] = p[:, 2], p[:, 3]
    if mode <= 2:
        sx = sy = torch.full_like(quality, s0[0]) if mode == 1 else p[:, 4]
    else:
        sx, sy = p[:, 4] / math.sqrt(2.0), p[:, 5] / math.sqrt(2.0)
    th = p[:, 6] if mode == 4 else torch.full_like(quality, th0 if mode == 3 else 0.0)
    vals = {7: torch.where((p[:, 1] > 1e-7) & (sx > 1e-7) & (sy > 1e-7), 2 * math.pi * p[:, 1] * sx * sy, -torch.ones_like(sx)),
            8: sx, 9: sy, 10: th, 11: quality, 13: p[:, 1], 14: p[:, 0],
            17: torch.where((sx > 1e-7) & (sy > 1e-7), torch.minimum(sx, sy) / torch.maximum(sx, sy), torch.ones_like(sx))}
    for c, val in vals.items():
        rows[sel[good], c] = val[good]
    return rows.cpu().numpy()
