"""What this framework is timed on: the calls its users make, through the public entry points.

Each case is a dict of plain values.  ``listed()`` holds the fixed ones, ``draw(rng)`` makes more of the same
ranges, ``prepare`` builds a user's inputs and the plan or weights such a program keeps, ``run`` makes one pass,
``work`` counts what a pass cannot do without and ``exact`` gives a pass's outputs in 64 bits from plain torch.

The kinds:

* ``fan``      a forward projection and a backprojection on one plan (distance-driven or Siddon), one slice or a
               ragged batch of slices: the step of every iterative solver;
* ``fan_grad`` the projector as a differentiable layer, forward and backward, on multi-row, multi-channel batches;
* ``host``     the same pair through the host (numpy) class that scripts written for the reference call;
* ``fbp``      short-scan filtered backprojection: weights, ramp filter, pixel-driven backprojection;
* ``ossqs``    iterations of the TV-regularised ordered-subset solver on a ragged batch;
* ``tomo``     the flat-detector distance-driven pair of tomosynthesis, on device pointers;
* ``cone``     the Siddon cone-beam pair with per-view geometry, on a tomosynthesis arc or a circular orbit;
* ``cyl``      the cylindrical-detector cone-beam pair, on an ordered subset of a full scan's views;
* ``cnn``      the convolutional prior: a training step's output and gradients, or a denoising pass.

Images are sums of random ellipsoids (semi-axes 5-120 mm, attenuation 0-0.04/mm) and the measured data are their
line integrals with Poisson noise, as in ``reconnet_b200.phantom``.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

PITCH = 1.2858 / 1085.6     # the arc detector's angular pitch
DSD, DSO = 1085.6, 595.0    # source to detector, source to isocentre (mm)
START = 0.0123              # gantry angle of the first view
MM5, MM120 = 5.0, 120.0     # ellipsoid semi-axes


def listed():
    return [
        # one small slice: plan.project + plan.backproject of an interactive or per-slice program, where launches
        # and the few thread blocks of a single slice count
        {"name": "fan_one_slice", "kind": "fan", "projector": "dd", "slices": 1, "nx": 256, "ny": 256, "dx": 1.0,
         "nu": 736, "views": 720, "views_max": 720, "bp": 2, "off_a": 0.0},
        # the large batch: 64 independent 512 x 512 slices, each with its own number of views
        {"name": "fan_batch", "kind": "fan", "projector": "dd", "slices": 64, "nx": 512, "ny": 512, "dx": 0.7,
         "nu": 888, "views": 576, "views_max": 1152, "bp": 2, "off_a": 0.0},
        # a projection layer inside a network: odd sizes, detector rows and channels, an off-centre detector, the
        # reference's registered gradient (its iterative backprojection)
        {"name": "fan_layer_odd", "kind": "fan_grad", "batch": 2, "channels": 2, "nz": 3, "nx": 301, "ny": 333,
         "dx": 0.9, "nu": 611, "views": 413, "bp": 0, "off_a": 0.25},
        # the Siddon pair, the projector of the reference's own solver, on a ragged batch
        {"name": "siddon_batch", "kind": "fan", "projector": "siddon", "slices": 8, "nx": 512, "ny": 512, "dx": 0.7,
         "nu": 888, "views": 576, "views_max": 1152, "bp": 3, "off_a": 0.0},
        # a drop-in call pair on host arrays, at the host class's own defaults
        {"name": "host_slice", "kind": "host", "nx": 512, "ny": 512, "dx": 1.0, "nu": 736, "views": 720, "bp": 0},
        # short-scan reconstruction of a stack of slices
        {"name": "fbp_stack", "kind": "fbp", "slices": 16, "nx": 512, "ny": 512, "dx": 0.7, "nu": 888, "views": 701,
         "filter": 0},
        # one iteration of the iterative solver, 24 subsets: many launches on small shares of the views
        {"name": "ossqs_tv", "kind": "ossqs", "slices": 16, "nx": 512, "ny": 512, "dx": 0.7, "nu": 888, "views": 576,
         "views_max": 1152, "subsets": 24, "iterations": 1},
        # tomosynthesis, distance driven
        {"name": "tomo_dd", "kind": "tomo", "nx": 512, "ny": 512, "nz": 128, "dx": 0.8, "dz": 1.0, "nu": 736,
         "nv": 736, "du": 0.6, "views": 25},
        # tomosynthesis, ray lengths
        {"name": "tomo_siddon", "kind": "cone", "orbit": "arc", "nx": 512, "ny": 512, "nz": 128, "dx": 0.8, "dz": 1.0,
         "nu": 736, "nv": 736, "du": 0.6, "dv": 0.6, "views": 25},
        # a flat detector on a circular orbit, ray lengths
        {"name": "cone_circular", "kind": "cone", "orbit": "circle", "nx": 256, "ny": 256, "nz": 128, "dx": 1.0,
         "dz": 1.0, "nu": 512, "nv": 128, "du": 1.3, "dv": 1.5, "views": 90},
        # one of eight ordered subsets of a 984-view cone-beam scan
        {"name": "cone_cylinder", "kind": "cyl", "nx": 512, "ny": 512, "nz": 128, "dx": 0.8, "dz": 1.0, "nu": 736,
         "nv": 64, "views": 123},
        # a training step of the convolutional prior at its training batch
        {"name": "cnn_train", "kind": "cnn", "images": 8, "h": 512, "w": 512, "train": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fan", "fan", "fan_grad", "host", "fbp", "ossqs", "tomo", "cone", "cone", "cyl", "cnn"])
    nx, ny = _log(rng, 128, 512), _log(rng, 128, 512)
    dx = round(min(rng.uniform(0.5, 1.2), 380.0 / max(nx, ny)), 3)
    views, nu = _log(rng, 90, 900), rng.randint(300, 888)
    flat = {"nx": _log(rng, 128, 400), "ny": _log(rng, 128, 400), "nz": _log(rng, 24, 128),
            "dx": round(rng.uniform(0.7, 0.9), 3), "dz": round(rng.uniform(0.8, 1.2), 3)}
    if kind == "fan":
        projector = rng.choice(["dd", "dd", "siddon"])
        return {"kind": kind, "projector": projector, "slices": _log(rng, 1, 24 if projector == "dd" else 6),
                "nx": nx, "ny": ny, "dx": dx, "nu": nu, "views": views, "views_max": int(views * rng.uniform(1, 1.25)),
                "bp": rng.choice([0, 1, 2, 2]) if projector == "dd" else 3, "off_a": round(rng.uniform(-2, 2), 3)}
    if kind == "fan_grad":
        return {"kind": kind, "batch": rng.randint(1, 4), "channels": rng.randint(1, 3), "nz": rng.randint(1, 4),
                "nx": nx, "ny": ny, "dx": dx, "nu": nu, "views": min(views, 500), "bp": rng.choice([0, 2]),
                "off_a": round(rng.uniform(-2, 2), 3)}
    if kind == "host":
        return {"kind": kind, "nx": nx, "ny": ny, "dx": dx, "nu": nu, "views": views, "bp": rng.choice([0, 1, 2])}
    if kind == "fbp":
        return {"kind": kind, "slices": _log(rng, 1, 16), "nx": nx, "ny": ny, "dx": dx, "nu": nu, "views": views,
                "filter": rng.randint(0, 3)}
    if kind == "ossqs":
        return {"kind": kind, "slices": _log(rng, 2, 16), "nx": nx, "ny": ny, "dx": dx, "nu": nu, "views": views,
                "views_max": int(views * rng.uniform(1, 1.25)), "subsets": rng.choice([8, 12, 24]), "iterations": 1}
    if kind == "tomo":
        return {"kind": kind, **flat, "nu": rng.randint(200, 700), "nv": rng.randint(200, 700),
                "du": round(rng.uniform(0.5, 0.8), 3), "views": rng.randint(5, 25)}
    if kind == "cone" and rng.random() < 0.5:
        return {"kind": kind, "orbit": "arc", **flat, "nu": rng.randint(200, 700), "nv": rng.randint(200, 700),
                "du": round(rng.uniform(0.5, 0.8), 3), "dv": round(rng.uniform(0.5, 0.8), 3),
                "views": rng.randint(5, 25)}
    if kind == "cone":
        n = _log(rng, 96, 256)
        return {"kind": kind, "orbit": "circle", **flat, "nx": n, "ny": n + rng.randint(-7, 7), "nz": _log(rng, 24, 96),
                "nu": rng.randint(200, 512), "nv": rng.randint(32, 128), "du": round(rng.uniform(1.0, 1.4), 3),
                "dv": round(rng.uniform(1.0, 1.6), 3), "views": rng.randint(24, 90)}
    if kind == "cyl":
        return {"kind": kind, **flat, "nu": rng.randint(300, 736), "nv": rng.randint(16, 64),
                "views": rng.randint(24, 123)}
    return {"kind": "cnn", "images": rng.randint(1, 8), "h": _log(rng, 96, 512), "w": _log(rng, 96, 512),
            "train": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _ellipsoids(rng, count, fov_x, fov_y, fov_z):
    """count sets of 10 ellipsoids: centre, semi-axes, in-plane angle, attenuation; flat (2D) where fov_z is 0."""
    size = (count, 10)
    r = 0.4 * min(fov_x, fov_y) * np.sqrt(rng.uniform(size=size))
    th = rng.uniform(0, 2 * np.pi, size)
    ax = rng.uniform(MM5, MM120, size + (3,))
    ax[..., 2] = rng.uniform(MM5, max(2 * MM5, fov_z / 2), size) if fov_z else 1e9
    return {"c": np.stack([r * np.cos(th), r * np.sin(th), rng.uniform(-0.4, 0.4, size) * fov_z], -1), "ax": ax,
            "ang": rng.uniform(0, np.pi, size), "mu": rng.uniform(0, 0.04, size)}


def _image(ell, nx, ny, nz, dx, dy, dz):
    """[count, nx, ny, nz] float32 images of the ellipsoid sets on a centred grid."""
    dev = _device()

    def axis(n, d):
        return (torch.arange(n, device=dev, dtype=torch.float32) - (n - 1) / 2.0) * d

    x, y, z = axis(nx, dx)[:, None, None], axis(ny, dy)[None, :, None], axis(nz, dz)[None, None, :]
    count = ell["mu"].shape[0]
    img = torch.zeros((count, nx, ny, nz), device=dev)
    for s in range(count):
        for k in range(10):
            (cx, cy, cz), (a, b, c) = ell["c"][s, k], ell["ax"][s, k]
            co, si = math.cos(ell["ang"][s, k]), math.sin(ell["ang"][s, k])
            u, v, w = ((x - cx) * co + (y - cy) * si) / a, ((y - cy) * co - (x - cx) * si) / b, (z - cz) / c
            img[s] += ((u * u + v * v) + w * w <= 1.0) * float(ell["mu"][s, k])
    return img


def _lines(ell, s, src, dst):
    """Line integrals of ellipsoid set s along rays src -> dst (mm, broadcastable triples of tensors)."""
    d = [q - p for p, q in zip(src, dst)]
    norm = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    total = 0.0
    for k in range(10):
        c, ax = ell["c"][s, k], ell["ax"][s, k]
        co, si = math.cos(ell["ang"][s, k]), math.sin(ell["ang"][s, k])
        p = [src[i] - float(c[i]) for i in range(3)]
        pe = [(p[0] * co + p[1] * si) / ax[0], (p[1] * co - p[0] * si) / ax[1], p[2] / ax[2]]
        de = [(d[0] * co + d[1] * si) / ax[0], (d[1] * co - d[0] * si) / ax[1], d[2] / ax[2]]
        a = de[0] * de[0] + de[1] * de[1] + de[2] * de[2]
        b = pe[0] * de[0] + pe[1] * de[1] + pe[2] * de[2]
        e = pe[0] * pe[0] + pe[1] * pe[1] + pe[2] * pe[2] - 1.0
        total = total + torch.sqrt((b * b - a * e).clamp_min(0)) / a * (2 * float(ell["mu"][s, k]))
    return total * norm


def _measure(line, seed, i0=5e4):
    """Noisy log data and the photon counts (the statistical weights) of line integrals."""
    gen = torch.Generator(device=line.device).manual_seed(int(seed) * 7919 + 17)
    counts = torch.poisson(i0 * torch.exp(-line.double()), generator=gen).clamp_min(1.0)
    return (-torch.log(counts / i0)).float(), counts.float()


def _fan_lines(ell, s, angles, nu, off_a, da=PITCH):
    """[nu, nview] fan-beam line integrals of set s: source (dso sin t, -dso cos t), cell u at fan angle
    (-(u - (nu-1)/2) - off_a) da."""
    dev = _device()
    t = torch.as_tensor(np.asarray(angles, np.float64), device=dev)[None, :]
    a = ((-(torch.arange(nu, device=dev, dtype=torch.float64) - (nu - 1) / 2.0) - off_a) * da)[:, None]
    src = (DSO * torch.sin(t), -DSO * torch.cos(t), torch.zeros_like(t))
    dst = (src[0] + DSD * torch.sin(a - t), src[1] + DSD * torch.cos(a - t), torch.zeros_like(t))
    return _lines(ell, s, src, dst)


def _angles(n, span=2 * math.pi):
    return (START + np.arange(n) * span / n).astype(np.float32)


def _view_counts(case):
    """The slices' view counts: a property of the case, whatever the inputs."""
    lo, hi = case["views"], max(case["views"], case["views_max"])
    return np.random.default_rng(1).integers(lo, hi + 1, size=case["slices"]).astype(np.int32)


def _fan_geometry(case, **more):
    from reconnet_b200.geometry import FanGeometry
    return FanGeometry(nx=case["nx"], ny=case["ny"], dx=case["dx"], dy=case["dx"], nu=case["nu"], da=PITCH, dsd=DSD,
                       dso=DSO, off_a=case.get("off_a", 0.0), **more)


def _slices(case, seed, count):
    rng = np.random.default_rng(seed)
    ell = _ellipsoids(rng, count, case["nx"] * case["dx"], case["ny"] * case["dx"], 0.0)
    return ell, _image(ell, case["nx"], case["ny"], 1, case["dx"], case["dx"], 1.0)[..., 0]


def _ragged_data(case, seed):
    """Images [S, nx, ny], concatenated angles, and the packed noisy data and weights of a ragged batch."""
    counts = _view_counts(case)
    ell, img = _slices(case, seed, case["slices"])
    ang = [_angles(n) for n in counts]
    off_a = case.get("off_a", 0.0)
    line = torch.cat([_fan_lines(ell, s, ang[s], case["nu"], off_a).reshape(-1) for s in range(case["slices"])])
    b, w = _measure(line, seed)
    return counts, img, np.concatenate(ang), b, w


def _stack_data(case, seed, angles, count):
    """Images [count, nx, ny] and noisy data [count, nu, nview] of slices that share their angles."""
    ell, img = _slices(case, seed, count)
    line = torch.stack([_fan_lines(ell, s, angles, case["nu"], case.get("off_a", 0.0)) for s in range(count)])
    return img, _measure(line, seed)[0]


def _fan_grad_data(case, seed):
    """Image [B, nx, ny, nz, C] and a data-like cotangent [B, nu, nview, nz, C]."""
    n = case["batch"] * case["nz"] * case["channels"]
    img, b = _stack_data(case, seed, _angles(case["views"]), n)
    fold = (case["batch"], case["nz"], case["channels"])
    img = img.reshape(*fold, case["nx"], case["ny"]).permute(0, 3, 4, 1, 2).contiguous()
    return img, b.reshape(*fold, case["nu"], case["views"]).permute(0, 3, 4, 1, 2).contiguous()


def _short_scan(case):
    """View angles of a short scan of 180 degrees plus the fan."""
    return (np.arange(case["views"]) * (math.pi + 1.05 * case["nu"] * PITCH) / (case["views"] - 1)).astype(np.float32)


def _flat_views(case):
    """(detCenter, detU, detV, src), each [views, 3]: sources on a +-20 degree arc at 650 mm over a fixed detector
    80 mm below the isocentre, or a circular orbit with the detector opposite the source."""
    n = case["views"]
    if case.get("orbit", "arc") == "arc":
        a = np.radians(np.linspace(-20, 20, n)) if n > 1 else np.zeros(1)
        zero, one = np.zeros(n), np.ones(n)
        dc = np.stack([zero, zero, -80 * one], 1)
        du, dv = np.stack([one, zero, zero], 1), np.stack([zero, one, zero], 1)
        src = np.stack([650 * np.sin(a), zero, 650 * np.cos(a)], 1)
    else:
        t = START + np.arange(n) * 2 * np.pi / n
        zero, one = np.zeros(n), np.ones(n)
        src = np.stack([DSO * np.sin(t), -DSO * np.cos(t), zero], 1)
        dc = np.stack([-(DSD - DSO) * np.sin(t), (DSD - DSO) * np.cos(t), zero], 1)
        du, dv = np.stack([np.cos(t), np.sin(t), zero], 1), np.stack([zero, zero, one], 1)
    return [np.ascontiguousarray(v, np.float32) for v in (dc, du, dv, src)]


def _flat_cells(case, views):
    """Source and cell-centre coordinates (float64 triples broadcasting to [nu, views, nv])."""
    dev = _device()
    dc, du, dv, src = (torch.as_tensor(v, device=dev).double()[None, :, None, :] for v in views)
    u = ((torch.arange(case["nu"], device=dev) - (case["nu"] - 1) / 2.0) * case["du"]).double()[:, None, None, None]
    v = ((torch.arange(case["nv"], device=dev) - (case["nv"] - 1) / 2.0) * case.get("dv", case["du"])).double()
    dst = dc + du * u + dv * v[None, None, :, None]
    return [src[..., i] for i in range(3)], [dst[..., i] for i in range(3)]


def _volume(case, seed):
    ell = _ellipsoids(np.random.default_rng(seed), 1, case["nx"] * case["dx"], case["ny"] * case["dx"],
                      case["nz"] * case["dz"])
    return ell, _image(ell, case["nx"], case["ny"], case["nz"], case["dx"], case["dx"], case["dz"])


def _flat_data(case, seed):
    ell, vol = _volume(case, seed)
    views = _flat_views(case)
    src, dst = _flat_cells(case, views)
    line = torch.stack([_lines(ell, 0, [c[:, k] for c in src], [c[:, k] for c in dst])
                        for k in range(case["views"])], 1)
    return vol[..., None], _measure(line, seed)[0][None, ..., None].contiguous(), views


def _cyl_geometry(case):
    from reconnet_b200.geometry import CylGeometry
    return CylGeometry(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=case["dx"], dy=case["dx"], dz=case["dz"],
                       nu=case["nu"], nv=case["nv"], da=PITCH, dv=1.0, dsd=DSD, dso=DSO)


def _cyl_data(case, seed):
    dev = _device()
    ell, vol = _volume(case, seed)
    t = torch.as_tensor(_angles(case["views"]).astype(np.float64), device=dev)[None, :, None]
    a = (-(torch.arange(case["nu"], device=dev).double() - (case["nu"] - 1) / 2.0) * PITCH)[:, None, None]
    h = (torch.arange(case["nv"], device=dev).double() - (case["nv"] - 1) / 2.0)[None, None, :]
    src = [DSO * torch.sin(t), -DSO * torch.cos(t), torch.zeros_like(t)]
    dst = [src[0] + DSD * torch.sin(a - t), src[1] + DSD * torch.cos(a - t), h]
    return vol, _measure(_lines(ell, 0, src, dst), seed)[0][None].contiguous()


def _cnn_data(case, seed):
    """Weights of the network (FP32 masters), a noisy input and its clean target, in the network's units."""
    rng = np.random.default_rng(seed)
    state = {"scale": np.float64(50.0)}
    for i, (co, ci) in enumerate([(32, 1), (32, 32), (32, 32), (32, 32), (1, 32)]):
        std = math.sqrt(2.0 / (9 * ci)) * (0.1 if i == 4 else 1.0)
        state["w%d" % i] = (rng.standard_normal((co, 3, 3, ci)) * std).astype(np.float32)
        state["b%d" % i] = (rng.standard_normal(co) * 0.02).astype(np.float32)
    ell = _ellipsoids(rng, case["images"], case["h"] * 0.7, case["w"] * 0.7, 0.0)
    clean = _image(ell, case["h"], case["w"], 1, 0.7, 0.7, 1.0)[..., 0] * 50.0
    gen = torch.Generator(device=clean.device).manual_seed(int(seed) + 3)
    noise = torch.randn(clean.shape, generator=gen, device=clean.device)
    return state, clean + 0.15 * noise, clean


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fan":
        from reconnet_b200.torch_ops import FanPlan
        counts, img, ang, b, _ = _ragged_data(case, seed)
        geom = _fan_geometry(case)
        if case["slices"] == 1:
            plan = FanPlan(geom, ang)
            img, b = img[..., None, None].contiguous(), b.reshape(1, geom.nu, int(counts[0]), 1, 1)
        else:
            plan = FanPlan(geom, ang, nbatches=case["slices"], nview_per_slice=counts)
        return {"case": case, "plan": plan, "img": img, "sino": b}
    if kind == "fan_grad":
        from reconnet_b200.torch_ops import FanPlan
        img, cot = _fan_grad_data(case, seed)
        geom = _fan_geometry(case, nz=case["nz"], nv=case["nz"])
        plan = FanPlan(geom, _angles(case["views"]), nbatches=case["batch"], nchannels=case["channels"])
        return {"case": case, "plan": plan, "img": img.requires_grad_(True), "cot": cot}
    if kind == "host":
        from reconnet_b200.reconnet import ReconNet
        r = ReconNet()
        r.nx, r.ny, r.dx, r.dy, r.nu, r.rotview = case["nx"], case["ny"], case["dx"], case["dx"], case["nu"], case["views"]
        ang = _angles(case["views"])
        r.angles = ang.tolist()
        img, b = _stack_data(case, seed, ang, 1)
        return {"case": case, "rec": r, "img": img.cpu().numpy()[..., None, None],
                "sino": b.cpu().numpy()[..., None, None]}
    if kind == "fbp":
        from reconnet_b200.torch_ops import FanPlan, shortscan_weights
        geom, ang = _fan_geometry(case), _short_scan(case)
        b = _stack_data(case, seed, ang, case["slices"])[1]
        weights = shortscan_weights(torch.from_numpy(ang).cuda(), geom, "parker")
        return {"case": case, "plan": FanPlan(geom, ang, nbatches=case["slices"]), "geom": geom, "weights": weights,
                "sino": b[..., None, None].contiguous()}
    if kind == "ossqs":
        from reconnet_b200.learned_prior import tv_weight
        from reconnet_b200.ossqs import BatchedOSSQS
        counts, img, ang, b, w = _ragged_data(case, seed)
        solver = BatchedOSSQS(_fan_geometry(case), counts, ang, b, w, n_subsets=case["subsets"], lb=0.0)
        solver.set_beta(tv_weight(solver))
        return {"case": case, "solver": solver, "x0": torch.zeros_like(img)}
    if kind == "tomo":
        from reconnet_b200 import _native as N
        vol, prj, (dc, _, _, src) = _flat_data(case, seed)
        sizes = ctypes.c_size_t(), ctypes.c_size_t()
        N.check(N.lib.rn_tomo_sat_bytes(case["nx"], case["ny"], case["nz"], case["nu"], case["views"], case["nv"],
                                        ctypes.byref(sizes[0]), ctypes.byref(sizes[1])))
        sat = torch.empty(max(s.value for s in sizes) // 8 + 1, dtype=torch.float64, device=vol.device)
        return {"case": case, "lib": N, "vol": vol.contiguous(), "prj": prj, "sat": sat,
                "dc": torch.from_numpy(dc).to(vol.device), "src": torch.from_numpy(src).to(vol.device)}
    if kind == "cone":
        from reconnet_b200.torch_ops import ConeGeometry, ConePlan
        vol, prj, views = _flat_data(case, seed)
        geom = ConeGeometry(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=case["dx"], dy=case["dx"], dz=case["dz"],
                            nu=case["nu"], nv=case["nv"], du=case["du"], dv=case["dv"])
        return {"case": case, "plan": ConePlan(geom, *views), "vol": vol.contiguous(), "prj": prj}
    if kind == "cyl":
        from reconnet_b200.torch_ops import CylPlan
        vol, prj = _cyl_data(case, seed)
        return {"case": case, "plan": CylPlan(_cyl_geometry(case), _angles(case["views"]),
                                              device=torch.device("cuda", torch.cuda.current_device())),
                "vol": vol, "prj": prj}
    from reconnet_b200.learned_prior import PriorCNN
    state, noisy, clean = _cnn_data(case, seed)
    net = PriorCNN()
    net.load_state_dict(state)
    return {"case": case, "net": net, "noisy": noisy, "clean": clean}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fan":
        plan = state["plan"]
        return [plan.project(state["img"], siddon=case["projector"] == "siddon"),
                plan.backproject(state["sino"], case["bp"])]
    if kind == "fan_grad":
        from reconnet_b200.torch_ops import fan_project
        y = fan_project(state["img"], state["plan"], case["bp"])
        return [y.detach(), torch.autograd.grad(y, state["img"], state["cot"])[0]]
    if kind == "host":
        r = state["rec"]
        return [r.cDDFanProjection4d(state["img"]),
                r.cDDFanBackprojection4d(state["sino"], type_projector=case["bp"])]
    if kind == "fbp":
        from reconnet_b200.torch_ops import fbp
        return [fbp(state["sino"], state["plan"], state["geom"], case["filter"], weights=state["weights"])]
    if kind == "ossqs":
        return [state["solver"].run(state["x0"], case["iterations"])]
    if kind == "tomo":
        lib, vol, prj = state["lib"].lib, state["vol"], state["prj"]
        out_p, out_v = torch.empty_like(prj), torch.empty_like(vol)
        geo = (1, 1, case["nx"], case["ny"], case["nz"], case["dx"], case["dx"], case["dz"], 0.0, 0.0, 0.0,
               case["nu"], case["views"], case["nv"], case["du"], case["du"], 0.0, 0.0)
        st = torch.cuda.current_stream().cuda_stream
        fixed = state["dc"].data_ptr(), state["src"].data_ptr(), state["sat"].data_ptr()
        state["lib"].check(lib.rn_tomo_project(out_p.data_ptr(), vol.data_ptr(), *fixed, *geo, st))
        state["lib"].check(lib.rn_tomo_backproject(out_v.data_ptr(), prj.data_ptr(), *fixed, *geo, 1, st))
        return [out_p, out_v]
    if kind in ("cone", "cyl"):
        return [state["plan"].project(state["vol"]), state["plan"].backproject(state["prj"])]
    net = state["net"]
    if not case["train"]:
        return [net.denoise(state["noisy"] / 50.0)]
    out, acts = net.forward(state["noisy"], keep=True)
    diff = out - state["clean"]
    dws, dbs = net.backward(acts, ((2.0 / diff.numel()) * diff).contiguous())
    return [out, dws, dbs]


# ---------------------------------------------------------------------------
# What a pass cannot do without: each input read once, each output written once; one footprint integral per ray
# and image line (forward) or pixel and view (back) at 4 operations, one rectangle per ray or voxel and plane at 8
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "cnn":
        px = case["images"] * case["h"] * case["w"]
        layers = 2 * 9 * px * (2 * 32 + 3 * 32 * 32)
        return {"bytes": 4.0 * px * (3 if case["train"] else 2), "flops": float(layers * (3 if case["train"] else 1))}
    if kind in ("fan", "fan_grad", "host", "fbp", "ossqs"):
        if "views_max" in case:
            views = int(_view_counts(case).sum())
            slices = case["slices"]
        else:
            slices = case.get("slices", case.get("batch", 1) * case.get("nz", 1) * case.get("channels", 1))
            views = slices * case["views"]
        img, sino = slices * case["nx"] * case["ny"], views * case["nu"]
        fp = 4.0 * sino * (case["nx"] + case["ny"]) / 2
        bp = 4.0 * views * case["nx"] * case["ny"]
        if kind == "fbp":
            n = 2.0 ** math.ceil(math.log2(2 * case["nu"] - 1))
            return {"bytes": 4.0 * (img + sino), "flops": bp + views * 5.0 * n * math.log2(n)}
        if kind == "ossqs":
            return {"bytes": 4.0 * case["iterations"] * (2 * img + 2 * sino), "flops": case["iterations"] * (fp + bp)}
        return {"bytes": 8.0 * (img + sino), "flops": fp + bp}
    vox, cells = case["nx"] * case["ny"] * case["nz"], case["views"] * case["nu"] * case["nv"]
    planes = case["nz"] if kind == "tomo" or case.get("orbit") == "arc" else (case["nx"] + case["ny"]) / 2
    return {"bytes": 8.0 * (vox + cells), "flops": 8.0 * cells * planes + 8.0 * vox * case["views"]}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------
def _fetch(table, pos):
    """Rows of prefix sums [rows, n + 1] read at positions [..., rows], clamped, linear in between."""
    n = table.shape[1] - 1
    p = pos.clamp(0, n)
    i = p.floor().clamp_(max=n - 1)
    p = p - i
    i = i.long() + torch.arange(table.shape[0], device=pos.device) * (n + 1)
    lo = table.reshape(-1).take(i)
    return lo + p * (table.reshape(-1).take(i + 1) - lo)


def _put(table, pos, val):
    """Transpose of _fetch: adds val at pos."""
    n = table.shape[1] - 1
    p = pos.clamp(0, n)
    i = p.floor().clamp_(max=n - 1)
    p = p - i
    i = (i.long() + torch.arange(table.shape[0], device=pos.device) * (n + 1)).reshape(-1)
    flat = table.view(-1)
    flat.scatter_add_(0, i, (val * (1 - p)).reshape(-1))
    flat.scatter_add_(0, i + 1, (val * p).reshape(-1))


def _prefix(rows):
    return torch.nn.functional.pad(rows.cumsum(1), (1, 0))


def _suffix(adj):
    """Transpose of _prefix."""
    return adj[:, 1:].flip(1).cumsum(1).flip(1)


class _Fan64:
    """The fan pair of one slice in 64 bits: rows of prefix sums along the lines of a view's class, footprints
    between cell edges (distance driven: lines are the averages of neighbouring rows, border zero) or the two ends
    of a cell-centre ray in a row (Siddon)."""

    def __init__(self, case, angles, siddon):
        self.case, self.siddon = case, siddon
        self.t = torch.as_tensor(np.asarray(angles, np.float32).astype(np.float64), device=_device())
        self.xcls = self.t.cos().abs() > self.t.sin().abs()
        self.da = float(np.float32(PITCH))
        self.off = float(np.float32(case.get("off_a", 0.0)))
        self.d, self.dso = float(np.float32(case["dx"])), float(np.float32(DSO))

    def _a(self, first, count):
        u = torch.arange(count, device=self.t.device, dtype=torch.float64) + first
        return (-(u - (self.case["nu"] - 1) / 2.0) - self.off) * self.da

    def _chunks(self):
        """(view indices, class, positions [views, cells, lines], length factors [views, nu]) of views at a time."""
        nu = self.case["nu"]
        for cls in (True, False):
            nlat, nline = (self.case["nx"], self.case["ny"]) if cls else (self.case["ny"], self.case["nx"])
            which = torch.nonzero(self.xcls == cls)[:, 0]
            step = max(1, int(3e7 // (nu * nline)))
            line = torch.arange(nline + (1 if self.siddon else 0), device=self.t.device, dtype=torch.float64)
            for k in range(0, len(which), step):
                v = which[k:k + step]
                t = self.t[v][:, None]
                sx, sy = self.dso * t.sin() / self.d, -self.dso * t.cos() / self.d
                a = self._a(0.0, nu)[None] if self.siddon else self._a(-0.5, nu + 1)[None]
                slope = torch.tan(a - t) if cls else 1 / torch.tan(a - t)
                lat, main = (sx, sy) if cls else (sy, sx)
                pos = (lat + nlat / 2.0)[..., None] + slope[..., None] * (line - (main + nline / 2.0))[:, None, :]
                c = self._a(0.0, nu)[None]
                ln = self.d / (torch.cos(t - c) if cls else torch.sin(t - c)).abs()
                yield v, cls, pos, ln

    def _rows(self, img, cls):
        """Prefix rows of an [nx, ny] image for a view class."""
        rows = img.double().t() if cls else img.double()
        if not self.siddon:
            rows = 0.5 * (rows + torch.nn.functional.pad(rows, (0, 0, 1, 0))[:-1])
        return _prefix(rows.contiguous())

    def project(self, img):
        out = torch.empty((self.case["nu"], len(self.t)), dtype=torch.float64, device=self.t.device)
        table = {c: self._rows(img, c) for c in (True, False)}
        for v, cls, pos, ln in self._chunks():
            if self.siddon:
                a, b = pos[..., :-1], pos[..., 1:]
                b = torch.where((b - a).abs() < 1e-6, a + 1e-6, b)
                m = (_fetch(table[cls], b) - _fetch(table[cls], a)) / (b - a)
            else:
                f = _fetch(table[cls], pos)
                m = (f[:, 1:] - f[:, :-1]) / (pos[:, 1:] - pos[:, :-1])
            out[:, v] = (m.sum(-1) * ln).t()
        return out

    def transpose(self, sino):
        nx, ny = self.case["nx"], self.case["ny"]
        adj = {c: torch.zeros((ny, nx + 1) if c else (nx, ny + 1), dtype=torch.float64, device=self.t.device)
               for c in (True, False)}
        for v, cls, pos, ln in self._chunks():
            w = (sino[:, v].double().t() * ln)[..., None]
            if self.siddon:
                a, b = pos[..., :-1], pos[..., 1:]
                b = torch.where((b - a).abs() < 1e-6, a + 1e-6, b)
                s = w / (b - a)
                _put(adj[cls], a, -s)
                _put(adj[cls], b, s)
            else:
                s = torch.nn.functional.pad(w / (pos[:, 1:] - pos[:, :-1]), (0, 0, 1, 1))
                _put(adj[cls], pos, s[:, :-1] - s[:, 1:])
        img = 0.0
        for cls in (True, False):
            rows = _suffix(adj[cls])
            if not self.siddon:
                rows = 0.5 * (rows + torch.nn.functional.pad(rows, (0, 0, 0, 1))[1:])
            img = img + (rows.t() if cls else rows)
        return img

    def _pixels(self, v, shift=0.0):
        """(rx, ry + dso) of the pixel centres, moved by shift pixels along the view class's lateral axis."""
        dev, nx, ny = self.t.device, self.case["nx"], self.case["ny"]
        x = ((torch.arange(nx, device=dev, dtype=torch.float64) - (nx - 1) / 2.0) * self.d)[None, :, None]
        y = ((torch.arange(ny, device=dev, dtype=torch.float64) - (ny - 1) / 2.0) * self.d)[None, None, :]
        cls = self.xcls[v][:, None, None].double()
        x, y = x + shift * self.d * cls, y + shift * self.d * (1 - cls)
        co, si = self.t[v].cos()[:, None, None], self.t[v].sin()[:, None, None]
        return x * co + y * si, y * co - x * si + self.dso

    def gather(self, sinos, bp):
        """The reference's own backprojections of [slices, nu, nview] data: bp 0 (length weight) and 1 (distance
        weight) between a pixel's two edges, 4 pixel driven."""
        nu, out = self.case["nu"], 0.0
        step = max(1, int(3e7 // (self.case["nx"] * self.case["ny"])))
        for k in range(0, len(self.t), step):
            v = torch.arange(k, min(k + step, len(self.t)), device=self.t.device)
            rows = sinos[:, :, v].double().transpose(1, 2)                   # [slices, views, nu]
            if bp == 0:
                c = self.t[v][:, None] - self._a(0.0, nu)[None]
                rows = rows * self.d / torch.where(self.xcls[v][:, None], c.cos().abs(), c.sin().abs())
            rx, ry = self._pixels(v)
            weight = self.dso ** 2 / (rx * rx + ry * ry) if bp else 1.0
            flat = torch.arange(len(v), device=v.device)[:, None, None] * (nu + (1 if bp == 4 else 2))
            if bp == 4:
                pu = -(torch.atan(rx / ry) / self.da + self.off) + (nu - 1) / 2.0 + 1   # one zero cell before
                i = pu.floor().clamp(0, nu)
                f = ((pu - i) * ((pu > 0) & (pu < nu + 1))).clamp(0, 1)
                inside = ((pu > 0) & (pu < nu + 1)).double()
                padded = torch.nn.functional.pad(rows, (1, 1))
                i = i.long() + torch.arange(len(v), device=v.device)[:, None, None] * (nu + 2)
                add = [(((1 - f) * p.reshape(-1).take(i) + f * p.reshape(-1).take(i + 1)) * inside * weight).sum(0)
                       for p in padded]
            else:
                ends = []
                for shift in (-0.5, 0.5):
                    ex, ey = self._pixels(v, shift)
                    ends.append(-(torch.atan(ex / ey) / self.da + self.off) + nu / 2.0)
                lo, hi = torch.minimum(*ends), torch.maximum(*ends)
                table = torch.nn.functional.pad(rows.cumsum(-1), (1, 1), mode="constant")
                table[..., -1] = table[..., -2]
                parts = []
                for e in (lo, hi):
                    p = e.clamp(0, nu)
                    i = p.floor()
                    parts.append((i.long() + flat, p - i))
                add = []
                for p in table:
                    p = p.reshape(-1)
                    at = [p.take(i) + f * (p.take(i + 1) - p.take(i)) for i, f in parts]
                    add.append(((at[1] - at[0]) / (hi - lo) * weight).sum(0))
            out = out + torch.stack(add)
        return out

    def back(self, sino, bp):
        return self.transpose(sino) if bp in (2, 3) else self.gather(sino[None], bp)[0]


def _exact_fan(case, seed):
    counts, img, ang, b, _ = _ragged_data(case, seed)
    prj, back, o = [], [], 0
    for s, n in enumerate(counts):
        op = _Fan64(case, ang[o:o + n], case["projector"] == "siddon")
        prj.append(op.project(img[s]).reshape(-1))
        back.append(op.back(b[case["nu"] * o:case["nu"] * (o + n)].reshape(case["nu"], n), case["bp"]))
        o += n
    if case["slices"] == 1:
        return [prj[0].reshape(1, case["nu"], -1, 1, 1), back[0][None, ..., None, None]]
    return [torch.cat(prj), torch.stack(back)]


def _exact_stack(case, images, sinos, angles, bp):
    """[n, nx, ny] and [n, nu, nview] through the pair, slice by slice."""
    op = _Fan64(case, angles, False)
    return torch.stack([op.project(x) for x in images]), torch.stack([op.back(y, bp) for y in sinos])


def _exact_fbp(case, seed):
    ang = _short_scan(case)
    b = _stack_data(case, seed, ang, case["slices"])[1].double()
    nu, n = case["nu"], case["views"]
    op = _Fan64(case, ang, False)
    pi = 3.141592657                                    # as the filter and its scale have it
    # Parker's weights
    beta = op.t[None, :]
    gamma = (beta[0, -1] - math.pi) / 2
    alpha = ((torch.arange(nu, device=b.device).double() - (nu - 1) / 2.0) * PITCH)[:, None]
    rise = torch.sin(math.pi / 4 * beta / (gamma - alpha)) ** 2
    fall = torch.sin(math.pi / 4 * (math.pi + 2 * gamma - beta) / (gamma + alpha)) ** 2
    w = torch.where(beta < 2 * gamma - 2 * alpha, rise, torch.where(beta <= math.pi - 2 * alpha, torch.ones_like(rise), fall))
    # the equiangular ramp with its window, as a linear convolution
    k = torch.arange(-(nu - 1), nu, device=b.device).double()
    h = torch.where(k.long() % 2 != 0, -1 / (pi * torch.sin(k * op.da)) ** 2, torch.zeros_like(k))
    h[nu - 1] = 1 / (4 * op.da ** 2)
    if case["filter"]:
        i = torch.arange(2 * nu - 1, device=b.device).double() / (2 * nu - 2)
        window = {1: 0.54 + 0.46 * torch.cos(2 * pi * i), 2: 0.5 + 0.5 * torch.cos(2 * pi * i),
                  3: torch.cos(pi * i).abs()}[case["filter"]]
        h = torch.fft.ifft(torch.fft.fft(h) * window).real
    size = 1 << (3 * nu).bit_length()
    spectrum = torch.fft.rfft(h, size)[None, :, None]
    x = b * w[None] * torch.cos(alpha)[None]
    f = torch.stack([torch.fft.irfft(torch.fft.rfft(s, size, dim=0) * spectrum[0], size, dim=0)[nu - 1:2 * nu - 1]
                     for s in x])
    f = f * (pi / n * op.da / op.dso)
    return [op.gather(f, 4)[..., None, None]]


def _exact_ossqs(case, seed):
    counts, img, ang, b, w = _ragged_data(case, seed)
    m, nu = case["subsets"], case["nu"]
    parts, norms, o = [], [], 0
    for n in counts:
        data, wt = (v[nu * o:nu * (o + n)].reshape(nu, n).double() for v in (b, w))
        subs = [(_Fan64(case, ang[o + k:o + n:m], False), data[:, k::m], wt[:, k::m]) for k in range(m)]
        ones = torch.ones_like(img[0]).double()
        norms.append(sum(op.transpose(op.project(ones) * ws) for op, _, ws in subs))
        parts.append(subs)
        o += n
    beta = 0.05 * torch.stack(norms).reshape(-1).median() / (4 / math.sqrt(1e-6))
    res = []
    for subs, norm in zip(parts, norms):
        x = torch.zeros_like(norm)
        for _ in range(case["iterations"]):
            for op, bs, ws in subs:
                p = torch.nn.functional.pad(x, (1, 1, 1, 1))
                d = [x - p[:-2, 1:-1], x - p[2:, 1:-1], x - p[1:-1, :-2], x - p[1:-1, 2:]]
                psi = [torch.sqrt(q * q + float(np.float32(1e-6))) for q in d]
                grad = sum(q / r for q, r in zip(d, psi)) / 2
                num = m * op.transpose((op.project(x) - bs) * ws) + beta * grad
                x = (x - num / (norm + beta * sum(1 / r for r in psi) + 1e-6)).clamp_min(0)
        res.append(x)
    return [torch.stack(res)]


def _overlap(lo, hi, n):
    """[..., n]: how much of each of n unit cells lies in [lo, hi], over hi - lo."""
    i = torch.arange(n, device=lo.device, dtype=torch.float64)
    part = (hi[..., None] - i).clamp(0, 1) - (lo[..., None] - i).clamp(0, 1)
    return part / (hi - lo)[..., None]


def _exact_tomo(case, seed):
    vol, prj, (dc, _, _, src) = _flat_data(case, seed)
    vol, prj = vol[0, ..., 0].double(), prj[0, ..., 0].double()
    dev, nx, ny, nz, nu, nv = vol.device, *(case[k] for k in ("nx", "ny", "nz", "nu", "nv"))
    dx, dz, du = (float(np.float32(case[k])) for k in ("dx", "dz", "du"))

    def ar(n):
        return torch.arange(n, device=dev, dtype=torch.float64)

    out, back = torch.zeros_like(prj), torch.zeros_like(vol)
    zpix = ar(nz)
    for k in range(case["views"]):
        s, d = src[k].astype(np.float64), dc[k].astype(np.float64)
        sz, ez = s[2] / dz + nz / 2.0, d[2] / dz + nz / 2.0

        def faces(n, cells, axis, edge):
            """Where a cell's edge ray meets the integer z planes, [nz, cells], in voxels."""
            c = (ar(cells) - (cells - 1) / 2.0 + edge) * du + d[axis]
            s0 = s[axis] / dx + n / 2.0
            return s0 + ((c / dx + n / 2.0) - s0)[None] / (ez - sz) * (zpix - sz)[:, None]

        wx = _overlap(faces(nx, nu, 0, -0.5), faces(nx, nu, 0, 0.5), nx)      # [nz, nu, nx]
        wy = _overlap(faces(ny, nv, 1, -0.5), faces(ny, nv, 1, 0.5), ny)
        p = sum(wx[z] @ vol[:, :, z] @ wy[z].t() for z in range(nz))
        cu, cv = ((ar(n) - (n - 1) / 2.0) * du for n in (nu, nv))
        gap = s[2] - d[2]
        ln = dz / abs(gap) * torch.sqrt((s[0] - d[0] - cu)[:, None] ** 2 + (s[1] - d[1] - cv)[None] ** 2 + gap ** 2)
        out[:, k] = p * ln
        z = (zpix - (nz - 1) / 2.0) * dz
        r = (d[2] - s[2]) / (z - s[2])

        def shadow(n, cells, axis):
            c = (ar(n) - (n - 1) / 2.0) * dx
            e = [(s[axis] - d[axis] + r[:, None] * (c + h * dx - s[axis])[None]) / du + (cells - 1) / 2.0
                 for h in (-0.5, 0.5)]
            return _overlap(e[0], e[1], cells)

        bx, by = shadow(nx, nu, 0), shadow(ny, nv, 1)
        weighted = prj[:, k] * ln
        for q in range(nz):
            back[:, :, q] += bx[q] @ weighted @ by[q].t()
    return [out[None, ..., None], back[None, ..., None]]


def _exact_cone(case, seed):
    vol, prj, views = _flat_data(case, seed)
    vol, prj = vol[0, ..., 0].double(), prj[0, ..., 0].double()
    case = dict(case, **{k: float(np.float32(case[k])) for k in ("dx", "dz", "du", "dv")})
    n, d = (case["nx"], case["ny"], case["nz"]), (case["dx"], case["dx"], case["dz"])
    src, dst = _flat_cells(case, views)
    stride = (n[1] * n[2], n[2], 1)
    out, back = torch.zeros_like(prj), torch.zeros(vol.numel(), dtype=torch.float64, device=vol.device)
    flat = vol.reshape(-1)
    rows = max(1, int(6e6 // (case["nv"] * max(n))))
    for k in range(case["views"]):
        mid = [float(dst[i][:, k].mean() - src[i][:, k].mean()) / d[i] for i in range(3)]
        m = max(range(3), key=lambda i: abs(mid[i]))
        a, b = [i for i in range(3) if i != m]
        slab = torch.arange(n[m] + 1, device=vol.device, dtype=torch.float64)
        for u in range(0, case["nu"], rows):
            cut = slice(u, u + rows)
            s = [(src[i][:, k] / d[i] + n[i] / 2.0)[0, 0] for i in range(3)]
            e = [(dst[i][cut, k] / d[i] + n[i] / 2.0).expand(-1, case["nv"]) for i in range(3)]
            length = torch.sqrt(sum(((e[i] - s[i]) * d[i]) ** 2 for i in range(3))) / (e[m] - s[m]).abs()
            knots, at = [], []
            for i in (a, b):
                slope = (e[i] - s[i]) / (e[m] - s[m])
                p = s[i] + slope[..., None] * (slab - s[m])
                p0, p1 = p[..., :-1], p[..., 1:]
                at.append((p0, p1 - p0))
                first = torch.minimum(p0, p1).floor() + 1
                step = torch.where((p1 - p0).abs() < 1e-12, torch.full_like(p0, 1e-12), p1 - p0)
                knots += [((first + j - p0) / step).clamp(0, 1) for j in range(int(math.ceil(float(slope.abs().max()))))]
            knots = [torch.zeros_like(knots[0])] + knots + [torch.ones_like(knots[0])]
            for i in range(1, len(knots) - 2):                              # sort the crossings of a slab
                for j in range(1, len(knots) - 1 - i):
                    knots[j], knots[j + 1] = torch.minimum(knots[j], knots[j + 1]), torch.maximum(knots[j], knots[j + 1])
            base = torch.arange(n[m], device=vol.device) * stride[m]
            w = prj[cut, k] * length
            total = 0.0
            for t0, t1 in zip(knots[:-1], knots[1:]):
                tm, part = 0.5 * (t0 + t1), t1 - t0
                ia, ib = ((p0 + tm * dp).floor().long() for p0, dp in at)
                part = part * ((ia >= 0) & (ia < n[a]) & (ib >= 0) & (ib < n[b]))
                idx = base + ia.clamp_(0, n[a] - 1) * stride[a] + ib.clamp_(0, n[b] - 1) * stride[b]
                total = total + (part * flat.take(idx)).sum(-1)
                back.scatter_add_(0, idx.reshape(-1), (part * w[..., None]).reshape(-1))
            out[cut, k] = total * length
    return [out[None, ..., None], back.reshape(1, *n, 1)]


def _exact_cyl(case, seed):
    vol, prj = _cyl_data(case, seed)
    vol, prj = vol[0].double(), prj[0].double()
    dev, nx, ny, nz, nu, nv = vol.device, *(case[k] for k in ("nx", "ny", "nz", "nu", "nv"))
    d, dz, dsd, dso, da = (float(np.float32(v)) for v in (case["dx"], case["dz"], DSD, DSO, PITCH))

    def ar(n, dtype=torch.float64):
        return torch.arange(n, device=dev, dtype=dtype)

    out, back = torch.empty_like(prj), torch.zeros_like(vol)
    rise = (ar(nv + 1) - nv / 2.0) / dsd
    centre = torch.sqrt(1 + ((ar(nv) - (nv - 1) / 2.0) / dsd) ** 2)
    for k, t in enumerate(_angles(case["views"]).astype(np.float64)):
        cls = abs(math.cos(t)) > abs(math.sin(t))
        nplane, nlat = (ny, nx) if cls else (nx, ny)
        main, lat = (-dso * math.cos(t), dso * math.sin(t)) if cls else (dso * math.sin(t), -dso * math.cos(t))

        def slope(a):
            return torch.tan(a - t) if cls else 1 / torch.tan(a - t)

        a = -(ar(nu) - (nu - 1) / 2.0) * da
        depth = (ar(nplane) + 0.5 - nplane / 2.0) * d - main                     # [planes]
        ends = [(lat + slope(a + h * da)[None] * depth[:, None]) / d + nlat / 2.0 for h in (-0.5, 0.5)]
        lo, hi = torch.minimum(*ends), torch.maximum(*ends)                      # [planes, nu]
        rc = slope(a)
        inplane = torch.sqrt(1 + rc * rc)
        wl = _overlap(lo, hi, nlat)                                              # [planes, nu, nlat]
        dist = depth.abs()[:, None] * inplane[None]
        z = rise * dist[..., None] / dz + nz / 2.0                               # [planes, nu, nv + 1]
        pos = z.clamp(0, nz)
        i = pos.floor().clamp_(max=nz - 1)
        f, i = pos - i, i.long()
        scale = d * inplane[None, :, None] * centre / (z[..., 1:] - z[..., :-1])
        planes = vol.transpose(0, 1) if cls else vol                             # [planes, nlat, nz]
        table = torch.nn.functional.pad((wl @ planes).cumsum(-1), (1, 0))
        at = table.gather(-1, i)
        at = at + f * (table.gather(-1, i + 1) - at)
        out[:, k] = ((at[..., 1:] - at[..., :-1]) * scale).sum(0)
        s = torch.nn.functional.pad(prj[:, k][None] * scale, (1, 1))
        c = s[..., :-1] - s[..., 1:]
        adj = torch.zeros_like(table).scatter_add_(-1, i, c * (1 - f)).scatter_add_(-1, i + 1, c * f)
        adj = adj[..., 1:].flip(-1).cumsum(-1).flip(-1)
        add = wl.transpose(1, 2) @ adj
        back += add.transpose(0, 1) if cls else add
    return [out[None], back[None]]


def _exact_cnn(case, seed):
    state, noisy, clean = _cnn_data(case, seed)
    dev = noisy.device
    ws = [torch.as_tensor(state["w%d" % i], device=dev).double().requires_grad_(True) for i in range(5)]
    bs = [torch.as_tensor(state["b%d" % i], device=dev).double().requires_grad_(True) for i in range(5)]
    outs, grads = [], None
    for u, t in zip(noisy.double(), clean.double()):      # one image at a time: the activations are large
        x = (u if case["train"] else (u / 50.0).float().double() * 50.0)[None, None]
        for i in range(5):
            taps = torch.nn.functional.unfold(x, 3, padding=1)[0]               # [cin * 9, pixels]
            x = (ws[i].permute(0, 3, 1, 2).reshape(ws[i].shape[0], -1) @ taps + bs[i][:, None]).reshape(
                1, -1, *u.shape)
            x = x.relu() if i < 4 else x
        y = x[0, 0] + u
        outs.append(y.detach())
        if case["train"]:
            g = torch.autograd.grad(y, ws + bs, 2.0 / noisy.numel() * (y.detach() - t))
            grads = g if grads is None else [p + q for p, q in zip(grads, g)]
    out = torch.stack(outs)
    return [out, list(grads[:5]), list(grads[5:])] if case["train"] else [out / 50.0]


def exact(case, seed):
    kind = case["kind"]
    with torch.enable_grad() if kind == "cnn" else torch.no_grad():
        if kind == "fan":
            return _exact_fan(case, seed)
        if kind == "fan_grad":
            img, cot = _fan_grad_data(case, seed)
            x, y = (v.permute(0, 3, 4, 1, 2).reshape(-1, *v.shape[1:3]) for v in (img, cot))
            prj, back = _exact_stack(case, x, y, _angles(case["views"]), case["bp"])
            fold = (case["batch"], case["nz"], case["channels"])
            return [v.reshape(*fold, *v.shape[1:]).permute(0, 3, 4, 1, 2).contiguous() for v in (prj, back)]
        if kind == "host":
            ang = _angles(case["views"])
            prj, back = _exact_stack(case, *_stack_data(case, seed, ang, 1), ang, case["bp"])
            return [prj[..., None, None], back[..., None, None]]
        return {"fbp": _exact_fbp, "ossqs": _exact_ossqs, "tomo": _exact_tomo, "cone": _exact_cone,
                "cyl": _exact_cyl, "cnn": _exact_cnn}[kind](case, seed)
