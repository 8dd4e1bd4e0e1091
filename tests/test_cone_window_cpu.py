"""The backprojection window of the tomosynthesis tiles (csrc/cone_tile.cu): the patch that the plan sizes holds every
tile's rows and columns of rays, over random geometries of the kernels' range.  Both sides' formulas restated in FP64;
the kernel's FP32 arithmetic is inside the 0.01 it adds."""
import math

import numpy as np

TX, TY, TZ = 32, 64, 4   # voxels of a tile


def _patch(views, nz, nu, nv):
    """The plan's patch (floats) and the rows of rays over a voxel, or None outside its limits."""
    lo_u = lo_v = 1e300
    hi = ru_hi = rv_hi = 0.0
    for su, sv, sm, ru0, ru1, rv0, rv1 in views:
        for pm in (0, nz, nz + TZ):
            lo_u, lo_v = min(lo_u, (pm - sm) * ru1), min(lo_v, (pm - sm) * rv1)
        hi = max([hi] + [(pm - sm) * r for pm in (0, nz) for r in (ru1, rv1)])
        ru_hi = max(ru_hi, abs(ru0), abs(ru0 + (nu - 1) * ru1))
        rv_hi = max(rv_hi, abs(rv0), abs(rv0 + (nv - 1) * rv1))
    if not (lo_u >= 0.3 and lo_v >= 0.3 and hi <= 1.9 and ru_hi <= 1 and rv_hi <= 1):
        return None
    kv = max(int((1 + rv_hi + 2e-2) / lo_v) + 1, 3)
    if kv > 4:
        return None
    rows = (TX + TZ * ru_hi) / lo_u + 4.0
    cols = (TY + TZ * rv_hi) / lo_v + kv + 10.0
    return (int(rows) + 1) * ((int(cols) + 4) & ~3), kv


def _windows(view, nx, ny, nz, nu, nv, kv):
    su, sv, sm, ru0, ru1, rv0, rv1 = view
    z0 = np.arange(0, nz, TZ)[:, None]
    M = np.stack([z0 - sm, z0 + TZ - sm])

    def span(s, r0, r1, first, size):
        a = (first - (s + M * r0)) / (M * r1)
        b = (first + size - (s + M * r0)) / (M * r1)
        return a.min(0), b.max(0)

    ulo, uhi = span(su, ru0, ru1, np.arange(0, nx, TX)[None], TX)
    vlo, vhi = span(sv, rv0, rv1, np.arange(0, ny, TY)[None], TY)
    ub = np.maximum(np.floor(ulo - 0.01), 0)
    rows = np.minimum(np.ceil(uhi + 0.01), nu - 1) - ub + 1
    vb = np.floor(np.maximum(np.floor(vlo - 0.01), 0) / 4) * 4
    cols = np.floor((np.maximum(np.minimum(np.ceil(vhi + 0.01), nv - 1) - vb, 0) + kv + 4) / 4) * 4
    return rows[:, :, None] * cols[:, None, :]


def test_patch_holds_every_window():
    rng = np.random.default_rng(11)
    seen = 0
    while seen < 300:
        nx, ny, nz = rng.integers(1, 300), rng.integers(1, 400), rng.integers(1, 150)
        nu, nv = rng.integers(1, 600, 2)
        views = []
        g = rng.uniform(0.3, 1.9)
        far = nz + rng.uniform(1, 900)           # the source above the grid, seen from its lowest face
        for _ in range(3):
            # spacing g at the far face along u, up to 1.3 times it along v
            ru1, rv1 = g / far, g * rng.uniform(0.8, 1.3) / far
            sm = -(far - nz)
            mid = nz / 2 - sm
            su, sv = rng.uniform(-0.6, 1.6) * nx, rng.uniform(-0.6, 1.6) * ny
            ru0 = (nx / 2 - su) / mid - (nu - 1) / 2 * ru1 + rng.uniform(-0.2, 0.2)
            rv0 = (ny / 2 - sv) / mid - (nv - 1) / 2 * rv1 + rng.uniform(-0.2, 0.2)
            views.append((su, sv, sm, ru0, ru1, rv0, rv1))
        p = _patch(views, nz, nu, nv)
        if p is None:
            continue
        seen += 1
        for v in views:
            assert _windows(v, nx, ny, nz, nu, nv, p[1]).max() <= p[0]
    assert math.isfinite(seen)
