"""The separable tile kernels of the tomosynthesis pair (tomo_fp_tile_kernel,
tomo_bp_tile_kernel) and their choice by footprint width, at the sizes where
they can go wrong, against the FP64 oracle.

Tolerance of the tile kernels: a value is a sum of products of two shares and a
voxel, each within a few FP32 roundings (6e-8) of its FP64 value, at FP64
positions; ten roundings' worth is 6e-7, taken as 1e-6 relative L2.  Views
outside the tiles' limits run the table kernels, whose FP32 positions have the
pair's own bar of 1e-5."""
import ctypes
from types import SimpleNamespace as NS

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _views(n, arc=20.0, dist=650.0, below=80.0):
    a = np.radians(np.linspace(-arc, arc, n)) if n > 1 else np.zeros(1)
    src = np.stack([dist * np.sin(a), 7.0 * np.cos(a), dist * np.cos(a)], 1).astype(np.float32)
    return np.tile(np.float32([3.0, -2.0, -below]), (n, 1)), src


def _pair(img, prj, dc, src, g, nu, nv, weight_all=1):
    import torch
    from reconnet_b200 import _native as N
    B, nx, ny, nz, C = img.shape
    n = dc.shape[0]
    sizes = ctypes.c_size_t(), ctypes.c_size_t()
    N.lib.rn_tomo_sat_bytes(nx, ny, nz, nu, n, nv, ctypes.byref(sizes[0]), ctypes.byref(sizes[1]))
    # a scratch that starts on an 8-byte boundary only, filled with NaN patterns
    sat = torch.full((max(s.value for s in sizes) // 8 + 2,), float("nan"), dtype=torch.float64, device="cuda")[1:]
    t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (img, prj, dc, src)]
    op, oi = torch.empty((B, nu, n, nv, C), device="cuda"), torch.empty_like(t[0])
    geo = (B, C, nx, ny, nz, g.dx, g.dy, g.dz, g.cx, g.cy, g.cz, nu, n, nv, g.du, g.dv, g.off_u, g.off_v)
    st = torch.cuda.current_stream().cuda_stream
    fix = t[2].data_ptr(), t[3].data_ptr(), sat.data_ptr()
    N.check(N.lib.rn_tomo_project(op.data_ptr(), t[0].data_ptr(), *fix, *geo, st))
    N.check(N.lib.rn_tomo_backproject(oi.data_ptr(), t[1].data_ptr(), *fix, *geo, weight_all, st))
    return op.cpu().numpy(), oi.cpu().numpy()


def _grid(**kw):
    g = dict(dx=0.8, dy=0.8, dz=1.0, cx=1.5, cy=-2.5, cz=0.5, du=0.6, dv=0.6, off_u=0.25, off_v=-0.5)
    g.update(kw)
    return NS(**g)


# name: ((B, nx, ny, nz, C), nu, nv, views, grid overrides)
CASES = {
    # ragged tiles on every axis, batches and channels
    "ragged": ((2, 37, 70, 9, 2), 67, 131, 3, {}),
    # enough 64 x 128-cell tiles for the wide blocks, several per axis
    "wide_blocks": ((1, 70, 75, 6, 1), 130, 260, 50, {}),
    # footprints over one voxel (three taps), voxels over two cells (four)
    "fine_voxels": ((1, 66, 45, 8, 1), 70, 66, 4, dict(du=1.1, dv=1.0)),
    "fine_cells": ((1, 34, 67, 8, 1), 140, 150, 4, dict(du=0.4, dv=0.38)),
    # one axis wide, the other narrow
    "anisotropic": ((1, 40, 33, 7, 1), 41, 70, 3, dict(du=1.2, dv=0.5, dy=0.7)),
    # a single plane; a detector of one cell under many planes
    "one_plane": ((1, 33, 65, 1, 1), 40, 70, 3, {}),
    "one_cell": ((1, 9, 8, 40, 1), 1, 1, 3, {}),
}


@pytest.mark.parametrize("name", CASES)
def test_tiles_match_oracle(name, rng):
    from oracle import oracle as O
    shape, nu, nv, n, over = CASES[name]
    g, (dc, src) = _grid(**over), _views(n)
    img = rng.random(shape).astype(np.float32)
    prj = rng.random((shape[0], nu, n, nv, shape[4])).astype(np.float32)
    fp, bp = _pair(img, prj, dc, src, g, nu, nv)
    assert rel_l2(fp, O.tomo_fp(img, dc, src, g, nu, nv)) <= 1e-6
    # a one-cell detector has no room for the tiles' scratch: table kernels
    tol = 1e-5 if name == "one_cell" else 1e-6
    assert rel_l2(bp, O.tomo_bp(prj, dc, src, g, shape[1:4], 1)) <= tol
    if name == "ragged":   # the reference's weighting of view 0 only
        _, bp0 = _pair(img, prj, dc, src, g, nu, nv, 0)
        assert rel_l2(bp0, O.tomo_bp(prj, dc, src, g, shape[1:4], 0)) <= 1e-6


def test_views_outside_the_limits(rng):
    """Footprints wider than the tiles take, alone and beside views that do not
    need the tables; a detector finer than a third of a voxel."""
    from oracle import oracle as O
    dc, src = _views(5)
    src[1:3, 2] = 150.0      # near sources: magnified footprints shrink on the grid, voxels spread on the detector
    dc[4, 2] = -900.0        # a far detector: narrow footprints
    img = rng.random((1, 21, 35, 6, 1)).astype(np.float32)
    for over in ({}, dict(du=1.7, dv=1.6), dict(du=2.6, dv=2.7), dict(du=0.2, dv=0.21)):
        g = _grid(**over)
        prj = rng.random((1, 30, 5, 36, 1)).astype(np.float32)
        fp, bp = _pair(img, prj, dc, src, g, 30, 36)
        assert rel_l2(fp, O.tomo_fp(img, dc, src, g, 30, 36)) <= 1e-5, over
        assert rel_l2(bp, O.tomo_bp(prj, dc, src, g, (21, 35, 6), 1)) <= 1e-5, over


@pytest.mark.parametrize("over,near,tol", [(dict(du=1.1, dv=1.0), False, 1e-6), ({}, True, 1e-5),
                                           (dict(du=2.6, dv=2.7), False, 1e-5)],
                         ids=["all_three_taps", "mixed", "tables"])
def test_other_classes_beside_wide_blocks(over, near, tol, rng):
    """Calls large enough for the wide blocks whose views need the others' kernels: footprints over one voxel in every
    view; narrow ones in most views and none for the tiles in some; the tables for all, in two batches."""
    from oracle import oracle as O
    dc, src = _views(50)
    if near:
        src[::7, 2] = 50.0    # magnified footprints, down to nothing for the tiles
        src[3::7, 2] = -2.0   # the source between the planes
    g = _grid(**over)
    img = rng.random((2, 40, 45, 6, 1)).astype(np.float32)
    prj = rng.random((2, 130, 50, 260, 1)).astype(np.float32)
    fp, bp = _pair(img, prj, dc, src, g, 130, 260)
    keep = np.arange(50) % 7 != 3   # a source between the planes is compared nowhere else either
    assert rel_l2(fp[:, :, keep], O.tomo_fp(img, dc, src, g, 130, 260)[:, :, keep]) <= tol
    if not near:
        assert rel_l2(bp, O.tomo_bp(prj, dc, src, g, (40, 45, 6), 1)) <= tol
