"""The Siddon cone pair on tomosynthesis geometries (csrc/cone_tile.cu) at the
sizes where its tiles can go wrong, against the FP64 oracle, and geometries just
outside its limits, which stay on the general kernels.

Tolerance: the cone pair's bar, relative L2 <= 1e-5."""
from types import SimpleNamespace as NS

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _views(n, arc=15.0, dist=400.0, below=30.0, lift=6.0, flip=(1.0, 1.0), up=1.0, dcx=1.0, dcy=-0.5):
    a = np.radians(np.linspace(-arc, arc, n)) if n > 1 else np.zeros(1)
    src = np.stack([dist * np.sin(a), lift * np.ones(n), up * dist * np.cos(a)], 1).astype(np.float32)
    return [np.tile(np.float32([dcx, dcy, -up * below]), (n, 1)), np.tile(np.float32([flip[0], 0, 0]), (n, 1)),
            np.tile(np.float32([0, flip[1], 0]), (n, 1)), src]


def _geom(**kw):
    g = dict(nx=37, ny=41, nz=10, dx=1.0, dy=0.9, dz=1.3, cx=0.4, cy=-0.3, cz=0.2, nu=47, nv=45, du=1.0, dv=0.95,
             off_u=0.3, off_v=-0.4)
    g.update(kw)
    return g


# name: (grid and detector, views, batches, channels)
CASES = {
    "plain": (_geom(), dict(n=3), 1, 1),
    "batches_channels": (_geom(nz=7), dict(n=2), 2, 3),
    "source_below": (_geom(), dict(n=3, up=-1.0), 1, 1),
    "one_view_one_plane": (_geom(nz=1), dict(n=1), 1, 1),
    "tile_edges": (_geom(nx=33, ny=65, nz=5, nu=33, nv=65), dict(n=2), 1, 1),
    # detector and grid reaching far beyond each other
    "small_detector": (_geom(nx=70, ny=140, nz=5, nu=20, nv=18), dict(n=3), 1, 1),
    "large_detector": (_geom(nx=20, ny=18, nz=9, nu=140, nv=150), dict(n=3), 1, 1),
    # enough 64 x 128-ray tiles for the wide blocks
    "wide_blocks": (_geom(nx=66, ny=70, nz=6, nu=130, nv=260, du=0.8, dv=0.7), dict(n=50), 1, 1),
    # rays over a voxel apart (two voxel rows per column); four rows of rays over a voxel
    "coarse_cells": (_geom(nu=29, nv=30, du=1.7, dv=1.6), dict(n=3), 1, 1),
    "fine_cells": (_geom(nu=110, nv=112, du=0.52, dv=0.5), dict(n=3), 1, 1),
    # steep arcs: most columns cross a voxel line, in either direction
    "steep": (_geom(nz=14, dz=1.9), dict(n=4, arc=24.0, dist=160.0), 1, 1),
    # level rays in a voxel face: a detector row at the source's y, on a grid line
    "level_row": (_geom(nx=32, ny=32, dy=1.0, cx=0.0, cy=0.0, nu=40, nv=41, off_u=0.0, off_v=0.0), dict(n=4, lift=0.0, dcy=0.0), 1, 1),
    "level_row_fine": (_geom(nx=34, ny=128, dy=1.0, cx=0.0, cy=0.0, nu=80, nv=161, du=0.6, dv=0.6, off_u=0.0, off_v=0.0),
                       dict(n=4, lift=0.0, dcy=0.0), 1, 1),
    "level_row_and_column": (_geom(nx=32, ny=64, dy=1.0, cx=0.0, cy=0.0, nu=41, nv=81, off_u=0.0, off_v=0.0),
                             dict(n=1, lift=-7.0, dcx=0.0, dcy=-7.0), 1, 1),
    "level_row_reversed_v": (_geom(nx=32, ny=32, dy=1.0, cx=0.0, cy=0.0, nu=41, nv=41, off_u=0.0, off_v=0.0),
                             dict(n=1, lift=0.0, dcx=0.0, dcy=0.0, flip=(1.0, -1.0)), 1, 1),
    # outside the limits: a reversed axis, cells under 0.3 voxels, slopes over one
    "reversed_v": (_geom(), dict(n=3, flip=(1.0, -1.0)), 1, 1),
    "very_fine": (_geom(nu=90, nv=91, du=0.25, dv=0.25), dict(n=2), 1, 1),
    "oblique": (_geom(dz=2.5), dict(n=3, arc=40.0, dist=120.0), 1, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_tile_pair_matches_oracle(name, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g, views, B, C = CASES[name]
    geo = _views(**views)
    plan = ConePlan(ConeGeometry(**g), *geo, nbatches=B, nchannels=C)
    gn = NS(**g)
    x = rng.random(plan.img_shape).astype(np.float32)
    y = rng.random(plan.prj_shape).astype(np.float32)
    ax = plan.project(torch.from_numpy(x).cuda()).cpu().numpy()
    assert rel_l2(ax, O.cone_fp(x, *geo, gn, gn.nu, gn.nv)) <= TOL
    ref = O.cone_bp(y, *geo, gn, (gn.nx, gn.ny, gn.nz))
    yd = torch.from_numpy(y).cuda()
    aty = plan.backproject(yd)
    assert rel_l2(aty.cpu().numpy(), ref) <= TOL
    acc = plan.backproject(yd, out=torch.full(plan.img_shape, 0.5, device="cuda"), accumulate=True)
    assert torch.allclose(acc, aty + 0.5, rtol=1e-6, atol=1e-6)
