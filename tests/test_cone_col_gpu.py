"""The Siddon cone pair on upright detectors (csrc/cone_col.cu) at the sizes and
geometries where its kernels can go wrong, against the FP64 oracle, and the
limits beyond which a plan stays on the general kernels.

Tolerance: the cone pair's bar, relative L2 <= 1e-5 (positions are good to
2.4e-7 of a voxel or ray, which a crossing of a nearly level ray turns into a
few 1e-6 of its length); the adjoint identity 1e-5, as in the other pairs."""
from types import SimpleNamespace as NS

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _orbit(nview, dso=120.0, dod=90.0, up=1.0, height=0.0, det_height=0.0, start=0.3):
    """Sources on a circle at `height`, flat detectors opposite; `up` scales and orients v along z."""
    t = start + np.arange(nview) * 2 * np.pi / nview
    zero, one = np.zeros(nview), np.ones(nview)
    src = np.stack([dso * np.cos(t), dso * np.sin(t), height * one], 1)
    dc = np.stack([-dod * np.cos(t), -dod * np.sin(t), det_height * one], 1)
    du = np.stack([-np.sin(t), np.cos(t), zero], 1)
    dv = np.stack([zero, zero, up * one], 1)
    return [v.astype(np.float32) for v in (dc, du, dv, src)]


def _geom(**kw):
    g = dict(nx=23, ny=19, nz=17, dx=1.0, dy=1.1, dz=0.9, cx=0.7, cy=-0.4, cz=0.3, nu=41, nv=22, du=1.3, dv=1.2,
             off_u=0.25, off_v=-0.5)
    g.update(kw)
    return g


# name: (grid and detector, orbit, batches, channels)
CASES = {
    "plain": (_geom(), dict(nview=7), 1, 1),
    "v_downwards": (_geom(), dict(nview=6, up=-1.0), 1, 1),
    "source_above": (_geom(), dict(nview=5, height=11.0, det_height=-8.0), 1, 1),
    "batches_channels": (_geom(nz=6, nv=9), dict(nview=4), 2, 3),
    "one_plane_one_row": (_geom(nz=1, nv=1, cz=0.0, off_v=0.0), dict(nview=5), 1, 1),
    "chunk_edges_32": (_geom(nx=9, ny=10, nz=32, nv=33), dict(nview=33), 1, 1),
    "chunk_edges_33": (_geom(nx=9, ny=10, nz=33, nv=32), dict(nview=32), 1, 1),
    "chunk_edges_65": (_geom(nx=7, ny=6, nz=65, dz=0.5, nv=65, dv=0.7), dict(nview=9), 1, 1),
    "chunk_edges_129": (_geom(nx=6, ny=7, nz=129, dz=0.4, nv=64, dv=1.0), dict(nview=5), 1, 1),
    "many_rays_per_voxel": (_geom(nx=9, ny=8, nz=9, dz=2.0, nv=90, dv=0.45), dict(nview=5), 1, 1),
    "many_voxels_per_ray": (_geom(nx=9, ny=8, nz=40, dz=0.25, nv=9, dv=4.0), dict(nview=5), 1, 1),
    "steep": (_geom(nx=12, ny=13, nz=24, dz=1.0, nv=60, dv=3.2), dict(nview=6), 1, 1),
    # level rays in a voxel face: the source's height on one, a detector row at that height
    "level_row": (_geom(nz=16, dz=1.0, cz=0.0, nv=21, off_v=0.0), dict(nview=7), 1, 1),
    "level_single_row": (_geom(nz=16, dz=1.0, cz=0.0, nv=1, off_v=0.0), dict(nview=7), 1, 1),
    "level_row_downwards": (_geom(nz=16, dz=1.0, cz=0.0, nv=21, off_v=0.0), dict(nview=7, up=-1.0), 1, 1),
    "level_row_higher": (_geom(nz=40, dz=1.0, cz=0.0, nv=21, off_v=0.0), dict(nview=7, height=5.0, det_height=5.0), 1, 1),
    "level_row_top_face": (_geom(nz=16, dz=1.0, cz=0.0, nv=21, off_v=0.0), dict(nview=5, height=8.0, det_height=8.0), 1, 1),
    "level_row_bottom_face": (_geom(nz=16, dz=1.0, cz=0.0, nv=21, off_v=0.0), dict(nview=5, height=-8.0, det_height=-8.0), 1, 1),
    "level_row_chunk_edge": (_geom(nx=9, ny=8, nz=256, dz=1.0, cz=0.0, nv=33, dv=2.0, off_v=0.0), dict(nview=5), 1, 1),
    # outside the column kernels' limits: rays rising more than a voxel per step, a tilted detector axis
    "too_steep": (_geom(nx=12, ny=13, nz=40, dz=0.4, nv=60, dv=3.2), dict(nview=4), 1, 1),
    "tilted": (_geom(), dict(nview=5), 1, 1),
    "axis_aligned": (_geom(cx=0.0, cy=0.0, nx=20, ny=20, dy=1.0, nu=40, off_u=0.0), dict(nview=4, start=0.0), 1, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_column_pair_matches_oracle(name, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g, orbit, B, C = CASES[name]
    geo = _orbit(**orbit)
    if name == "tilted":
        geo[2][:, 0] = 0.1
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


# in-plane rays that run exactly along a grid line (a column at the axis, views along the axes): which of the two
# voxels such a ray meets is the sign of a rounding, but the pair has to agree on it
@pytest.mark.parametrize("nview", [1, 4, 8])
def test_rays_along_grid_lines_are_adjoint(nview, rng):
    import torch
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g = _geom(nx=24, ny=20, nz=16, dy=1.0, dz=1.0, cx=0.0, cy=0.0, cz=0.0, nu=41, nv=21, off_u=0.0, off_v=0.0)
    plan = ConePlan(ConeGeometry(**g), *_orbit(nview, start=0.0))
    # the rays in question alone
    y = torch.zeros(plan.prj_shape, device="cuda")
    y[:, 20] = torch.from_numpy(rng.random(tuple(y[:, 20].shape)).astype(np.float32)).cuda()
    x = torch.from_numpy(rng.random(plan.img_shape).astype(np.float32)).cuda()
    lhs = float((plan.project(x).double() * y.double()).sum())
    rhs = float((x.double() * plan.backproject(y).double()).sum())
    assert abs(lhs - rhs) <= 1e-5 * abs(lhs)


def test_column_backprojection_on_two_streams(rng):
    """Calls of one plan on several streams have a scratch each."""
    import torch
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g = _geom(nx=64, ny=60, nz=40, nu=96, nv=48)
    plan = ConePlan(ConeGeometry(**g), *_orbit(24))
    ys = [torch.from_numpy(rng.random(plan.prj_shape).astype(np.float32)).cuda() for _ in range(2)]
    want = [plan.backproject(y) for y in ys]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in ys]
    outs = [[], []]
    for _ in range(6):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs[k].append(plan.backproject(ys[k]))
    torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(o, want[k]) for o in outs[k])


def test_more_rows_of_pixels_than_a_grid_holds(rng):
    """131072 pixels along y are more blocks than a launch takes along one axis."""
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g = _geom(nx=2, ny=131072, nz=1, dx=1e-3, dy=1e-3, dz=1e-3, cx=0.0, cy=0.0, cz=0.0, nu=140, nv=1, du=1.3, dv=1.2,
              off_u=0.0, off_v=0.0)
    geo = _orbit(1, start=0.0)
    plan = ConePlan(ConeGeometry(**g), *geo)
    y = rng.random(plan.prj_shape).astype(np.float32)
    got = plan.backproject(torch.from_numpy(y).cuda()).cpu().numpy()
    assert rel_l2(got, O.cone_bp(y, *geo, NS(**g), (2, 131072, 1))) <= TOL
