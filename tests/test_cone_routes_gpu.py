"""Both routes of the Siddon cone pair (csrc/cone.cu: the general kernels, and those of
the upright and tomosynthesis geometries) over all the geometries of their tests:
each against the FP64 oracle whichever the plan would choose, and what a route that
the geometry does not have answers.

Tolerance: the cone pair's bar, relative L2 <= 1e-5, for the kernels of the geometry's
family and the general ones."""
from types import SimpleNamespace as NS

import numpy as np
import pytest

import test_cone_col_gpu as col
import test_cone_tile_gpu as tile
from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5
# outside the families' limits
OTHER = {"too_steep", "many_rays_per_voxel", "reversed_v", "level_row_reversed_v", "very_fine", "oblique"}


def _case(family, name):
    g, views, B, C = family.CASES[name]
    return g, (col._orbit if family is col else tile._views)(**views), B, C


@pytest.mark.parametrize("route", ["own", "general"])
@pytest.mark.parametrize("family,name", [(f, n) for f in (col, tile) for n in f.CASES if n not in OTHER],
                         ids=lambda v: v if isinstance(v, str) else v.__name__)
def test_route_matches_oracle(family, name, route, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g, geo, B, C = _case(family, name)
    plan = ConePlan(ConeGeometry(**g), *geo, nbatches=B, nchannels=C)
    plan.set_route(route, route)
    gn = NS(**g)
    x = rng.random(plan.img_shape).astype(np.float32)
    y = rng.random(plan.prj_shape).astype(np.float32)
    before = plan.launches()
    ax = plan.project(torch.from_numpy(x).cuda()).cpu().numpy()
    assert plan.launches() - before == (2 * B * C if route == "own" and family is tile else 1)
    assert rel_l2(ax, O.cone_fp(x, *geo, gn, gn.nu, gn.nv)) <= TOL
    ref = O.cone_bp(y, *geo, gn, (gn.nx, gn.ny, gn.nz))
    yd = torch.from_numpy(y).cuda()
    aty = plan.backproject(yd)
    assert rel_l2(aty.cpu().numpy(), ref) <= TOL
    acc = plan.backproject(yd, out=torch.full(plan.img_shape, 0.5, device="cuda"), accumulate=True)
    assert torch.allclose(acc, aty + 0.5, rtol=1e-6, atol=1e-6)
    plan.set_route()
    assert rel_l2(plan.backproject(yd).cpu().numpy(), ref) <= TOL


# rays in a voxel face: the forward and back kernels of either family have to give them to the same voxel
@pytest.mark.parametrize("routes", [("own", "own"), ("own", "general"), ("general", "own"), ("general", "general")],
                         ids="-".join)
@pytest.mark.parametrize("family,name", [(f, n) for f in (col, tile) for n in f.CASES if n.startswith("level") and n not in OTHER]
                         + [(col, f"along{n}") for n in (1, 4, 8)], ids=lambda v: v if isinstance(v, str) else v.__name__)
def test_rays_in_a_face_are_adjoint(family, name, routes, rng):
    import torch
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    if name.startswith("along"):
        g = col._geom(nx=24, ny=20, nz=16, dy=1.0, dz=1.0, cx=0.0, cy=0.0, cz=0.0, nu=41, nv=21, off_u=0.0, off_v=0.0)
        geo, B, C = col._orbit(int(name[5:]), start=0.0), 1, 1
    else:
        g, geo, B, C = _case(family, name)
    plan = ConePlan(ConeGeometry(**g), *geo, nbatches=B, nchannels=C)
    plan.set_route(*routes)
    x = torch.from_numpy(rng.random(plan.img_shape).astype(np.float32)).cuda()
    r = torch.from_numpy(rng.random(plan.prj_shape).astype(np.float32)).cuda()
    ax = plan.project(x).double()
    for part in ("row", "column"):
        y = torch.zeros_like(r)   # the middle rays alone
        if part == "row":
            y[:, :, :, g["nv"] // 2] = r[:, :, :, g["nv"] // 2]
        else:
            y[:, g["nu"] // 2] = r[:, g["nu"] // 2]
        lhs = float((ax * y.double()).sum())
        rhs = float((x.double() * plan.backproject(y).double()).sum())
        assert abs(lhs - rhs) <= 1e-5 * abs(lhs), part


@pytest.mark.parametrize("name", sorted(OTHER))
def test_route_that_is_not_there(name):
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    family = col if name in col.CASES else tile
    g, geo, B, C = _case(family, name)
    plan = ConePlan(ConeGeometry(**g), *geo, nbatches=B, nchannels=C)
    plan.set_route("general", "general")
    for way in (("own", "auto"), ("auto", "own")):
        with pytest.raises(Exception):
            plan.set_route(*way)
