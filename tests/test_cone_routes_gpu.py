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
