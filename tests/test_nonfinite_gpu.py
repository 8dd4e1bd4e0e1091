"""One value that is not finite among the inputs: how far it reaches in the outputs.

The expected reach comes from the FP64 oracle on inputs that are 1 where the value
(and, for the fan tables' running sums, what lies after it) is and 0 elsewhere."""
from types import SimpleNamespace as NS

import numpy as np
import pytest

from conftest import rel_l2, small_fan, to_geometry

pytestmark = pytest.mark.gpu

BAD = [float("nan"), float("inf")]


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("type_projector", [0, 1, 2])
def test_fan_backprojection_keeps_the_channels_before(type_projector, bad, rng):
    """The tables hold sums over the channels up to each one: pixels that see only channels before the value (or its
    neighbour: a pixel's edge within a few hundredths of a cell of a channel's edge may count to either) stay as
    they are."""
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import FanPlan
    g = small_fan(nx=64, ny=60, nu=100, da=0.0018)
    ang = (np.arange(6) * 1.03 + 0.05).astype(np.float32)
    plan = FanPlan(to_geometry(g), ang)
    y = rng.random(plan.sino_shape).astype(np.float32)
    u, v = 47, 3
    yb, after = y.copy(), np.zeros_like(y)
    yb[0, u, v] = bad
    after[0, u - 1:, v] = 1
    got = plan.backproject(torch.from_numpy(yb).cuda(), type_projector).cpu().numpy()
    reach = O.fan_bp(after, ang, g, (g.nx, g.ny, 1), type_projector) > 0
    assert (~np.isfinite(got)).any() and not reach.all()
    assert np.isfinite(got[~reach]).all()
    clean = plan.backproject(torch.from_numpy(y).cuda(), type_projector).cpu().numpy()
    assert rel_l2(got[~reach], clean[~reach]) <= 1e-5


def _cone(kind):
    if kind == "upright":
        n = 24
        t = 0.3 + np.arange(n) * 2 * np.pi / n
        zero, one = np.zeros(n), np.ones(n)
        geo = [np.stack([-180 * np.cos(t), -180 * np.sin(t), zero], 1), np.stack([-np.sin(t), np.cos(t), zero], 1),
               np.stack([zero, zero, one], 1), np.stack([240 * np.cos(t), 240 * np.sin(t), zero], 1)]
        g = dict(nx=40, ny=36, nz=33, dx=1.0, dy=1.0, dz=1.0, nu=60, nv=40, du=1.2, dv=1.2)
    else:
        n = 5
        a = np.radians(np.linspace(-12, 12, n))
        zero, one = np.zeros(n), np.ones(n)
        geo = [np.stack([zero, zero, -30 * one], 1), np.stack([one, zero, zero], 1), np.stack([zero, one, zero], 1),
               np.stack([400 * np.sin(a), 3.3 * one, 400 * np.cos(a)], 1)]
        d = 1.8 if kind == "tomosynthesis_wide" else 0.9
        g = dict(nx=40, ny=64, nz=16, dx=1.0, dy=1.0, dz=1.0, nu=60, nv=80, du=d, dv=d)
    return g, [v.astype(np.float32) for v in geo]


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("kind", ["upright", "tomosynthesis", "tomosynthesis_wide"])
def test_cone_backprojection_reaches_the_ray_only(kind, bad, rng):
    """The voxels that the value's ray meets and no others, in any slice but its own nothing; the rest as without it
    (relative L2 <= 1e-5, the pair's bar); accumulated onto an image too."""
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    g, geo = _cone(kind)
    plan = ConePlan(ConeGeometry(**g), *geo, nbatches=2)
    plan.set_route("own", "own")
    gn = NS(**g, cx=0.0, cy=0.0, cz=0.0, off_u=0.0, off_v=0.0)
    y = rng.random(plan.prj_shape).astype(np.float32)
    yb, ray = y.copy(), np.zeros_like(y)
    at = (1, 33, 2, 41 if kind != "upright" else 22, 0)
    yb[at], ray[at] = bad, 1
    base = torch.full(plan.img_shape, 0.5, device="cuda")
    got = plan.backproject(torch.from_numpy(yb).cuda()).cpu().numpy()
    add = plan.backproject(torch.from_numpy(yb).cuda(), out=base.clone(), accumulate=True).cpu().numpy()
    met = O.cone_bp(ray, *geo, gn, (gn.nx, gn.ny, gn.nz))
    lost = ~np.isfinite(got)
    assert not (lost & (met == 0)).any() and lost[met > 1e-6].all() and (met > 1e-6).any()
    assert (lost == ~np.isfinite(add)).all()
    y[at] = 0
    ref = O.cone_bp(y, *geo, gn, (gn.nx, gn.ny, gn.nz))
    assert rel_l2(got[~lost], ref[~lost]) <= 1e-5
    assert rel_l2(add[~lost], ref[~lost] + 0.5) <= 1e-5
