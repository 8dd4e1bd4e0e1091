"""Edges of the fan pair's preparation kernels (csrc/fan.cu): image lines of one
position, at and beside a block of 128, and too long for shared memory;
backprojection tables of one channel, at and beside a block, and longer than one
pass, against the FP64 oracle.

Tolerance: the fan pair's bar, relative L2 <= 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2, small_fan, to_geometry

pytestmark = pytest.mark.gpu

TOL = 1e-5

# name: (geometry, views, backprojection type)
CASES = {
    "lines_127": (dict(nx=127, ny=129, nu=64), 9, 2),
    "lines_128": (dict(nx=128, ny=16, nu=64), 9, 0),
    "one_row": (dict(nx=96, ny=1, nu=64), 9, 2),
    "one_column": (dict(nx=1, ny=33, nu=64), 9, 1),
    "long_lines": (dict(nx=17, ny=1030, dx=1.0, dy=0.5, nu=64), 9, 2),
    "one_channel": (dict(nx=20, ny=20, nu=1, da=0.04), 9, 2),
    "channels_129": (dict(nx=20, ny=20, nu=129), 9, 0),
    "channels_1024": (dict(nx=20, ny=20, nu=1024, da=9e-4), 5, 2),
    "channels_1025": (dict(nx=20, ny=20, nu=1025, da=9e-4), 5, 2),
    "channels_2500": (dict(nx=20, ny=20, dx=0.5, dy=0.5, nu=2500, da=4e-4), 5, 2),
}


@pytest.mark.parametrize("name", CASES)
def test_fan_pair_at_edges_matches_oracle(name, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import FanPlan
    over, nview, typ = CASES[name]
    g = small_fan(**over)
    ang = (np.arange(nview) * 2 * np.pi / nview + 0.05).astype(np.float32)
    plan = FanPlan(to_geometry(g), ang)
    x = rng.random(plan.img_shape).astype(np.float32)
    y = rng.random(plan.sino_shape).astype(np.float32)
    ax = plan.project(torch.from_numpy(x).cuda()).cpu().numpy()
    aty = plan.backproject(torch.from_numpy(y).cuda(), typ).cpu().numpy()
    plan.check()
    assert rel_l2(ax, O.fan_fp(x, ang, g, g.nu, g.nv)) <= TOL
    assert rel_l2(aty, O.fan_bp(y, ang, g, (g.nx, g.ny, g.nz), typ)) <= TOL
