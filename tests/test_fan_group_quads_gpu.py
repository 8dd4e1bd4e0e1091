"""Backprojection of slices that share their views, two groups of four slices per
block (csrc/fan_group.cu): full and partial second groups, an odd number of groups
(the last block has one), ragged tiles of 32 rows, 3 and 4 cells per pixel, the
view split, against the FP64 oracle.

Tolerance: the fan backprojections' bar, relative L2 <= 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2, small_fan, to_geometry

pytestmark = pytest.mark.gpu

TOL = 1e-5

# name: (geometry, views, batches)
CASES = {
    "eight_slices": (dict(), 12, 8),
    "five_slices": (dict(nx=33, ny=31, nu=90), 13, 5),
    "five_groups": (dict(nx=20, ny=33), 9, 18),
    "wide_pixels": (dict(dx=2.6, dy=2.4, nx=40, ny=33, da=0.0019, nu=100), 10, 8),
    "very_wide_pixels": (dict(dx=3.0, dy=3.0, nx=40, ny=33, da=0.0012, nu=140), 10, 7),
}


@pytest.mark.parametrize("type_projector", [0, 1, 4])
@pytest.mark.parametrize("name", CASES)
def test_quads_match_oracle(name, type_projector, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import FanPlan
    over, nview, B = CASES[name]
    g = small_fan(**over)
    ang = (np.arange(nview) * 2 * np.pi / nview + 0.05).astype(np.float32)
    plan = FanPlan(to_geometry(g), ang, nbatches=B)
    y = rng.random(plan.sino_shape).astype(np.float32)
    if type_projector == 4:
        ref = O.pixel_bp(y, ang, g, (g.nx, g.ny, g.nz))
    else:
        ref = O.fan_bp(y, ang, g, (g.nx, g.ny, g.nz), type_projector)
    yd = torch.from_numpy(y).cuda()
    got = plan.backproject(yd, type_projector)
    plan.check()
    assert rel_l2(got.cpu().numpy(), ref) <= TOL
    plan.set_tuning(bp_parts=1)
    assert rel_l2(plan.backproject(yd, type_projector).cpu().numpy(), ref) <= TOL
