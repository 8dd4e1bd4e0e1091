"""The matched fan backprojection's blocks (csrc/fan_matched.cu) and the forward
projection's pairs of ray groups (csrc/fan.cu) at the sizes where they can go wrong:
images at and beside a block of 31 and a tile of 62 pixels, one block, views of one
class only, view chunks of 8 and one more, tiles that reach past the source (indices
clamped), wide pixels, channels at and beside groups of 31 in odd and even numbers,
against the FP64 oracle and the adjoint identity.

Tolerance: the fan pair's bar, relative L2 <= 1e-5; adjoint 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2, small_fan, to_geometry

pytestmark = pytest.mark.gpu

TOL = 1e-5

ALL = np.pi * 2
# name: (geometry, views, range of the angles)
CASES = {
    "one_block": (dict(nx=31, ny=31), 9, ALL),
    "block_and_one": (dict(nx=32, ny=30), 9, ALL),
    "tile": (dict(nx=62, ny=62), 8, ALL),
    "tile_and_one": (dict(nx=63, ny=125), 7, ALL),
    "x_class_only": (dict(nx=40, ny=70), 9, 0.6),
    "one_view": (dict(nx=33, ny=35), 1, 0.0),
    "past_the_source": (dict(nx=64, ny=64, dx=2.0, dy=2.0, dso=220.0, dsd=400.0, da=0.012), 11, ALL),
    # the quartic's bound at 0.0495 of 0.05 cells for the diagonal views
    "quartic_just_inside": (dict(nx=64, ny=64, dx=1.0, dy=1.0, dso=328.0, dsd=600.0, da=0.0012, nu=230), 16, ALL),
    "wide_pixels": (dict(nx=40, ny=33, dx=3.0, dy=3.0, da=0.0012, nu=140), 10, ALL),
    # table windows of 232 entries (eight views per chunk), 472 (four), 832 (two)
    "window_232": (dict(nx=70, ny=75, dx=1.2, dy=1.2, nu=300, da=0.0009), 17, ALL),
    "window_472": (dict(nx=70, ny=75, dx=1.2, dy=1.2, nu=600, da=0.00043), 17, ALL),
    "window_832": (dict(nx=200, ny=800, dx=2.0, dy=0.5, nu=2000, da=0.0005), 9, ALL),
    "one_group": (dict(nu=30), 9, ALL),
    "group": (dict(nu=31), 9, ALL),
    "two_groups": (dict(nu=62), 6, ALL),
    "three_groups": (dict(nu=63), 5, ALL),
    "off_centre": (dict(nx=50, ny=45, nu=90, off_a=5.3), 17, ALL),
}


@pytest.mark.parametrize("name", CASES)
def test_matched_pair_matches_oracle(name, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import FanPlan
    over, nview, span = CASES[name]
    g = small_fan(**over)
    ang = (np.arange(nview) * span / max(nview, 1) + 0.05).astype(np.float32)
    plan = FanPlan(to_geometry(g), ang, nbatches=2)
    x = rng.random(plan.img_shape).astype(np.float32)
    y = rng.random(plan.sino_shape).astype(np.float32)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    ax, aty = plan.project(xd), plan.backproject(yd, 2)
    plan.check()
    assert rel_l2(ax.cpu().numpy(), O.fan_fp(x, ang, g, g.nu, g.nv)) <= TOL
    assert rel_l2(aty.cpu().numpy(), O.fan_bp(y, ang, g, (g.nx, g.ny, g.nz), 2)) <= TOL
    lhs, rhs = float((ax.double() * yd.double()).sum()), float((xd.double() * aty.double()).sum())
    assert abs(lhs - rhs) <= 1e-5 * abs(lhs)
    acc = plan.backproject(yd, 2, out=torch.full(plan.img_shape, 0.5, device="cuda"), accumulate=True)
    assert torch.allclose(acc, aty + 0.5, rtol=1e-6, atol=1e-6)
    plan.set_tuning(bp_parts=1)
    assert rel_l2(plan.backproject(yd, 2).cpu().numpy(), aty.cpu().numpy()) <= 1e-6


@pytest.mark.parametrize("nu,fp_views", [(217, 4), (248, 4), (249, 3), (249, 2), (744, 1), (745, 1), (775, 2)])
def test_pairs_and_single_ray_groups(nu, fp_views, rng):
    """Work items with more groups of rays than warps go in pairs (odd and even numbers of groups, a last group of one
    ray), others one group per warp; on either side of that line."""
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import FanPlan
    g = small_fan(nu=nu, da=0.16 / nu)
    ang = (np.arange(11) * ALL / 11 + 0.05).astype(np.float32)
    plan = FanPlan(to_geometry(g), ang, nbatches=2)
    x = rng.random(plan.img_shape).astype(np.float32)
    ref = O.fan_fp(x, ang, g, g.nu, g.nv)
    xd = torch.from_numpy(x).cuda()
    assert rel_l2(plan.project(xd).cpu().numpy(), ref) <= TOL
    plan.set_tuning(fp_views=fp_views)
    assert rel_l2(plan.project(xd).cpu().numpy(), ref) <= TOL
    plan.check()
