"""Backprojection of slices that share their views (csrc/fan_group.cu): groups
of four slices, partial groups, ragged tiles and view chunks, wide and narrow
pixel intervals, offsets, row mixing, channels, the view split, against the FP64
oracle.

Tolerance: the fan backprojections' bar, relative L2 <= 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2, small_fan, to_geometry

pytestmark = pytest.mark.gpu

TOL = 1e-5

# name: (geometry, views, batches, channels)
CASES = {
    "four_slices": (dict(), 12, 4, 1),
    "partial_groups": (dict(nx=33, ny=65, nu=90), 13, 7, 1),
    "planes_and_channels": (dict(nz=2, nv=2, nx=31, ny=17), 9, 2, 2),
    "row_mixing": (dict(nz=3, nv=4, dv=0.8, off_v=0.3, dz=1.1), 7, 1, 1),
    "offset": (dict(off_a=3.4, nx=64, ny=63), 11, 3, 1),
    "narrow_detector": (dict(nu=20, nx=70, ny=66), 10, 5, 1),
    "wide_pixels": (dict(dx=2.6, dy=2.4, nx=40, ny=33, da=0.0019, nu=100), 10, 3, 1),
    "very_wide_pixels": (dict(dx=3.0, dy=3.0, nx=40, ny=33, da=0.0012, nu=140), 10, 3, 1),
    "one_view": (dict(), 1, 3, 1),
    "many_views": (dict(nx=16, ny=16), 90, 3, 1),
}


@pytest.mark.parametrize("type_projector", [0, 1, 4])
@pytest.mark.parametrize("name", CASES)
def test_group_backprojection_matches_oracle(name, type_projector, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import FanPlan
    over, nview, B, C = CASES[name]
    g = small_fan(**over)
    ang = (np.arange(nview) * 2 * np.pi / nview + 0.05).astype(np.float32)
    plan = FanPlan(to_geometry(g), ang, nbatches=B, nchannels=C)
    y = rng.random(plan.sino_shape).astype(np.float32)
    if type_projector == 4:
        ref = O.pixel_bp(y, ang, g, (g.nx, g.ny, g.nz))
    else:
        ref = O.fan_bp(y, ang, g, (g.nx, g.ny, g.nz), type_projector)
    yd = torch.from_numpy(y).cuda()
    got = plan.backproject(yd, type_projector)
    plan.check()
    assert rel_l2(got.cpu().numpy(), ref) <= TOL
    acc = plan.backproject(yd, type_projector, out=torch.full(plan.img_shape, 0.25, device="cuda"), accumulate=True)
    assert torch.allclose(acc, got + 0.25, rtol=1e-6, atol=1e-6)
    plan.set_tuning(bp_parts=1)
    whole = plan.backproject(yd, type_projector).cpu().numpy()
    assert rel_l2(whole, ref) <= TOL


def test_group_wait_timeout_is_reported(rng):
    """Every chunk wait gives up at once: reported, and the plan recovers."""
    import torch
    from reconnet_b200 import _native as N
    from reconnet_b200.torch_ops import FanPlan
    g = small_fan()
    plan = FanPlan(to_geometry(g), (np.arange(20) * 0.3).astype(np.float32), nbatches=4)
    y = torch.from_numpy(rng.random(plan.sino_shape).astype(np.float32)).cuda()
    want = plan.backproject(y, 0)
    plan.set_spin_limit(0)
    plan.backproject(y, 0)
    with pytest.raises(N.ReconNetError):
        plan.check()
    plan.set_spin_limit(-1)
    assert torch.equal(plan.backproject(y, 0), want)
    plan.check()
