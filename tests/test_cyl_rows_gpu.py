"""The cylindrical pair's row and height groups (csrc/cyl.cu): the summed columns
of 64 and 96 heights and the direct reads beyond, a last group of one row,
heights outside the volume, and backprojection runs of 64 voxels and one more,
against the FP64 oracle.

Tolerance: the cylindrical pair's bar, relative L2 <= 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5

# name: geometry (64 rows span about 38 dv / dz heights)
CASES = {
    "heights_64": dict(nv=64, dv=1.0, nz=64),
    "heights_96": dict(nv=65, dv=2.2, nz=65),
    "heights_beyond": dict(nv=80, dv=4.0, nz=66),
    "flat_voxels": dict(nv=64, dv=1.0, nz=129, dz=0.25),
    "thick_voxels": dict(nv=66, dv=0.5, nz=3, dz=9.0),
    "above_the_volume": dict(nv=130, dv=1.0, nz=20, off_v=60.0, cz=-8.0),
    "one_row": dict(nv=1, dv=20.0, nz=5),
    "wide_footprints": dict(nu=12, da=0.014, nv=64, dv=1.0, nz=31),
}


@pytest.mark.parametrize("name", CASES)
def test_cyl_row_groups_match_oracle(name, rng):
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import CylGeometry, CylPlan
    kw = dict(nx=20, ny=18, nz=12, dx=2.0, dy=2.0, dz=1.0, nu=24, nv=8, da=0.004, dv=2.0, dsd=1085.6, dso=595.0)
    kw.update(CASES[name])
    g = CylGeometry(**kw)
    ang = (0.013 + np.arange(37) * 2 * np.pi / 37).astype(np.float32)   # more views than one group of 32
    plan = CylPlan(g, ang)
    x = rng.random(plan.vol_shape).astype(np.float32)
    y = rng.random(plan.prj_shape).astype(np.float32)
    ax = plan.project(torch.from_numpy(x).cuda()).cpu().numpy()
    aty = plan.backproject(torch.from_numpy(y).cuda()).cpu().numpy()
    assert rel_l2(ax, O.cyl_fp(x, ang, g)) <= TOL
    assert rel_l2(aty, O.cyl_bp(y, ang, g, (g.nx, g.ny, g.nz))) <= TOL


def test_even_volume_sums_in_groups():
    """Equal terms on every plane: a group's 32 sums, each rounded by up to half a unit of a sum that grows evenly, come
    to 32 / 2 * 2^-25 of the result where all round the same way (4.8e-7; the 6 groups, tables and lengths add less).
    One chain over the 190 planes may be 2.8e-6 off."""
    import torch
    from oracle import oracle as O
    from reconnet_b200.torch_ops import CylGeometry, CylPlan
    g = CylGeometry(nx=190, ny=180, nz=40, dx=1.4, dy=1.4, dz=0.8, nu=260, nv=16, da=0.0021, dv=1.0, dsd=1085.6, dso=595.0)
    ang = (0.05 + np.arange(16) * 2 * np.pi / 16).astype(np.float32)
    plan = CylPlan(g, ang)
    err = []
    for value in (0.0213, 0.0271, 0.0339):
        x = np.full(plan.vol_shape, value, np.float32)
        err.append(rel_l2(plan.project(torch.from_numpy(x).cuda()).cpu().numpy(), O.cyl_fp(x, ang, g)))
    assert max(err) <= 5e-7, err
