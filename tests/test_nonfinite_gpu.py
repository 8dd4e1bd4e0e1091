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
