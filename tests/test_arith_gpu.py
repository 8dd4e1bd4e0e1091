"""The solver kernels' reciprocal and inverse root (Newton steps on the hardware's
estimates) over their whole ranges, through the operators that hold little else.

Tolerances: the inverse root is one Newton step from a 1e-7 estimate, good to about one
FP32 rounding; with the rounding of its argument and of the sum of four 3e-7.  The
reciprocal is FP64's to a few 1e-16, so the update is the FP64 value rounded to FP32:
1e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_inverse_root_of_single_pixels():
    """A 1 x 1 image's four differences are its value x: norm = 4 / sqrt(x^2 + 1e-6), grad = x norm / 2."""
    import torch
    from reconnet_b200 import _native as N
    x = np.concatenate([[0.0, np.inf, -np.inf, np.nan, 1.8e19, -1.8e19, 1.85e19, 3e38, -3e38, 1e-45],
                        np.logspace(-30, 19, 400), -np.logspace(-8, 10, 300)]).astype(np.float32)
    img = torch.from_numpy(x).cuda()
    grad, norm = torch.empty_like(img), torch.empty_like(img)
    N.check(N.lib.rn_tv_sqs(grad.data_ptr(), norm.data_ptr(), None, img.data_ptr(), x.size, 1, 1,
                            torch.cuda.current_stream().cuda_stream))
    with np.errstate(all="ignore"):
        a = (x.astype(np.float64) ** 2 + 1e-6)
        a[a > np.finfo(np.float32).max] = np.inf   # where the FP32 square overflows
        r = 4 / np.sqrt(a)
        g = x.astype(np.float64) * r / 2
    np.testing.assert_allclose(norm.cpu().numpy(), r, rtol=3e-7, atol=0)
    np.testing.assert_allclose(grad.cpu().numpy(), g, rtol=3e-7, atol=0)


def test_reciprocal_in_the_surrogate_step():
    """x = -lam M bp / (norm + 1e-6) from x = 0 and residuals of known backprojection, for denominators over the whole
    range of the division and beyond that of its short form."""
    import torch
    from conftest import small_fan, to_geometry
    from reconnet_b200.torch_ops import FanPlan
    g = small_fan(nx=48, ny=40)
    plan = FanPlan(to_geometry(g), (np.arange(12) * 0.52 + 0.05).astype(np.float32))
    b = -torch.ones(plan.sino_shape, device="cuda")
    w = torch.ones(plan.sino_shape, device="cuda")
    bp = plan.backproject(-b * w, 2).cpu().numpy().astype(np.float64)
    x0 = torch.zeros(plan.img_shape, device="cuda")
    rng = np.random.default_rng(3)
    n = (10.0 ** rng.uniform(-12, 38, bp.shape) * rng.choice([-1, 1], bp.shape)).astype(np.float32)
    n.reshape(-1)[:6] = [0.0, np.float32(-1e-6), np.inf, -np.inf, 3e38, 1e-45]
    out = torch.empty_like(x0)
    plan.sqs_update(out, x0, b, w, torch.from_numpy(n).cuda(), lam=0.7, n_subsets=3)
    with np.errstate(all="ignore"):
        want = (-np.float64(np.float32(0.7)) * (3.0 * bp) / (n.astype(np.float64) + 1e-6)).astype(np.float32)
    got = out.cpu().numpy()
    normal = np.abs(want) > 1e-37
    np.testing.assert_allclose(got[normal], want[normal], rtol=1e-7, atol=0)
    np.testing.assert_allclose(got[~normal], want[~normal], rtol=0, atol=2e-45)
