"""The cone pair's call scratch (csrc/cone.cu): calls captured in a CUDA graph give
what eager calls give, on new inputs too, for the upright and the tomosynthesis
kernels; two streams at a time do not share it.

Tolerance: equality (the same kernels in the same order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(kind):
    import torch  # noqa: F401
    from reconnet_b200.torch_ops import ConeGeometry, ConePlan
    n = 5
    if kind == "upright":
        a = np.arange(n) * 2 * np.pi / n + 0.1
        src = np.stack([200 * np.sin(a), -200 * np.cos(a), 0 * a], 1).astype(np.float32)
        cen = -src
        u = np.stack([np.cos(a), np.sin(a), 0 * a], 1).astype(np.float32)
        v = np.tile(np.float32([0, 0, 1]), (n, 1))
    else:
        a = np.radians(np.linspace(-12, 12, n))
        src = np.stack([400 * np.sin(a), 0 * a, 400 * np.cos(a)], 1).astype(np.float32)
        cen = np.tile(np.float32([0, 0, -30]), (n, 1))
        u = np.tile(np.float32([1, 0, 0]), (n, 1))
        v = np.tile(np.float32([0, 1, 0]), (n, 1))
    g = ConeGeometry(nx=24, ny=20, nz=12, dx=1.0, dy=1.0, dz=1.0, nu=30, nv=22, du=1.2, dv=1.2)
    return ConePlan(g, cen, u, v, src)


@pytest.mark.parametrize("kind", ["upright", "tomosynthesis"])
def test_captured_and_concurrent_calls(kind):
    import torch
    plan = _plan(kind)
    gen = torch.Generator(device="cuda").manual_seed(3)
    vols = [torch.rand(plan.img_shape, device="cuda", generator=gen) for _ in range(3)]
    want = []
    for v in vols:
        p = plan.project(v)
        want.append((p.clone(), plan.backproject(p).clone()))
    x, p, b = vols[0].clone(), torch.empty_like(want[0][0]), torch.empty_like(want[0][1])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        plan.project(x, out=p)
        plan.backproject(p, out=b)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.project(x, out=p)
        plan.backproject(p, out=b)
    for v, (wp, wb) in zip(vols, want):
        x.copy_(v)
        graph.replay()
        assert torch.equal(p, wp) and torch.equal(b, wb)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [(torch.empty_like(p), torch.empty_like(b)) for _ in range(2)]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    for _ in range(4):
        for s, v, (op, ob) in zip(streams, vols[1:], outs):
            with torch.cuda.stream(s):
                plan.project(v, out=op)
                plan.backproject(op, out=ob)
    torch.cuda.synchronize()
    for (op, ob), (wp, wb) in zip(outs, want[1:]):
        assert torch.equal(op, wp) and torch.equal(ob, wb)
