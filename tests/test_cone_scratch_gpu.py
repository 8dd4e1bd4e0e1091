"""The cone pair's call scratch (csrc/cone.cu): calls captured in a CUDA graph give
what eager calls give, on new inputs too, for the upright, the tomosynthesis and the
separable kernels, also in child graphs; streams and threads at a time do not share it.

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
    else:   # tomosynthesis, or with a reversed v axis, which the general separable kernel takes
        a = np.radians(np.linspace(-12, 12, n))
        src = np.stack([400 * np.sin(a), 0 * a, 400 * np.cos(a)], 1).astype(np.float32)
        cen = np.tile(np.float32([0, 0, -30]), (n, 1))
        u = np.tile(np.float32([1, 0, 0]), (n, 1))
        v = np.tile(np.float32([0, -1 if kind == "separable" else 1, 0]), (n, 1))
    g = ConeGeometry(nx=24, ny=20, nz=12, dx=1.0, dy=1.0, dz=1.0, nu=30, nv=22, du=1.2, dv=1.2)
    plan = ConePlan(g, cen, u, v, src)
    if kind != "separable":
        plan.set_route("own", "own")   # (calls as small as these would go to the general kernels)
    return plan


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


@pytest.mark.parametrize("kind", ["upright", "tomosynthesis", "separable"])
def test_captured_calls_as_child_graphs(kind):
    """Captured calls add no allocation nodes, so their graph can be a child of another one; its scratch stays its own
    while later captures come and go."""
    import torch
    from cuda.bindings import runtime as rt
    plan = _plan(kind)
    gen = torch.Generator(device="cuda").manual_seed(4)
    vols = [torch.rand(plan.img_shape, device="cuda", generator=gen) for _ in range(3)]
    want = []
    for v in vols:
        p = plan.project(v)
        want.append((p.clone(), plan.backproject(p).clone()))

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1] if len(r) > 1 else None

    def capture():
        x, p, b = vols[0].clone(), torch.empty_like(want[0][0]), torch.empty_like(want[0][1])
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g):
            plan.project(x, out=p)
            plan.backproject(p, out=b)
            plan.backproject(p, out=b)
        return g, x, p, b

    runs = []
    for _ in range(2):
        g, x, p, b = capture()
        parent = ok(rt.cudaGraphCreate(0))
        ok(rt.cudaGraphAddChildGraphNode(parent, None, 0, rt.cudaGraph_t(g.raw_cuda_graph())))
        del g   # the parent has its own copy
        runs.append((parent, ok(rt.cudaGraphInstantiate(parent, 0)), x, p, b))
    capture()   # a graph that is gone again: its scratch goes to the next one
    last = capture()
    last[0].instantiate()
    streams = [torch.cuda.Stream() for _ in runs]
    for k in range(3):
        for q, (_, ex, x, _, _) in enumerate(runs):
            x.copy_(vols[(k + q) % 3])
        last[1].copy_(vols[(k + 2) % 3])
        torch.cuda.synchronize()
        for s, (_, ex, _, _, _) in zip(streams, runs):
            ok(rt.cudaGraphLaunch(ex, s.cuda_stream))
        last[0].replay()
        torch.cuda.synchronize()
        for q, (p, b) in enumerate([r[3:] for r in runs] + [last[2:]]):
            wp, wb = want[(k + q) % 3]
            assert torch.equal(p, wp) and torch.equal(b, wb)
    for parent, ex, *_ in runs:
        ok(rt.cudaGraphExecDestroy(ex))
        ok(rt.cudaGraphDestroy(parent))


@pytest.mark.parametrize("kind", ["upright", "tomosynthesis", "separable"])
def test_call_beside_one_that_waits(kind):
    """A call whose plan's buffers are all in use on another stream, which is far behind."""
    import torch
    plan = _plan(kind)
    gen = torch.Generator(device="cuda").manual_seed(6)
    ys = [torch.rand(plan.prj_shape, device="cuda", generator=gen) for _ in range(6)]
    want = [plan.backproject(y).clone() for y in ys]
    got = [torch.empty_like(w) for w in want]
    torch.cuda.synchronize()
    for y, o in zip(ys, got):
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(20_000_000)   # some 10 ms
            plan.backproject(y, out=o)
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(got, want))


def test_routes_back_and_forth_keep_the_scratch():
    """Choosing routes again and again allocates no more than choosing each once."""
    import torch
    plan = _plan("tomosynthesis")
    ways = [("general", "general"), ("own", "own"), ("auto", "auto"), ("own", "general")]
    for way in ways:
        plan.set_route(*way)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(5000):
        plan.set_route(*ways[_ % 4])
    assert free - torch.cuda.mem_get_info()[0] <= 4 << 20


@pytest.mark.parametrize("kind", ["upright", "tomosynthesis", "separable"])
def test_threads_and_many_streams(kind):
    """More streams and threads than the plan has buffers: calls queue for them and never share one."""
    import threading
    import torch
    plan = _plan(kind)
    gen = torch.Generator(device="cuda").manual_seed(5)
    ys = [torch.rand(plan.prj_shape, device="cuda", generator=gen) for _ in range(8)]
    want = [plan.backproject(y).clone() for y in ys]
    torch.cuda.synchronize()
    outs = [[torch.empty_like(want[0]) for _ in range(10)] for _ in ys]

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for o in outs[k]:
                plan.backproject(ys[k], out=o)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(ys))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for k, w in enumerate(want):
        assert all(torch.equal(o, w) for o in outs[k])
