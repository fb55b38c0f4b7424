"""SART's row sums: every solve reads sums that a pass of its own geometry has stored."""
import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


def sweep(angle, nx=24):
    return linear_sweep(nx, 40, 16, 0.5, 0.5, 2.0, 5, 40, 64, 0.4, 0.4, angle)


def fresh(ctx, g, p, n):
    x = np.zeros(g.volume_shape, np.float32)
    engine.Plan(ctx, g, "exact").sart(p, x, n, 0.5)
    return x


def test_a_solve_after_a_failed_one(ctx):
    """A pass that gives up leaves row sums unwritten; the next solve, with another kernel, must not read them (its
    sums differ from a fresh plan's by a few roundings).  The first solve runs a shape tuned for a narrower sweep of the
    same sizes, whose boxes rays of this one leave unless the plan sizes its own; it may fail or not."""
    narrow, wide = sweep(1.0), sweep(30.0)
    engine.Plan(ctx, narrow, "exact").autotune()
    p = np.random.default_rng(1).random(wide.proj_shape, dtype=np.float32)
    ref = fresh(ctx, wide, p, 4)
    for host in (True, False):
        torch = pytest.importorskip("torch")
        plan = engine.Plan(ctx, wide, "exact")
        plan.autotune()
        x = np.zeros(wide.volume_shape, np.float32) if host else torch.zeros(wide.volume_shape, device="cuda")
        try:
            plan.sart(p if host else torch.from_numpy(p).cuda(), x, 4, 0.5)
            ctx.sync()
        except engine.KvError:
            pass
        plan.set_slab(0)
        x = np.zeros(wide.volume_shape, np.float32)
        plan.sart(p, x, 4, 0.5)
        assert np.linalg.norm(x - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("nx", [24, 23])   # whole and broken 16-byte rows
def test_solves_on_two_streams(ctx, nx):
    """A second solve on another stream, with nothing between them on the host, reads the first one's sums."""
    torch = pytest.importorskip("torch")
    g = sweep(20.0, nx)
    p = np.random.default_rng(2).random(g.proj_shape, dtype=np.float32)
    ref = fresh(ctx, g, p, 3)
    pd = torch.from_numpy(p).cuda()
    xs = [torch.zeros(g.volume_shape, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    plan = engine.Plan(ctx, g, "exact")
    streams = [torch.cuda.Stream() for _ in range(2)]
    for i, x in enumerate(xs):
        # the plan's workspaces serve one solve at a time
        streams[i % 2].wait_stream(streams[1 - i % 2])
        with torch.cuda.stream(streams[i % 2]):
            plan.sart(pd, x, 3, 0.5)
    torch.cuda.synchronize()
    for x in xs:
        assert np.array_equal(x.cpu().numpy(), ref)


@pytest.mark.parametrize("before", [False, True])
def test_solve_in_a_captured_graph(ctx, before):
    """A solve recorded in the caller's graph, before or after a plain one: replays equal a fresh plan's solve, also
    where another solve with other data ran in between."""
    torch = pytest.importorskip("torch")
    g = sweep(20.0)
    p = np.random.default_rng(3).random(g.proj_shape, dtype=np.float32)
    ref = fresh(ctx, g, p, 3)
    pd, x = torch.from_numpy(p).cuda(), torch.zeros(g.volume_shape, device="cuda")
    plan = engine.Plan(ctx, g, "exact")
    other = torch.ones(g.volume_shape, device="cuda")
    plan.mlem(pd, other, 1)                 # workspaces
    if before:
        plan.sart(pd, other, 2, 0.5)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        plan.sart(pd, x, 3, 0.5)
    for _ in range(2):
        x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(x.cpu().numpy(), ref)
        plan.sart(pd, other, 2, 0.5)
        torch.cuda.synchronize()
    del graph
