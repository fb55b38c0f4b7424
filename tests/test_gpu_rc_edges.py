"""The reference-compatible family at its edges."""
import dataclasses

import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


def test_index_that_is_not_a_number_is_no_voxel(ctx):
    """A source at 1e38 mm: its position in voxels overflows, a segment's index along x is NaN, and no segment meets a
    voxel."""
    g = linear_sweep(16, 12, 6, 1e-3, 0.5, 1.0, 3, 20, 18, 0.4, 0.4, 10.0)
    src = g.src.copy()
    src[:, 0] = 1e38
    plan = engine.Plan(ctx, dataclasses.replace(g, src=src), "rc")
    assert not plan.forward(np.ones(g.volume_shape, np.float32)).any()


def test_more_views_than_a_grid_is_high(ctx):
    """65,537 views: the backprojector, whose grid is the volume's, takes them; equal to the oracle, bit for bit."""
    from oracle import oracle as O
    g = linear_sweep(6, 5, 3, 0.5, 0.5, 1.0, 65537, 4, 4, 1.0, 1.0, 10.0)
    p = np.ones(g.proj_shape, np.float32)
    assert np.array_equal(engine.Plan(ctx, g, "rc").back(p), O.rc_back(g, p))


def test_plan_made_while_its_stream_captures(ctx):
    """In a relaxed capture: the plan's tables are not part of the graph, which holds what was launched beside them."""
    torch = pytest.importorskip("torch")
    g = linear_sweep(16, 12, 6, 0.5, 0.5, 1.0, 3, 20, 18, 0.4, 0.4, 10.0)
    x, y = torch.zeros(64, device="cuda"), np.random.default_rng(1).random(g.proj_shape, dtype=np.float32)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        ctx.use_torch_stream()
        plan = engine.Plan(ctx, g, "rc")
        x += 1
    ctx.use_torch_stream()
    graph.replay()
    assert float(x.sum()) == 64.0
    assert np.array_equal(plan.back(y), engine.Plan(ctx, g, "rc").back(y))
