"""Backprojector shapes on volumes of few blocks, whose sums are formed by groups of views."""
import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu

GEOMS = [
    (24, 20, 6, 0.5, 0.5, 1.0, 3, 40, 36, 0.4, 0.4, 15.0),      # eight groups, fewer views than groups
    (33, 9, 3, 0.5, 0.5, 1.0, 8, 40, 36, 0.4, 0.4, 15.0),       # eight groups of one view, a row left over
    (64, 65, 40, 0.5, 0.5, 1.0, 13, 96, 96, 0.4, 0.4, 15.0),    # four groups
    (70, 130, 60, 0.5, 0.5, 1.0, 5, 64, 64, 0.4, 0.4, 15.0),    # one
]
SHAPES = [(8, 1), (4, 1), (4, 2), (2, 1), (2, 2), (1, 1), (0, 1)]


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


@pytest.mark.parametrize("geom", GEOMS)
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_every_shape_gives_the_same_bits(ctx, geom, storage):
    """Also the shape that is read and set again, the staged kernel, and slabs of slices (host buffers)."""
    torch = pytest.importorskip("torch")
    g = linear_sweep(*geom)
    y = np.random.default_rng(6).random(g.proj_shape, dtype=np.float32)
    ref = engine.Plan(ctx, g, "exact", storage).back(y)
    plan = engine.Plan(ctx, g, "exact", storage)
    assert plan.back_shape == (8, 1)
    for shape in SHAPES + [(8, 1)]:
        plan.set_back_shape(*shape)
        assert np.array_equal(plan.back(y), ref), shape
        assert np.array_equal(plan.back(torch.from_numpy(y).cuda()).cpu().numpy(), ref), shape
    if storage == "f32":
        plan.set_back_shape(4, 1)
        for shape in ((8, 2), (4, 3)):
            plan.set_back_staging(*shape)
            assert np.array_equal(plan.back(y), ref), shape


def test_setting_the_shape_that_was_read_keeps_its_speed(ctx):
    """A volume of 32 blocks under 49 views: one sum of all views a warp takes some five times as long as eight."""
    torch = pytest.importorskip("torch")
    g = linear_sweep(128, 64, 8, 0.5, 0.5, 1.0, 49, 96, 96, 0.4, 0.4, 15.0)
    plan = engine.Plan(ctx, g, "exact")
    y = torch.rand(g.proj_shape, device="cuda")
    out = torch.empty(g.volume_shape, device="cuda")

    def ms():
        for _ in range(3):
            plan.back(y, out)
        ctx.read_timing()
        ctx.set_timing(True)
        for _ in range(9):
            plan.back(y, out)
        ctx.set_timing(False)
        n, t = ctx.read_timing()["exact_back"]
        return t / n

    before = ms()
    plan.set_back_shape(*plan.back_shape)
    assert ms() < 2 * before
