"""The tuner on small plans and on plans of equal sizes."""
import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


def kernel_ms(ctx, name, fn):
    for _ in range(3):
        fn()
    ctx.read_timing()
    ctx.set_timing(True)
    for _ in range(9):
        fn()
    ctx.set_timing(False)
    n, t = ctx.read_timing()[name]
    return t / n


@pytest.mark.parametrize("geom", [
    (128, 64, 8, 0.5, 0.5, 1.0, 49, 96, 96, 0.4, 0.4, 15.0),    # eight groups of views
    (128, 128, 24, 0.5, 0.5, 1.0, 15, 96, 96, 0.4, 0.4, 15.0),  # four
])
def test_tuned_small_plan_is_not_slower(ctx, geom):
    """A view's cost in one warp's chain of all views is some five times that in eight groups (24 against 121 us)."""
    torch = pytest.importorskip("torch")
    g = linear_sweep(*geom)
    plan = engine.Plan(ctx, g, "exact")
    y, x = torch.rand(g.proj_shape, device="cuda"), torch.rand(g.volume_shape, device="cuda")
    out, proj = torch.empty(g.volume_shape, device="cuda"), torch.empty(g.proj_shape, device="cuda")
    back, fwd = lambda: plan.back(y, out), lambda: plan.forward(x, proj)
    before = kernel_ms(ctx, "exact_back", back), kernel_ms(ctx, "exact_fwd", fwd)
    want = out.clone(), proj.clone()
    plan.autotune()
    after = kernel_ms(ctx, "exact_back", back), kernel_ms(ctx, "exact_fwd", fwd)
    assert after[0] < 1.5 * before[0] and after[1] < 1.5 * before[1]
    assert torch.equal(out, want[0])
    assert float((proj - want[1]).norm() / want[1].norm()) < 1e-6


def test_plans_of_equal_sizes_keep_their_own_boxes(ctx):
    """The cached result of a narrow sweep is a shape; a wide sweep of the same sizes needs larger boxes for it."""
    def sweep(angle):
        return linear_sweep(24, 40, 16, 0.5, 0.5, 2.0, 5, 40, 64, 0.4, 0.4, angle)
    engine.Plan(ctx, sweep(2.0), "exact").autotune()
    g = sweep(30.0)
    rng = np.random.default_rng(1)
    x, y = rng.random(g.volume_shape, dtype=np.float32), rng.random(g.proj_shape, dtype=np.float32)
    plan, tuned = engine.Plan(ctx, g, "exact"), engine.Plan(ctx, g, "exact")
    tuned.autotune()
    ref = plan.forward(x)
    assert np.linalg.norm(tuned.forward(x) - ref) < 1e-6 * np.linalg.norm(ref)
    assert np.array_equal(tuned.back(y), plan.back(y))
