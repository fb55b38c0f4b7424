"""kv_batch_mlem against one kv_mlem after another, bit for bit: repeated plans, rows that are not whole 16-byte units,
more problems than side streams, volumes at any address."""
import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


def problems(ctx, scale=2):
    """Twelve problems on seven plans; the first plan four times, the second three."""
    plans = [engine.Plan(ctx, linear_sweep(scale * nx - scale // 2, scale * (28 + 4 * i), 6 + 2 * i, 0.5, 0.5, 1.0, 9 + i,
                                           scale * (40 + 8 * i), scale * 44, 0.4, 0.4, 15.0), "exact")
             for i, nx in enumerate((33, 32, 24, 41, 64, 30, 17))]
    pick = [0, 1, 0, 2, 3, 1, 4, 0, 5, 6, 1, 0]
    rng = np.random.default_rng(9)
    data = [rng.random(plans[k].geometry.proj_shape, dtype=np.float32) for k in pick]
    return [plans[k] for k in pick], data


def work(g):
    return g.n_rays * g.nz + 0.3 * g.n_voxels * g.n_views


@pytest.mark.parametrize("host", [True, False])
@pytest.mark.parametrize("iterations", [0, 1, 4])
def test_batch_equals_one_by_one(ctx, host, iterations):
    torch = pytest.importorskip("torch")
    plans, data = problems(ctx)
    assert all(work(p.geometry) > 4e5 for p in plans)
    start = [np.full(p.geometry.volume_shape, 0.5 + 0.1 * i, np.float32) for i, p in enumerate(plans)]
    want = []
    for plan, p, x0 in zip(plans, data, start):
        x = x0.copy()
        if iterations:
            plan.mlem(p, x, iterations, 0.9)
        want.append(x)
    if host:
        xs = [x.copy() for x in start]
        engine.batch_mlem(ctx, plans, data, xs, iterations, 0.9)
    else:
        xs = [torch.from_numpy(x).cuda() for x in start]
        engine.batch_mlem(ctx, plans, [torch.from_numpy(p).cuda() for p in data], xs, iterations, 0.9)
        xs = [x.cpu().numpy() for x in xs]
    for i, (x, w) in enumerate(zip(xs, want)):
        assert np.array_equal(x, w), i


def test_batch_takes_volumes_at_any_address(ctx):
    """Device volumes that start 4 bytes past a 16-byte boundary."""
    torch = pytest.importorskip("torch")
    plans, data = problems(ctx)
    want, xs = [], []
    for plan, p in zip(plans, data):
        x = np.ones(plan.geometry.volume_shape, np.float32)
        plan.mlem(p, x, 3)
        want.append(x)
        n = x.size
        xs.append(torch.ones(n + 1, device="cuda")[1:].view(x.shape))
    engine.batch_mlem(ctx, plans, [torch.from_numpy(p).cuda() for p in data], xs, 3)
    for i, (x, w) in enumerate(zip(xs, want)):
        assert np.array_equal(x.cpu().numpy(), w), i


@pytest.mark.parametrize("host", [True, False])
def test_batch_of_tiny_problems(ctx, host):
    """Tiny problems (persistent kernels over their tiles) among larger ones, with repeated plans of both kinds, against
    one by one: the same terms summed in another order, at the bound of test_batch_matches_one_by_one."""
    torch = pytest.importorskip("torch")
    tiny = [engine.Plan(ctx, linear_sweep(5 + 3 * i, 9 + i, 3 + i, 0.5, 0.5, 1.0, 2 + i, 12 + 5 * i, 11 + 2 * i, 0.4, 0.4,
                                          15.0), "exact") for i in range(9)]
    assert all(work(p.geometry) <= 4e5 for p in tiny)
    large, data = problems(ctx)
    plans = tiny[:4] + large[:5] + tiny[4:] + [tiny[0], large[0], tiny[8], tiny[0]]
    rng = np.random.default_rng(5)
    data = [rng.random(p.geometry.proj_shape, dtype=np.float32) for p in plans]
    want, xs = [], []
    for plan, p in zip(plans, data):
        x = np.ones(plan.geometry.volume_shape, np.float32)
        plan.mlem(p, x, 4, 0.8)
        want.append(x)
        xs.append(np.ones_like(x) if host else torch.ones(x.shape, device="cuda"))
    engine.batch_mlem(ctx, plans, data if host else [torch.from_numpy(p).cuda() for p in data], xs, 4, 0.8)
    for i, (x, w) in enumerate(zip(xs, want)):
        x = x if host else x.cpu().numpy()
        assert np.linalg.norm(x - w) <= 1e-5 * np.linalg.norm(w), i
        if plans[i] in large or i >= len(plans) - 4:   # its plan's own kernels
            assert np.array_equal(x, w), i


def test_batch_with_voxels_that_are_not_finite(ctx):
    """They reach the rays that meet them and no others, on whole and broken 16-byte rows: against one solve after
    another with the one-thread-per-ray kernel, which reads only what a ray meets."""
    torch = pytest.importorskip("torch")
    plans, data = problems(ctx)
    plans, data = plans[:5], data[:5]
    want, xs = [], []
    for i, (plan, p) in enumerate(zip(plans, data)):
        x = np.random.default_rng(i).random(plan.geometry.volume_shape, dtype=np.float32) + 0.5
        x[2, x.shape[1] // 2, x.shape[2] // 3] = (np.inf, np.nan)[i % 2]
        xs.append(torch.from_numpy(x.copy()).cuda())
        ray = engine.Plan(ctx, plan.geometry, "exact")
        ray.set_slab(0)
        ray.mlem(p, x, 2)
        want.append(x)
    engine.batch_mlem(ctx, plans, [torch.from_numpy(p).cuda() for p in data], xs, 2)
    for x, w in zip(xs, want):
        x, ok = x.cpu().numpy(), np.isfinite(w)
        assert np.array_equal(np.isfinite(x), ok)
        assert np.linalg.norm((x - w)[ok]) < 1e-6 * np.linalg.norm(w[ok])
