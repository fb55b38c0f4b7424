"""The slab forward projector at its edges: voxels a ray does not meet, boxes at the shared-memory limit."""
import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


@pytest.mark.parametrize("geom", [
    (24, 40, 16, 0.5, 0.5, 3.0, 5, 40, 64, 0.4, 0.4, 30.0),     # up to four rows a slice
    (24, 40, 16, 0.5, 0.5, 1.0, 7, 40, 64, 0.4, 0.4, 15.0),     # one or two
])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonfinite_row_reaches_only_the_rays_that_meet_it(ctx, geom, bad):
    """One voxel row of infinities or NaN: a detector row none of whose rays meets it (by the one-thread-per-ray
    kernel, which reads only the voxels that a ray meets) stays as it is without that row, bit for bit."""
    g = linear_sweep(*geom)
    plan = engine.Plan(ctx, g, "exact")
    ray = engine.Plan(ctx, g, "exact")
    ray.set_slab(0)
    clean = np.random.default_rng(4).random(g.volume_shape, dtype=np.float32)
    clean[:, 17, :] = 0
    vol = clean.copy()
    vol[:, 17, :] = bad
    meets = ~np.isfinite(ray.forward(vol)).all(axis=2)          # [view][detector row]
    assert meets.any() and not meets.all()
    shapes = [plan.slab] + [(8, 4, 2, 4), (4, 4, 3, 4), (4, 2, 3, 4), (2, 4, 3, 4), (2, 2, 2, 4)]
    for shape in shapes:
        plan.set_slab(*shape)
        assert np.array_equal(plan.forward(vol)[~meets], plan.forward(clean)[~meets]), shape


def test_slab_shape_at_the_shared_memory_limit(ctx):
    """A shape whose boxes, with the two rows of margin a ray needs, take 183 of the 200 KB."""
    g = linear_sweep(64, 64, 8, 0.5, 0.5, 1.0, 5, 48, 160, 0.4, 0.4, 25.0)
    plan = engine.Plan(ctx, g, "exact")
    vol = np.random.default_rng(2).random(g.volume_shape, dtype=np.float32)
    ref = plan.forward(vol)
    plan.set_slab(4, 8, 4, 5)
    assert plan.slab == (4, 8, 4, 5)
    # the same lengths, a slice's sums in the same order: equal bits for every shape
    assert np.array_equal(plan.forward(vol), ref)


@pytest.mark.parametrize("storage,tol", [("f32", 1e-6), ("bf16", 2 ** -7), ("f16", 2 ** -10)])
@pytest.mark.parametrize("nx", [33, 34, 36, 39])
def test_padded_rows_of_a_thick_volume(ctx, storage, tol, nx):
    """Iterations on rows that are not whole 16-byte units, in a volume thick enough for the padded copy, against the
    one-thread-per-ray kernel, at the bounds of test_padded_rows_match_the_ray_kernel."""
    g = linear_sweep(nx, 29, 13, 0.7, 0.45, 1.3, 4, 37, 41, 0.55, 0.35, 22.0)
    p = np.random.default_rng(3).random(g.proj_shape, dtype=np.float32)
    for sart in (False, True):
        xs = []
        for ray in (False, True):
            plan = engine.Plan(ctx, g, "exact", storage)
            if ray:
                plan.set_slab(0)
            x = np.full(g.volume_shape, 0.0 if sart else 1.0, np.float32)
            ctx.read_timing()
            ctx.set_timing(True)
            (plan.sart if sart else plan.mlem)(p, x, 3)
            ctx.set_timing(False)
            whole = nx * (4 if storage == "f32" else 2) % 16 == 0
            assert ("pad_rows" in ctx.read_timing()) == (not ray and not whole)
            xs.append(x)
        assert np.linalg.norm(xs[0] - xs[1]) < tol * np.linalg.norm(xs[1])


@pytest.mark.parametrize("geom,padded", [
    ((13, 13, 4, 0.5, 0.5, 1.0, 9, 20, 20, 0.4, 0.4, 15.0), False),
    ((5, 5, 20, 0.5, 0.5, 1.0, 25, 6, 6, 0.4, 0.4, 15.0), False),
    ((13, 13, 12, 0.5, 0.5, 1.0, 9, 20, 20, 0.4, 0.4, 15.0), True),
    ((61, 61, 3, 0.5, 0.5, 1.0, 27, 96, 96, 0.4, 0.4, 15.0), True),
])
def test_thin_volumes_of_few_rays_are_not_padded(ctx, geom, padded):
    g = linear_sweep(*geom)
    plan = engine.Plan(ctx, g, "exact")
    x = np.ones(g.volume_shape, np.float32)
    ctx.read_timing()
    ctx.set_timing(True)
    plan.mlem(np.ones(g.proj_shape, np.float32), x, 1)
    ctx.set_timing(False)
    assert ("pad_rows" in ctx.read_timing()) == padded


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonfinite_voxel_reaches_only_the_rays_that_meet_it(ctx, storage, bad):
    """Iterations on padded rows against the one-thread-per-ray kernel, from a volume with voxels that are not finite: the
    same voxels become so, the others agree at the bounds above (the slab's lockstep reads, at length zero, up to two
    columns beside a ray's own)."""
    g = linear_sweep(39, 46, 19, 0.5, 0.5, 2.0, 5, 61, 54, 0.4, 0.4, 20.0)
    rng = np.random.default_rng(8)
    p = rng.random(g.proj_shape, dtype=np.float32)
    start = rng.random(g.volume_shape, dtype=np.float32) + 0.5
    start[9, 20, 17] = start[3, 11, 30] = bad
    for sart in (False, True):
        for n in (1, 2):
            xs = []
            for ray in (False, True):
                plan = engine.Plan(ctx, g, "exact", storage)
                if ray:
                    plan.set_slab(0)
                x = start.copy()
                if sart:
                    plan.sart(p, x, n, 0.5)
                else:
                    plan.mlem(p, x, n)
                xs.append(x)
            ok = np.isfinite(xs[1])
            assert np.array_equal(np.isfinite(xs[0]), ok) and not ok.all()
            d = np.linalg.norm((xs[0] - xs[1])[ok]) / np.linalg.norm(xs[1][ok])
            assert d < (1e-6 if storage == "f32" else 2 ** -7)
