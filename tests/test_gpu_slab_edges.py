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
