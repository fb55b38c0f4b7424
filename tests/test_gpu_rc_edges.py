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
