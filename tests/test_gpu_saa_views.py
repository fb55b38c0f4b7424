"""Shift-and-add of many views."""
import numpy as np
import pytest

from kevernals_gb300 import build, engine
from kevernals_gb300.geometry import linear_sweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    build.build()
    return engine.Context(0)


@pytest.mark.parametrize("n_views", [1600, 3000])
def test_many_views_over_a_wide_band(ctx, n_views):
    """More views than the direct kernel takes, slices spread over most of the 256 rows a band may have: the sums are
    compensated, so only the result's rounding to FP32 is left (2^-24, and as much again in hand)."""
    g = linear_sweep(16, 16, 16, 0.5, 0.5, 8.0, n_views, 32, 300, 0.1, 0.1, 35.0)
    p = np.random.default_rng(7).random(g.proj_shape, dtype=np.float32)
    got = engine.Plan(ctx, g, "exact").shift_and_add(p)
    shifts = np.clip(engine.shift_and_add_shifts(g, "exact").reshape(g.nz, n_views), -g.nv, g.nv)
    for k in range(g.nz):
        ref = np.zeros((g.nv, g.nu))
        for i, s in enumerate(shifts[k]):
            lo, hi = max(0, -s), min(g.nv, g.nv - s)      # rows v with v + s on the detector
            if lo < hi:
                ref[lo:hi] += p[i, lo + s:hi + s]
        ref /= n_views
        assert np.abs(got[k] - ref).max() <= 2.0 ** -23 * np.abs(ref).max()
