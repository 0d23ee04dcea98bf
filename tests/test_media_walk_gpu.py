"""Walks through density grids (tracking to the next event and shadow rays' transmittance) against
the analytic medium: a grid of constant density 1 is the homogeneous medium of the same
coefficients, which other code tracks.  Image sizes and grid sides about the walks' rules: fewer
paths than a warp has lanes, a few more than whole warps, and grids of one, some and odd cells."""

import pathlib
import sys

import numpy as np
import pytest

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent))

from sprout_b200 import capi, scenes  # noqa: E402

pytestmark = pytest.mark.gpu

SEEDS = 12


def _means(side, spp, density, spectral):
    """Mean radiance of SEEDS independent renders."""
    out = []
    for seed in range(SEEDS):
        su = capi.SuLibrary()
        assert su.su_init(False) == 0
        try:
            scenes.volume(su, side, side, spp, density, max_bounces=8,
                          integrator={"seed": 1 + seed, "spectral": spectral})
            assert su.su_render_frame(0) == 0, su.messages
            assert su.su_postprocess() == 0
            out.append(float(su.framebuffer(side, side)[0][:, :, :3].mean()))
        finally:
            su.su_release()
    return np.array(out)


@pytest.mark.parametrize("spectral", [False, True], ids=["rgb", "spectral"])
@pytest.mark.parametrize("side,spp,grid", [(1, 4096, 8), (5, 256, 40), (33, 16, 17)])
def test_constant_grid_is_the_homogeneous_medium(side, spp, grid, spectral):
    a = _means(side, spp, np.ones((grid, grid, grid), np.float32), spectral)
    b = _means(side, spp, None, spectral)
    assert np.isfinite(a).all() and (a > 0).all()
    # five standard errors of the difference of two means of SEEDS independent renders
    bound = 5.0 * np.sqrt((a.var(ddof=1) + b.var(ddof=1)) / SEEDS)
    assert abs(a.mean() - b.mean()) <= bound, (a.mean(), b.mean(), bound)
