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


# With a grey medium of constant density a cell's minorant and majorant are equal and no collision is
# ever null.  The media below tell them apart: a coloured one (the majorant is that of the densest
# channel), thin enough that shadow rays cross several cells and draw several collisions.
COLOURED = {"attenuation_color": [0.75, 0.5, 0.25], "attenuation_distance": 0.5,
            "subsurface_color": [0.5, 0.3, 0.2], "anisotropy": 0.4}
SPLIT = {"light_sampling": {"strategy": "Adaptive", "splitting_threshold": 1.0}}
MODES = {"rgb": {}, "spectral": {"spectral": True}, "instanced": {"instancing": True}, "split": SPLIT,
         "split_instanced": dict(SPLIT, instancing=True)}


def _channel_means(side, spp, density, integrator, seeds=SEEDS, **scene):
    """Mean radiance of each channel in `seeds` independent renders, and the shadow rays a sample."""
    import ctypes

    from sprout_b200 import _lib

    out, shadows = [], 0.0
    for seed in range(seeds):
        su = capi.SuLibrary()
        assert su.su_init(False) == 0
        try:
            scenes.volume(su, side, side, spp, density, max_bounces=8, integrator=dict(integrator, seed=1 + seed), **scene)
            position = scene.get("position", (3.0, 2.0, -3.2))
            img, = su.render_views([(side, side, scenes.VOLUME_FOV, scenes._look_at(position))], spp)
            st = _lib.RenderStats()
            assert _lib.load().spb_render_last_stats(ctypes.byref(st)) == 0
            assert st.overflow == 0 and st.tracking_capped == 0
            shadows += st.shadow_rays / max(st.paths, 1) / seeds
            out.append(img[:, :, :3].astype(np.float64).mean(axis=(0, 1)))
        finally:
            su.su_release()
    return np.array(out), shadows


def _assert_same_mean(a, b):
    # five standard errors of the difference of two means of independent renders
    bound = 5.0 * np.sqrt((a.var(axis=0, ddof=1) + b.var(axis=0, ddof=1)) / len(a))
    assert np.isfinite(a).all() and (a > 0).all()
    assert np.all(np.abs(a.mean(axis=0) - b.mean(axis=0)) <= bound), (a.mean(axis=0), b.mean(axis=0), bound)


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("side,spp,grid", [(1, 16384, 8), (5, 4096, 40), (33, 256, 17)])
def test_coloured_constant_grid_is_the_homogeneous_medium(side, spp, grid, mode):
    """Null collisions on path segments, residual ratio tracking on shadow rays; "split": a pick for
    every triangle of the lamp and the environment in the second slot; instanced: the two-level walks."""
    a, shadow_a = _channel_means(side, spp, np.ones((grid, grid, grid), np.float32), MODES[mode], medium=COLOURED)
    b, shadow_b = _channel_means(side, spp, None, MODES[mode], medium=COLOURED)
    _assert_same_mean(a, b)
    if mode.startswith("split"):  # several shadow rays a vertex, so picks
        single = {k: v for k, v in MODES[mode].items() if k != "light_sampling"}
        single["light_sampling"] = {"strategy": "Single"}
        _, shadow_single = _channel_means(side, spp, None, single, seeds=1, medium=COLOURED)
        assert shadow_a > 1.2 * shadow_single and shadow_b > 1.2 * shadow_single, (shadow_a, shadow_b, shadow_single)


@pytest.mark.parametrize("side", [1, 2], ids=["9_lanes", "16_lanes"])
def test_coloured_constant_grid_in_waves_smaller_than_a_warp(side):
    """Progressive frames: a wave of one sample is 9 or 16 paths with the filter's border, so the
    collisions that wait for their events are fewer or hardly more than the walk's threshold of 14."""
    means = []
    for density in (np.ones((8, 8, 8), np.float32), None):
        out = []
        for seed in range(6):
            su = capi.SuLibrary()
            assert su.su_init(True) == 0
            try:
                scenes.volume(su, side, side, 1, density, max_bounces=8, integrator={"seed": 1 + seed}, medium=COLOURED)
                assert su.su_start_render_frame(0) == 0, su.messages
                for _ in range(1024):
                    assert su.su_render_iteration() == 0
                assert su.su_postprocess() == 0
                out.append(su.framebuffer(side, side)[0][:, :, :3].astype(np.float64).mean(axis=(0, 1)))
            finally:
                su.su_release()
        means.append(np.array(out))
    _assert_same_mean(*means)


@pytest.mark.parametrize("mode", ["rgb", "instanced", "spectral"])
def test_absorbing_grid_has_the_closed_form_transmittance(mode):
    """Density that varies from voxel to voxel, absorption only: what the camera sees through the grid
    is the environment times exp(-mu_t x the density along the ray), which numpy integrates.  The
    density is a product of a tent along each axis, so that the trilinear filter interpolates each tent
    linearly and wrapping or clamping at the border are the same."""
    n, side, spp, mu_t, sky = 21, 33, 512, 1.5, 0.4
    centre = (np.arange(n) + 0.5) / n
    tent = 1.0 - np.abs(2.0 * centre - 1.0)
    density = (tent[:, None, None] * tent[None, :, None] * tent[None, None, :]).astype(np.float32)
    medium = {"attenuation_color": [0.5] * 3, "attenuation_distance": float(np.log(2.0) / mu_t),
              "subsurface_color": [0.0] * 3, "anisotropy": 0.0}
    position = (0.25, 0.15, -1.9)  # the cube fills the view, the lamp is behind the camera's shoulder
    got, _ = _channel_means(side, spp, density, MODES[mode], medium=medium, position=position,
                            environment=(sky, sky, sky))
    # rays through 3 x 3 points of each pixel
    m = scenes._look_at(position).astype(np.float64)
    at = (np.arange(3 * side) + 0.5) / (3 * side) * 2.0 - 1.0
    half = np.tan(0.5 * scenes.VOLUME_FOV)
    d = at[None, :, None] * half * m[0, :3] - at[:, None, None] * half * m[1, :3] + m[2, :3]
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    o = np.asarray(position)
    t0, t1 = np.sort(np.stack([(-1.0 - o) / d, (1.0 - o) / d]), axis=0)
    near, far = t0.max(axis=2), t1.min(axis=2)
    assert (near > 0).all() and (far > near).all()
    steps = 400
    tau = np.zeros_like(near)
    for k in range(steps):
        p = o + (near + (far - near) * (k + 0.5) / steps)[:, :, None] * d
        tau += np.prod(np.interp(0.5 * (p + 1.0), centre, tent), axis=2)
    want = sky * np.exp(-mu_t * tau * (far - near) / steps).mean()
    # five standard errors, and 1e-3 for the pixel filter (a sample counts up to a pixel away from its
    # own: second order in a pixel, 2e-4 here) and the colours' conversions
    bound = 5.0 * got.std(axis=0, ddof=1) / np.sqrt(len(got)) + 1e-3 * want
    assert np.all(np.abs(got.mean(axis=0) - want) <= bound), (got.mean(axis=0), want, bound)
