"""Path numbering and pool bookkeeping of the wavefront engine.

A launch of S samples numbers its paths pixel by pixel, the samples of a
pixel consecutive; a launch of one sample numbers its pixels. Every sample's
random stream depends on (pixel, sample, seed) only and the film folds them
in sample order, so a film must not depend on how its samples are split over
launches: byte for byte."""

import numpy as np
import pytest

from sundog_b200 import abi, scene as sc
from sundog_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (8, 8), (9, 5), (61, 19)])
@pytest.mark.parametrize("spp", [1, 3, 32, 65])
def test_film_independent_of_launch_split(lib, size, spp):
    s = workloads.features()
    opts = dict(width=size[0], height=size[1], spp=spp, aov=True)
    with sc.Session(s, **opts) as whole:
        a = whole.render()
        fa = whole.read()
    with sc.Session(s, chunk_spp=1, **opts) as single:
        b = single.render()
        fb = single.read()
    assert a.rays_traced == b.rays_traced
    for x, y in zip(fa, fb):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("depth", [1, 7, 8, 9, 17, 40])
def test_deep_paths_match_megakernel(lib, depth):
    """The stages launch their iterations in groups of eight: paths that end
    at, just past and far past a group's end, between two facing mirrors that
    keep them alive, against the megakernel's loop. FP32 rounding of
    differently compiled kernels: 1e-4 relative for 99% of the pixels, and
    the same rays up to decisions that rounding flips."""
    s = sc.Scene()
    s.render(width=48, height=40, spp=4, max_depth=depth, seed=2, clamp=0.0)
    s.camera(lookfrom=[0, 0.3, 0.9], lookat=[0, 0.1, -1], vfov=50)
    s.background_solid([0.2, 0.3, 0.4])
    s.metal("mirror", color=[0.98, 0.97, 0.96], roughness=0.0)
    s.lambert("grey", color=[0.6, 0.6, 0.6])
    s.point_light(position=[0.2, 0.8, 0.0], intensity=[1, 1, 1], radius=0.0)
    s.add("rect", "mirror", sc.scale(4), sc.rotate_x(90), sc.translate(0, 0, -1))
    s.add("rect", "mirror", sc.scale(4), sc.rotate_x(-90), sc.translate(0, 0, 1))
    s.add("sphere", "grey", sc.scale(0.15), sc.translate(0.3, 0.0, -0.4))
    films, rays = [], []
    for engine in (0, 1):
        with sc.Session(s, engine=engine) as ses:
            rays.append(ses.render().rays_traced)
            films.append(ses.read()[..., :3].astype(np.float64))
    a, b = films
    err = np.abs(a - b) / np.maximum(np.abs(b), 1e-3)
    assert np.quantile(err, 0.99) <= 1e-4
    assert abs(rays[0] - rays[1]) <= 2e-3 * rays[1]


def test_vanished_camera_directions(lib):
    """A focus distance whose square overflows leaves camera rays without a
    direction. They are traced like any other (tile padding, which has no ray,
    is not): here they meet nothing, so every pixel is the background."""
    s = sc.Scene()
    s.render(width=21, height=13, spp=3, max_depth=4, seed=2, clamp=0.0)
    s.camera(lookfrom=[0, 0.3, 3.0], lookat=[0, 0, 0], vfov=40, focus_dist=1e20)
    s.background_solid([0.25, 0.5, 0.75])
    s.lambert("grey", color=[0.6, 0.6, 0.6])
    s.add("sphere", "grey", sc.scale(0.15), sc.translate(0.3, 0.0, -0.4))
    for engine in (0, 1):
        with sc.Session(s, engine=engine) as ses:
            assert ses.render().rays_traced == 21 * 13 * 3
            assert np.array_equal(ses.read()[..., :3],
                                  np.broadcast_to(np.float32([0.25, 0.5, 0.75]), (13, 21, 3)))


def test_shadow_stage_beside_flames(lib, tmp_path):
    """Opaque shadows in a scene with flames: shadow rays run on a second
    stream beside the next trace, and the flame march after it reads the
    radiance they add to. With stage timing everything runs on one stream:
    the same film byte for byte."""
    s = workloads.volumes(str(tmp_path), width=203, height=117, spp=5)
    s.render(transparent_shadows=False)
    with sc.Session(s, base_dir=str(tmp_path)) as ses:
        abi.check(ses.lib.sundog_session_set_stage_timing(ses.handle, 1), "timing", ses.lib)
        rays = ses.render().rays_traced
        film = ses.read()
        abi.check(ses.lib.sundog_session_set_stage_timing(ses.handle, 0), "timing", ses.lib)
        for _ in range(3):
            assert ses.render().rays_traced == rays
            assert np.array_equal(ses.read(), film)
