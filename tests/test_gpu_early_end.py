"""Small renders whose paths end early: the host stops launching iterations
when a report says that no rays are left."""

import numpy as np
import pytest

from sundog_b200 import abi
from sundog_b200 import scene as sc

pytestmark = pytest.mark.gpu


def view(kind, depth):
    s = sc.Scene()
    s.render(width=61, height=43, spp=4, max_depth=depth, seed=5, clamp=0.0)
    lookat = {"sky": [0, 2.5, 0], "away": [0, 1, 12]}.get(kind, [0, 0.5, 0])
    s.camera(lookfrom=[0, 1, 6], lookat=lookat, vfov=40)
    s.background_gradient(horizon=[0.6, 0.6, 0.7], zenith=[0.2, 0.3, 0.5])
    s.lambert("grey", color=[0.5, 0.5, 0.5])
    s.dielectric("glass", ior=1.5)
    if kind != "dark":
        s.point_light(position=[1, 4, 2], intensity=[30, 30, 30], radius=0.2)
    s.add("sphere", "grey", sc.scale(0.4))
    s.add("sphere", "glass", sc.scale(0.3), sc.translate(0.6, 0.8, 1.0))
    if kind == "flame":  # late vertices: no shadow stage beside the next trace
        s.flame(base=[-0.8, 0.0, 0.5], height=1.2, radius=0.4, intensity=10.0, sigma=2.0,
                noise_scale=3.0, seed=3, light_intensity=8.0, steps=32)
    return s


@pytest.mark.parametrize("depth", [1, 2, 3, 8, 11, 30])
@pytest.mark.parametrize("kind", ["away", "sky", "spheres", "dark", "flame"])
def test_film_independent_of_where_the_launches_stop(lib, kind, depth):
    """With stage timing every iteration of a group is launched: the same film
    byte for byte. Without, a group with no rays left is not launched to its
    end: three iterations of at most five launches each and a report for a view
    away from everything, however deep its paths may go."""
    with sc.Session(view(kind, depth)) as ses:
        abi.check(ses.lib.sundog_session_set_stage_timing(ses.handle, 1), "timing", ses.lib)
        rays = ses.render().rays_traced
        film = ses.read()
        abi.check(ses.lib.sundog_session_set_stage_timing(ses.handle, 0), "timing", ses.lib)
        for _ in range(20):
            res = ses.render()
            assert res.rays_traced == rays
            assert np.array_equal(ses.read(), film)
    if kind == "away":
        assert res.kernel_launches <= 2 + 3 * 5 + 2
