"""The two forms of a single ray's walk (traverse, sd_trace.cuh): the
megakernels' lean one (two children's boxes at a time, one pop for all
actions) against the wavefront stages' (all four as packed FMAs)."""

import numpy as np
import pytest

from sundog_b200 import scene as sc
from sundog_b200 import workloads

pytestmark = pytest.mark.gpu


def _leaves(tris, path):
    """A scene around a mesh of so many small triangles: one leaf (up to four),
    or inner nodes with leaves of one to four."""
    rng = np.random.default_rng(tris)
    c = rng.uniform(-0.8, 0.8, (tris, 1, 3))
    v = (c + rng.uniform(-0.5, 0.5, (tris, 3, 3))).reshape(-1, 3)
    workloads.write_obj(str(path / "tris.obj"), v, np.arange(3 * tris).reshape(-1, 3))
    s = sc.Scene()
    s.render(width=40, height=30, spp=4, max_depth=4, seed=3, clamp=0.0)
    s.camera(lookfrom=[0, 0.4, 3.2], lookat=[0, 0, 0], vfov=50)
    s.background_gradient(horizon=[0.6, 0.65, 0.7], zenith=[0.2, 0.3, 0.5])
    s.lambert("grey", color=[0.6, 0.6, 0.6])
    s.dielectric("glass", ior=1.4)
    s.point_light(position=[1.5, 4.0, 2.5], intensity=[40, 38, 34], radius=0.2)
    s.mesh("m", "tris.obj", normals="flat")
    s.add("mesh:m", "grey")
    s.add("mesh:m", "glass", sc.rotate_y(70), sc.scale(0.6), sc.translate(0.7, 0.2, 0.6))
    s.add("rect", "grey", sc.scale(4), sc.translate(0, -1.2, 0))
    return s


@pytest.mark.parametrize("what", ["cutouts", 1, 4, 5, 8, 37])
def test_walks_agree(lib, tmp_path, what):
    """Same nodes, same tests, so the same hits: the engines trace the same
    rays up to decisions that FP32 rounding of their shading flips, and their
    films agree to that rounding (1e-4 relative for 99% of the values)."""
    if what == "cutouts":
        s = workloads.textured(str(tmp_path), width=60, height=40, spp=8)
    else:
        s = _leaves(what, tmp_path)
    films, rays = [], []
    for engine in (1, 2):
        with sc.Session(s, base_dir=str(tmp_path), engine=engine) as ses:
            rays.append(ses.render().rays_traced)
            films.append(ses.read()[..., :3].astype(np.float64))
    err = np.abs(films[0] - films[1]) / np.maximum(np.abs(films[0]), 1e-3)
    assert abs(rays[0] - rays[1]) <= 2e-3 * rays[0]
    assert np.quantile(err, 0.99) <= 1e-4
