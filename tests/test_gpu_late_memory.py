"""Device memory of late vertices (paths that wait for their shadow ray before
they go on: flames along it, training records). They lie in a buffer of their
own, sized to the launch that has some."""

import pytest

from sundog_b200 import abi, scene as sc, serve
from sundog_b200 import workloads
from test_gpu_memory import SLACK, free_bytes

pytestmark = pytest.mark.gpu

LATE_BYTES = 80  # a late vertex


def test_small_flame_render_keeps_a_large_pool(lib, tmp_path):
    """A pool kept from a frame of 4.9 M paths serves a 16x16 render with a
    flame as it is: that render adds its own few vertices and the scene."""
    big = workloads.cornell(width=640, height=480, spp=16)
    small = workloads.volumes(str(tmp_path), width=16, height=16, spp=2)

    def render(s, **opts):
        with sc.Session(s, base_dir=str(tmp_path), **opts) as ses:
            ses.render()
            return ses.read()
    want = render(small)
    try:
        abi.check(lib.sundog_set_device_memory_cache(1), "cache", lib)
        render(big)
        held = free_bytes()
        film = render(small)
        assert held - free_bytes() <= SLACK
        assert film.tobytes() == want.tobytes()
    finally:
        abi.check(lib.sundog_set_device_memory_cache(0), "cache", lib)


def test_server_holds_late_vertices_from_its_first_flame_job(lib, tmp_path):
    cfg = dict(iteration_paths=1 << 22)
    plain = workloads.cornell(width=64, height=64, spp=2)
    flame = workloads.volumes(str(tmp_path), width=64, height=48, spp=2)
    with serve.Server(**cfg) as sv:
        sv.submit(plain).wait()
        before = free_bytes()
        a = sv.submit(flame, base_dir=str(tmp_path)).wait()
        grown = before - free_bytes()
        assert grown >= (1 << 22) * LATE_BYTES
        b = sv.submit(flame, base_dir=str(tmp_path)).wait()
        assert before - free_bytes() - grown <= SLACK
    assert a.tobytes() == b.tobytes()
