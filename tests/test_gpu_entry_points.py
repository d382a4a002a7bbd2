"""Every way to render, against the CPU oracle: a session with either engine,
a served job and the allocation-free tile render.

All take the same samples. Which product a sum of products fuses differs
between their kernels (Rounding, sd_bsdf.cuh), so a path through glass, water
or a rough interface may part from another kernel's in its last bits, and from
there on: films agree as two FP32 renders of the same samples do, not byte for
byte. Bounds are those of the whole-image parity tests (test_gpu_render.py).
The oracle's scene is this library's derivation, which test_scene_derivation.py
compares with sundog's own."""

import pytest

from oracle import oracle
from sundog_b200 import abi, serve, workloads
from sundog_b200 import scene as sc
from test_gpu_render import compare

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda d: workloads.cornell(width=64, height=64, spp=16),
    "features": lambda d: workloads.features(),
    "textured": lambda d: workloads.textured(d),
    "instancing": lambda d: workloads.instancing(d, width=96, height=54, spp=4),
    "volumes": lambda d: workloads.volumes(d, width=80, height=45, spp=4),
}


@pytest.fixture(scope="module")
def oracle_films(lib, oracle_lib, tmp_path_factory):
    base, kept = str(tmp_path_factory.mktemp("entry")), {}

    def get(name):
        if name not in kept:
            s = SCENES[name](base)
            h = s.build(base, lib)
            try:
                text, r = oracle.scene_text(sc.debug_json(h, lib), base)
            finally:
                lib.sundog_scene_destroy(h)
            osc = oracle.OracleScene(text)
            film, rays, _, _ = osc.render(0, 0, r["width"], r["height"], 0, r["spp"], threads=8)
            osc.close()
            kept[name] = s, r, film, rays
        return (base,) + kept[name]
    return get


def by_tile(s, base, r):
    import torch
    film = torch.zeros(r["height"], r["width"], 4, device="cuda")
    with sc.Session(s, base_dir=base) as ses:
        rays = abi.ctypes.c_uint64(0)
        abi.check(ses.lib.sundog_session_render_tile_noalloc(
            ses.handle, 0, 0, r["width"], r["height"], 0, r["spp"], film.data_ptr(),
            abi.ctypes.byref(rays), None), "tile", ses.lib)
    return film.cpu().numpy(), rays.value


def by_server(s, base, r):
    with serve.Server() as sv:
        film = sv.submit(s, base_dir=base).wait()
        return film, sv.stats().rays


def by_session(engine):
    def render(s, base, r):
        with sc.Session(s, base_dir=base, engine=engine) as ses:
            rays = ses.render().rays_traced
            return ses.read(), rays
    return render


WAYS = {"session": by_session(0), "megakernel": by_session(1), "server": by_server,
        "tile": by_tile}


@pytest.mark.parametrize("way", sorted(WAYS))
@pytest.mark.parametrize("name", sorted(SCENES))
def test_entry_point_matches_oracle(oracle_films, name, way):
    base, s, r, ofilm, orays = oracle_films(name)
    film, rays = WAYS[way](s, base, r)
    # Rare parted paths of the volumes scene reach its bright canopy light.
    compare("%s by %s" % (name, way), film, ofilm, rays, orays,
            relmse_max=1e-2 if name == "volumes" else 2e-3)
