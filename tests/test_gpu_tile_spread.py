"""The allocation-free tile render spreads its paths over warps by their number
and the scene: a film must not depend on how."""

import numpy as np
import pytest

from sundog_b200 import abi
from sundog_b200 import scene as sc
from sundog_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cornell", "volumes", "instancing"])
def test_tile_is_its_blocks(lib, tmp_path, name):
    """A tile against its blocks, rendered apart with other numbers of lanes a
    warp (1 to 32 paths), on both sides of the rules' lines at 148 and 4,736
    paths: byte for byte, as samples depend on pixel and sample alone."""
    import torch
    s = (workloads.cornell() if name == "cornell"
         else getattr(workloads, name)(str(tmp_path)))
    s.render(width=96, height=64, spp=16)
    with sc.Session(s, base_dir=str(tmp_path)) as ses:
        def tile(x, y, w, h, spp):
            film = torch.zeros(h, w, 4, device="cuda")
            rays = abi.ctypes.c_uint64(0)
            abi.check(ses.lib.sundog_session_render_tile_noalloc(
                ses.handle, x, y, w, h, 0, spp, film.data_ptr(), abi.ctypes.byref(rays), None),
                "tile", ses.lib)
            return film.cpu().numpy(), rays.value

        # 33x37 at 4 samples: 4,884 paths; at 3: 3,663; at 16: 19,536.
        for spp in (3, 4, 16):
            whole, rays = tile(21, 13, 33, 37, spp)
            parts, total = np.zeros_like(whole), 0
            for y0, y1 in ((0, 1), (1, 30), (30, 37)):
                for x0, x1 in ((0, 7), (7, 33)):
                    parts[y0:y1, x0:x1], r = tile(21 + x0, 13 + y0, x1 - x0, y1 - y0, spp)
                    total += r
            assert np.array_equal(whole, parts) and rays == total
