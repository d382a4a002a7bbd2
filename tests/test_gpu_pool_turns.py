"""Launches of more paths than the slot pool holds (64 M): the pool takes
them in turns, each through all its depths.

A film of few pixels has that many path indices at a modest cost: a row or
column of a tile is mostly padding. Its samples must not depend on the turns,
nor on how they are split over launches: byte for byte."""

import numpy as np
import pytest

from sundog_b200 import scene as sc
from sundog_b200 import workloads

pytestmark = pytest.mark.gpu

SLOTS = 1 << 26


@pytest.mark.parametrize("name,depth", [("cornell", 8), ("features", 19), ("opaque", 8),
                                        ("flames", 9)])
def test_film_independent_of_pool_turns(lib, tmp_path, name, depth):
    """Emission and NEE, depths past a group of iterations, opaque shadows
    beside flames (the shadow stage on the second stream when a turn ends),
    late vertices."""
    if name in ("opaque", "flames"):
        s = workloads.volumes(str(tmp_path))
        s.render(transparent_shadows=name == "flames")
    else:
        s = getattr(workloads, name)()
    w, h, spp = 9, 1, 540000
    s.render(max_depth=depth)
    padded = 16 * 8 * spp
    assert SLOTS < padded < 2 * SLOTS and padded % SLOTS
    opts = dict(base_dir=str(tmp_path), width=w, height=h, spp=spp, aov=name == "features")
    with sc.Session(s, chunk_spp=spp, **opts) as whole:
        a = whole.render()
        fa = whole.read()
    with sc.Session(s, chunk_spp=spp // 2 + 1, **opts) as halves:
        b = halves.render()
        fb = halves.read()
    assert a.rays_traced == b.rays_traced > w * h * spp
    for x, y in zip(fa, fb):  # rows, or film and AOVs
        assert np.array_equal(x, y)
