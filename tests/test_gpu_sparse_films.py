"""Megakernel films that are mostly tile padding number their samples first:
the same film as by pixels, and as one sample at a time."""

import numpy as np
import pytest

from sundog_b200 import scene as sc
from sundog_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (101, 1), (1, 37), (9, 2), (17, 9)])
def test_film_independent_of_numbering(lib, size):
    opts = dict(width=size[0], height=size[1], spp=33, aov=True, engine=1)
    with sc.Session(workloads.features(), **opts) as whole:
        a = whole.render()
        fa = whole.read()
    with sc.Session(workloads.features(), chunk_spp=1, **opts) as single:
        b = single.render()
        fb = single.read()
    assert a.rays_traced == b.rays_traced
    for x, y in zip(fa, fb):
        assert np.array_equal(x, y)
