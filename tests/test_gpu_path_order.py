"""Path numbering and pool bookkeeping of the wavefront engine.

A launch of S samples numbers its paths pixel by pixel, the samples of a
pixel consecutive; a launch of one sample numbers its pixels. Every sample's
random stream depends on (pixel, sample, seed) only and the film folds them
in sample order, so a film must not depend on how its samples are split over
launches: byte for byte."""

import numpy as np
import pytest

from sundog_b200 import scene as sc
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
