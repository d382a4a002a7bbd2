"""The arrays films are read into."""

import collections
import resource

import numpy as np

from sundog_b200 import scene as sc

Size = collections.namedtuple("Size", "width height")


def test_film_arrays_have_their_pages():
    """Every page of a new array has memory behind it before the device copies
    into it: writing all of it takes no page faults to speak of."""
    a = sc._host_film(Size(4096, 2000))  # 131 MB: never recycled heap memory
    assert a.shape == (2000, 4096, 4) and a.dtype == np.float32 and a.flags.c_contiguous
    before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
    a.fill(1.0)
    faults = resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before
    assert faults <= a.nbytes // 4096 // 100


def test_small_film_arrays():
    for w, h in ((1, 1), (3, 5), (64, 1), (257, 1)):
        a = sc._host_film(Size(w, h))
        assert a.shape == (h, w, 4)
        a[:] = 2.0
        assert (a == 2.0).all()
