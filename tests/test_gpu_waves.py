"""The ways a render's waves run give one image, bit for bit: hits shaded in the order they came or sorted. A path's
random numbers, state and sums are its own, so the tolerance is none."""
import numpy as np
import pytest

from threert_b200 import _native as N
from threert_b200 import prep
from util import small_city, small_crowd

pytestmark = pytest.mark.gpu


def sized(P, w, h, **kw):
    p = P.with_size(w, h)
    return prep.params_with(p, **kw) if kw else p


def same(S, params, spp, flags_a, flags_b, **kw):
    a, st_a = S.render_raw(params, spp, flags=flags_a, **kw)
    b, st_b = S.render_raw(params, spp, flags=flags_b, **kw)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert (st_a.closest_rays, st_a.shadow_rays, st_a.paths) == (st_b.closest_rays, st_b.shadow_rays, st_b.paths)
    return a


# Waves around the sort's threshold of 393,216 paths (a size below it, the first multiple of the tiles past it, and a
# wave of two halves), in scenes of many units, and of one unit of many sections.
@pytest.mark.parametrize("w,h,spp", [(627, 620, 1), (629, 631, 1), (517, 259, 5)])
@pytest.mark.parametrize("make", [small_city, lambda: small_crowd().desc])
def test_sorted_hits_shade_the_same_image(gpu, make, w, h, spp):
    P = prep.prepare(make())
    S = gpu.upload(P)
    same(S, sized(P, w, h), spp, 0, N.TRT_RENDER_UNSORTED_HITS)
