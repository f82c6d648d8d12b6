"""The orders a wave's queues can be walked and shaded in, at the sizes where the hit sort and the walks as streams of
rays are on: the optional sorts' orders given to the streams, the hit sort after the ray sort, and the hit sort of a
scene of a few hundred units that each have one section. A path's random numbers, state and sums are its own in each, so
the tolerance is none."""
import pytest

from threert_b200 import _native as N
from threert_b200 import crowd, prep

from test_gpu_waves import many_units, same, sized
from util import small_city

pytestmark = pytest.mark.gpu

SORT_HITS_MIN_MATERIALS = 32  # threert_cuda.h TRT_SORT_HITS_MIN_MATERIALS
RAYS, SHADOWS = N.TRT_RENDER_SORT_RAYS, N.TRT_RENDER_SORT_SHADOWS


def materials(P):
    return (int(P.params[126]) - int(P.params[125])) // 18


def launches(S, params, spp, flags):
    S.reset_totals()
    S.render_raw(params, spp, flags=flags)
    return S.totals()["launches"]


# A wave whose shadow rays walk as a stream (131,072 paths and more), one whose closest hits do too and whose hits are
# sorted where the scene has the materials (393,216), and one of two halves; the counted render walks ray by ray.
@pytest.mark.parametrize("sorts", [RAYS, SHADOWS, RAYS | SHADOWS])
@pytest.mark.parametrize("w,h", [(363, 363), (630, 640), (1030, 514)])
@pytest.mark.parametrize("make", [many_units, lambda: small_city(n_objects=260)])
def test_streams_in_a_sorted_order_hit_what_single_walks_hit(gpu, make, w, h, sorts):
    P = prep.prepare(make())
    assert int(P.params[71]) >= 256
    same(gpu.upload(P), sized(P, w, h), 1, sorts, N.TRT_RENDER_COUNT | N.TRT_RENDER_UNSORTED_HITS)


# The hit sort alone and after the ray sort (then it writes the raw queue's room, not the sorted one's), among few
# units and many, with the launches that say it ran: two a depth.
@pytest.mark.parametrize("sorts", [0, RAYS])
@pytest.mark.parametrize("n_objects", [80, 260])
def test_hits_sorted_after_rays_shade_the_same_image(gpu, n_objects, sorts):
    P = prep.prepare(small_city(n_objects=n_objects))
    assert materials(P) > SORT_HITS_MIN_MATERIALS
    S = gpu.upload(P)
    p = sized(P, 640, 632)
    same(S, p, 1, sorts, N.TRT_RENDER_UNSORTED_HITS)
    depths = int(p[22]) + 1
    assert launches(S, p, 1, sorts) == launches(S, p, 1, sorts | N.TRT_RENDER_UNSORTED_HITS) + 2 * depths


def test_a_crowds_sorted_hits_shade_the_same_image(gpu):
    body = crowd.humanoid(segments=8, hemi_rings=3, body_rings=4)
    P = prep.prepare(crowd.crowd(n=160, groups=3, width=64, height=36, max_depth=3, extent=12.0, ground_segments=12,
                                 n_emitters=40, body=body, sky_size=(64, 32), sky="gradient").desc)
    assert materials(P) > SORT_HITS_MIN_MATERIALS
    S = gpu.upload(P)
    for w, h, spp in [(629, 631, 1), (517, 259, 5)]:
        p = sized(P, w, h)
        same(S, p, spp, 0, N.TRT_RENDER_UNSORTED_HITS)
        assert launches(S, p, spp, 0) > launches(S, p, spp, N.TRT_RENDER_UNSORTED_HITS)
