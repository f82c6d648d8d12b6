"""The ways a render's waves run give one image, bit for bit: hits shaded in the order they came or sorted, and small
waves in one launch (a block's paths start to end) or as the wavefront's launches. A path's random numbers, state and
sums are its own in each, so the tolerance is none."""
import numpy as np
import pytest

from threert_b200 import _native as N
from threert_b200 import prep, scenes
from threert_b200.serve import Request, Server, run_stream
from util import scaled_units_scene, small_city, small_crowd

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


# One pixel, ragged tiles, a path a block and the most paths of one round of blocks (94,720 on 148 SMs: 256 x 368 tiles
# of one sample, 128 x 92 of eight), and one tile row past it; a sort flag keeps the wavefront.
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (1, 1, 37), (7, 5, 3), (33, 31, 1), (64, 64, 1), (250, 370, 1),
                                     (256, 370, 1), (256, 372, 1), (127, 92, 8)])
@pytest.mark.parametrize("make", [lambda: scenes.cornell(16, 16), small_city, scaled_units_scene])
def test_small_waves_render_the_wavefronts_image(gpu, make, w, h, spp):
    P = prep.prepare(make())
    S = gpu.upload(P)
    same(S, sized(P, w, h), spp, N.TRT_RENDER_DEPTH, N.TRT_RENDER_DEPTH | N.TRT_RENDER_SORT_RAYS)


@pytest.mark.parametrize("bounces", [0, 1, 12])
def test_small_waves_of_few_and_many_vertices(gpu, bounces):
    P = prep.prepare(scenes.cornell(16, 16))
    S = gpu.upload(P)
    same(S, sized(P, 40, 24, max_bounces=bounces), 5, 0, N.TRT_RENDER_SORT_RAYS)


def test_small_waves_resume_and_accumulate(gpu):
    P = prep.prepare(small_city())
    S = gpu.upload(P)
    p = sized(P, 50, 30)
    whole, _ = S.render_raw(p, 6)
    S.render_raw(p, 2)
    got, _ = S.render_raw(p, 4, first_sample=2, flags=N.TRT_RENDER_ACCUMULATE)
    assert np.array_equal(whole.view(np.uint32), got.view(np.uint32))


def test_a_scene_of_four_suns_and_one_of_no_lights(gpu):
    """Every shadow slot of a vertex in use, and none."""
    d = small_city()
    d.lights = [prep.DirLight(direction=(0.3 * k - 0.5, -1.0, 0.2 * k), intensity=3000.0 * (k + 1)) for k in range(4)]
    for desc in (d, prep.SceneDescription(d.meshes[:2], d.materials[:2], d.instances[:2], d.camera, preset=d.preset)):
        P = prep.prepare(desc)
        S = gpu.upload(P)
        same(S, sized(P, 61, 43), 3, 0, N.TRT_RENDER_SORT_RAYS)


def many_units():
    """264 units turned, scaled unevenly, mirrored or moved alone, some that cast no shadow."""
    d = scaled_units_scene()
    rng = np.random.default_rng(11)
    for k in range(240):
        w = scenes.translate_rot_y(rng.uniform(-9, 9, 3), rng.uniform(0, 6.28), rng.uniform(-1.5, 1.5, 3))
        if k % 3 == 0:
            w = scenes.translate_rot_y(rng.uniform(-9, 9, 3))
        d.instances.append(prep.Instance(k % 2, [k % 2], w, object=24 + k, cast_shadow=k % 4 != 0))
    return d


# Waves around the sizes from which the walks run as streams of rays (131,072 paths for shadow rays, 262,144 for the
# others), and of two halves; the counted render walks ray by ray.
@pytest.mark.parametrize("w,h,spp", [(359, 362, 1), (363, 363, 1), (515, 509, 1), (1030, 514, 1), (201, 163, 9)])
@pytest.mark.parametrize("make", [many_units, lambda: small_city(n_objects=260), lambda: small_crowd(260).desc])
def test_streams_of_rays_hit_what_single_walks_hit(gpu, make, w, h, spp):
    P = prep.prepare(make())
    assert int(P.params[71]) >= 256
    S = gpu.upload(P)
    same(S, sized(P, w, h), spp, N.TRT_RENDER_DEPTH, N.TRT_RENDER_DEPTH | N.TRT_RENDER_COUNT)


# The server's steps of several scenes, of the size classes 65,536 (ray by ray), 131,072 (the shadow rays as a stream) and
# 524,288 (both, and the hits sorted): each request's image is its own render's.
@pytest.mark.parametrize("side,spp", [(60, 3), (91, 3), (181, 3)])
def test_a_servers_streams_of_several_scenes_rays(gpu, side, spp):
    Ps = [prep.prepare(d) for d in (scenes.cornell(16, 16), small_city(), many_units())]
    S = [gpu.upload(P) for P in Ps]
    reqs = [Request(k % 3, sized(Ps[k % 3], side + 2 * k, side - k), spp) for k in range(4)]
    srv = Server(gpu, wave_slots=1 << 20)
    try:
        res = run_stream(srv, S, reqs, rate=0.0)
    finally:
        srv.close()
    assert res["failed"] == 0
    for r in reqs:
        alone, _ = S[r.scene].render_raw(r.params, r.spp)
        assert np.array_equal(r.accum.view(np.uint32), alone.view(np.uint32))


@pytest.mark.parametrize("w,h", [(363, 363), (630, 640)])
def test_a_leafs_count_is_any_number_but_zero(gpu, w, h):
    """A top leaf's count only says that it is a leaf: the streams take the largest there is as single walks do."""
    P = prep.prepare(many_units())
    P.nodes = P.nodes.copy()
    nodes = P.nodes.reshape(-1, 8)
    top, n = int(P.params[70]), int(P.params[71])
    leaves = top + np.flatnonzero(nodes[top:top + 2 * n - 1, 7] != 0)
    assert len(leaves) == n
    nodes[leaves[::2], 7] = 0xFFFFFFFF
    same(gpu.upload(P), sized(P, w, h), 1, 0, N.TRT_RENDER_COUNT)
