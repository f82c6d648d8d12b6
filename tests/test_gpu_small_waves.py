"""The last vertices of a small wave's paths (k_paths takes each path of a block from the camera to the end): where every
path of a block ends at once and none leaves a shadow ray, the vertex's light that needs no ray and the non-finite fix
still reach the image. Against the wavefront bit for bit (a path's sums are its own, so the tolerance is none), and
against the oracle."""
import numpy as np
import pytest

import oracle
from threert_b200 import _native as N
from threert_b200 import prep, scenes
from threert_b200.serve import Request, Server, run_stream

from test_gpu_pass import image_parity
from test_gpu_waves import same, sized

pytestmark = pytest.mark.gpu


def unshadowed(intensity=5000.0):
    """Dark rough metal under a light that casts no shadow and no sky: a vertex's light never asks for a ray, and
    Russian roulette from the first vertex and directions below the surface end most paths there."""
    metal = prep.Material(base=(0.3, 0.25, 0.2), metallic=1.0, roughness=0.8)
    inst = [prep.Instance(0, [0], object=0), prep.Instance(1, [0], scenes.translate_rot_y((0.0, 0.7, 0.0)), object=1)]
    light = prep.DirLight(direction=(-0.3, -1.0, -0.4), intensity=intensity, cast_shadow=False)
    cam = prep.Camera.look_at((0.0, 2.0, 4.0), (0.0, 0.4, 0.0), 45.0, 48, 48)
    return prep.SceneDescription([scenes.plane_mesh(12.0), scenes.sphere_mesh(0.7, 16, 10)], [metal], inst, cam,
                                 lights=[light], sky=prep.Sky("none"), preset=prep.Preset(max_bounces=4, rr_depth=0))


@pytest.mark.parametrize("w,h", [(1, 1), (16, 16), (33, 31), (64, 64)])
@pytest.mark.parametrize("spp", [1, 8])
def test_light_without_a_shadow_ray_at_the_last_vertices(gpu, w, h, spp):
    S = gpu.upload(P := prep.prepare(unshadowed()))
    acc = same(S, sized(P, w, h), spp, 0, N.TRT_RENDER_SORT_RAYS)
    assert (acc[:, 0:3] > 0).any()


def test_light_without_a_shadow_ray_is_the_oracles(gpu):
    P = prep.prepare(unshadowed())
    acc_g, _ = gpu.upload(P).render_raw(P.params, 8)
    acc_o, _ = oracle.Oracle(P).render(P.params, 8)
    frac, mean_err = image_parity(acc_g, acc_o, P.width, P.height, 8)
    assert frac >= 0.99 and mean_err <= 0.01, (frac, mean_err)


def test_a_served_request_of_that_scene_is_its_own_render(gpu):
    P = prep.prepare(unshadowed())
    S = gpu.upload(P)
    reqs = [Request(0, sized(P, 20 + 9 * k, 17), 2 + k) for k in range(3)]
    srv = Server(gpu, wave_slots=1 << 16)
    try:
        res = run_stream(srv, [S], reqs, rate=0.0)
    finally:
        srv.close()
    assert res["failed"] == 0
    for r in reqs:
        alone, _ = S.render_raw(r.params, r.spp)
        assert np.array_equal(r.accum.view(np.uint32), alone.view(np.uint32))


def infinite_emission():
    """The Cornell box with its light's emission infinite in the material's record (the light samples' table keeps its
    finite weights)."""
    P = prep.prepare(scenes.cornell(16, 16))
    P.tables = P.tables.copy()
    rows = P.tables.reshape(-1, 4)
    first, end = int(P.params[125]), int(P.params[126])
    n = (end - first) // 18
    mats = rows[first:first + 18 * n].reshape(n, 18, 4)  # (a view of the tables: base, emissive, ...)
    lit = mats[:, 1, :3].view(np.float32).max(1) > 0
    assert lit.sum() == 1
    mats[lit, 1, :3] = np.float32(np.inf).view(np.uint32)
    assert not np.isfinite(P.tables.view(np.float32)[4 * first:4 * end]).all()
    return P


@pytest.mark.parametrize("make", [infinite_emission, lambda: prep.prepare(unshadowed(float("inf")))])
@pytest.mark.parametrize("w,h,spp,bounces", [(1, 1, 1, 1), (16, 16, 1, 0), (33, 31, 1, 1), (40, 24, 8, 3), (64, 64, 1, 5)])
def test_a_paths_non_finite_radiance_is_dropped(gpu, make, w, h, spp, bounces):
    P = make()
    acc = same(gpu.upload(P), sized(P, w, h, max_bounces=bounces), spp, 0, N.TRT_RENDER_SORT_RAYS)
    assert np.isfinite(acc).all()
