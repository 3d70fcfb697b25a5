"""Rays and lights far away from a scene whose boxes stand in a turned frame:
turning a ray rounds by its origin's distance, which the boxes' padding alone
does not cover.  Hits by both trees and every traversal form equal the
oracle's plain search over every triangle, and steps lit from afar equal the
CPU restatement's."""
import numpy as np
import pytest

from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T
from test_gpu_small_step import _check

pytestmark = pytest.mark.gpu

TURNS = {"none": None, "any": 11, "other": 23}


def _scene(turn):
    R = np.eye(3) if TURNS[turn] is None else S.random_quaternion_matrix(TURNS[turn])
    return (*S.assemble(S.rotate(S.menger_tris(2, 2.0, None), R), S.floor_tris(-1.8, 1.5)), R)


def _far_rays(R, dist, n=4096, seed=7):
    """Aimed at the sponge's facets, half of them close to a facet's edge, from
    dist units off: along the world's axes, nearly along the facets' own, and
    from anywhere."""
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, T.ADRAY)
    target = rng.uniform(-1.0, 1.0, (n, 3))
    target[::2] = np.round((target[::2] + 1.0) * 4.5) / 4.5 - 1.0 + rng.normal(scale=1e-3, size=(n // 2, 3))
    target = target @ np.asarray(R).T
    d = rng.normal(size=(n, 3))
    k = n // 3
    axes = np.eye(3)[rng.integers(0, 3, 2 * k)] * rng.choice([-1.0, 1.0], (2 * k, 1))
    d[:k] = axes[:k]
    d[k: 2 * k] = (axes[k:] + rng.normal(scale=1e-3, size=(k, 3))) @ np.asarray(R).T
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    rays["pos"] = target - d.astype(np.float64) * dist
    rays["dir"] = d
    rays["ignore_tri"] = 1
    rays["status"] = T.STATUS_ACTIVE
    return rays


@pytest.mark.parametrize("dist", [600.0, 3000.0, 10000.0, 1.0e5])
@pytest.mark.parametrize("turn", list(TURNS))
def test_hits(turn, dist):
    from splat_gb300 import _lib as L
    from splat_gb300 import tracer

    tris, fd, R = _scene(turn)
    rays = _far_rays(R, dist)
    ref, tref = O.next_hit(rays, tris)
    assert int((ref != 1).sum()) > 500
    scene = tracer.Scene(tris, fd)
    d = tracer.rays_to_device(rays)
    lib = L.load()
    old = lib.splat_get_tuning(L.TUNE_BVH_PACKET)
    try:
        # a warp, eight lanes, one lane a ray; packets
        for hitter, packet, times in ((tracer.BVH, 1, 1), (tracer.BVH, 1, 4), (tracer.BVH, 1, 9), (tracer.BVH, 2, 1),
                                      (tracer.BVH2, 1, 1)):
            L.check(lib.splat_set_tuning(L.TUNE_BVH_PACKET, packet))
            hit, t = tracer.next_hit(scene, hitter, d.repeat(times), with_t=True)
            assert np.array_equal(hit.cpu().numpy(), np.tile(ref, times)), (hitter, packet, times)
            assert np.array_equal(t.cpu().numpy().view(np.uint32), np.tile(tref.view(np.uint32), times))
    finally:
        L.check(lib.splat_set_tuning(L.TUNE_BVH_PACKET, old))
    assert scene.errors() == 0


def _lit_from_afar(res, hitter="bvh"):
    tris, fd, _ = _scene("any")
    light = T.rect_light((0.0, 3000.0, 0.0), (0.0, -1.0, 0.0), (1.3, 0.0, 0.0), (0.0, 0.0, 1.3), *res)
    return S.Workload(name="far", tris=tris, first_diffuse=fd, light=light, upscale=1,
                      lambda_mode=(T.LAMBDA_STRATIFIED, 2, 400.0, 700.0), spectrum=S.stratified_spectrum(2), depth=3,
                      material=S.CAUCHY_GLASS, map_w=32, map_h=32, accum="i32", hitter=hitter, seed=4)


@pytest.mark.parametrize("hitter", ["bvh", "bvh2"])
@pytest.mark.parametrize("res", [(64, 64), (160, 128)])
def test_steps_lit_from_afar(res, hitter):
    _check(_lit_from_afar(res, hitter))


@pytest.mark.parametrize("dist", [600.0, 2000.0])
@pytest.mark.parametrize("turn", list(TURNS))
@pytest.mark.parametrize("n", [1024, 4096])
def test_brute_force(turn, dist, n):
    """The resident brute-force hitter's boxes stand in the world's frame and
    have their padding alone."""
    from splat_gb300 import tracer

    tris, fd, R = _scene(turn)
    rays = _far_rays(R, dist, n, 9)
    ref, tref = O.next_hit(rays, tris)
    scene = tracer.Scene(tris, fd, bvh=False)
    hit, t = tracer.next_hit(scene, tracer.BRUTE, tracer.rays_to_device(rays), with_t=True)
    assert np.array_equal(hit.cpu().numpy(), ref)
    assert np.array_equal(t.cpu().numpy().view(np.uint32), tref.view(np.uint32))
    assert scene.errors() == 0


@pytest.mark.parametrize("res", [(16, 16), (100, 90)])
def test_brute_force_steps_lit_from_afar(res):
    """One launch (a sponge of few facets), and separate ones."""
    wl = _lit_from_afar(res, "brute")
    if res[0] < 64:
        tris, fd = S.assemble(S.menger_tris(1, 2.0, 11), S.floor_tris(-1.8, 1.5))
        wl = wl.with_(tris=tris, first_diffuse=fd)
    _check(wl)
