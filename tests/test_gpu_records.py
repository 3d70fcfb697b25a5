"""The kernels that go over whole arrays of ray records: counts around a
warp's and a block's edges, record arrays at every alignment a caller's
pointer can have, and rays that are not active when run_evolution! starts."""
import ctypes as C

import numpy as np
import pytest

from helpers import assert_rays_equal, random_rays, small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu

SZ = T.ADRAY.itemsize


def _statuses(rays, seed, p=0.5):
    rng = np.random.default_rng(seed)
    n = len(rays)
    rays["status"] = np.where(rng.uniform(size=n) < p, T.STATUS_ACTIVE,
                              rng.choice([T.STATUS_DIFFUSE, T.STATUS_INFINITY], size=n))
    rays["dest"] = np.arange(n)
    return rays


@pytest.mark.parametrize("n", [1, 31, 33, 257, 1500])
@pytest.mark.parametrize("depth", [0, 1, 3])
@pytest.mark.parametrize("hitter", ["brute", "bvh"])
def test_run_evolution_with_idle_rays(n, depth, hitter):
    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    scene = tracer.Scene(tris, fd)
    rays = _statuses(random_rays(n, 7 + n, tris.shape[0]), n, 0.0 if n == 257 else 0.6)
    d = tracer.rays_to_device(rays)
    h = tracer.BVH if hitter == "bvh" else tracer.BRUTE
    hit = tracer.run_evolution(h, scene, d, depth, S.CAUCHY_GLASS, None, seed=3)
    ref, _ = O.run_evolution(rays, tris, depth, fd, S.CAUCHY_GLASS, None, seed=3)
    ref_hit, _ = O.next_hit(ref, tris)  # the realigning hit covers every ray, active or not
    assert_rays_equal(tracer.rays_to_host(d), ref, "idle rays")
    assert np.array_equal(hit.cpu().numpy(), ref_hit)
    assert scene.errors() == 0


@pytest.mark.parametrize("n", [1, 32, 255, 513])
@pytest.mark.parametrize("shift", [0, 1])
def test_records_at_odd_offsets(n, shift):
    """The record array one record into an allocation is 8-byte aligned only;
    every whole-array kernel gives the bytes of the aligned array and touches
    no neighbour."""
    import torch

    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    scene = tracer.Scene(tris, fd)
    light = T.rect_light((0.0, 3.0, 0.0), (0.0, -1.0, 0.0), (1.0, 0.0, 0.0), (0.0, 0.0, 1.0), n, 1)
    rays = O.rays_from_light(light, 1, (T.LAMBDA_UNIFORM, 1, 400.0, 700.0), seed=5)
    lib, L = tracer.L.load(), tracer.L
    buf = torch.full(((n + 2) * SZ,), 0xAB, dtype=torch.uint8, device="cuda")
    view = buf[shift * SZ: (shift + n) * SZ]
    li, lm = tracer._light(light), tracer._lmode((T.LAMBDA_UNIFORM, 1, 400.0, 700.0))
    L.check(lib.splat_rays_from_light(C.byref(li), 1, C.byref(lm), 5, 0, view.data_ptr(), tracer._stream()))
    assert_rays_equal(tracer.rays_to_host(view), rays, "generated")
    start = _statuses(rays.copy(), 3, 0.7)
    view.copy_(tracer.rays_to_device(start))
    hit = tracer.next_hit(scene, tracer.BVH, view)
    tracer.evolve(scene, view, hit, S.CAUCHY_GLASS, seed=11)
    ref_hit, _ = O.next_hit(start, tris)
    assert np.array_equal(hit.cpu().numpy(), ref_hit)
    draws = np.array([O.fresnel_draw(11, k, 1) for k in range(n)], np.float32)
    plain = tracer.rays_to_device(start)
    tracer.evolve(scene, plain, hit, S.CAUCHY_GLASS, seed=11)
    assert torch.equal(view, plain)
    assert_rays_equal(tracer.rays_to_host(view), O.evolve(start, ref_hit, tris, draws, fd, S.CAUCHY_GLASS), "evolve")
    h2 = tracer.run_evolution(tracer.BVH, scene, view, 2, S.CAUCHY_GLASS, None, seed=2)
    ref, _ = O.run_evolution(tracer.rays_to_host(plain), tris, 2, fd, S.CAUCHY_GLASS, None, seed=2)
    ref_hit2, _ = O.next_hit(ref, tris)
    assert np.array_equal(h2.cpu().numpy(), ref_hit2)
    assert_rays_equal(tracer.rays_to_host(view), ref, "run_evolution")
    tex = tracer.new_light_map(24, 16, 3, "i32")
    tracer.continuum_light_map2(scene, view, h2, S.stratified_spectrum(3), 2, tex)
    ref_tex = O.new_map(24, 16, 3, "i32")
    ref2 = O.continuum_light_map(ref, ref_hit2, tris, S.stratified_spectrum(3), 2, tex_i32=ref_tex)
    assert_rays_equal(tracer.rays_to_host(view), ref2, "light map")
    assert np.array_equal(tex.cpu().numpy().ravel(), ref_tex.ravel(order="F"))
    rows, raw = tracer.rays_to_host(view), view.cpu().numpy().reshape(n, SZ)
    count = int(tracer.partition(view).item())
    after = tracer.rays_to_host(view)
    assert count == int((rows["status"] == T.STATUS_ACTIVE).sum())
    assert (after["status"][:count] == T.STATUS_ACTIVE).all() and (after["status"][count:] != T.STATUS_ACTIVE).all()
    assert sorted(r.tobytes() for r in raw) == sorted(r.tobytes() for r in view.cpu().numpy().reshape(n, SZ))
    rest = torch.cat([buf[: shift * SZ], buf[(shift + n) * SZ:]])
    assert bool((rest == 0xAB).all())
    assert scene.errors() == 0
