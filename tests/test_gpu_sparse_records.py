"""Records of which few in each warp are to be changed: evolve and the light
map change those in place, and the light map spreads few rays' planes over
the block's threads.  Records and maps equal the oracle's either side of the
lines (12 records a warp; 64, 32, ... rays a block of 128), others keep their
bytes."""
import numpy as np
import pytest

from helpers import assert_rays_equal, random_rays, small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu


def _pick(n, per_warp, status, other, seed):
    """per_warp records of every 32 have the status."""
    rng = np.random.default_rng(seed)
    out = np.full(n, other, np.uint8)
    for w in range(0, n, 32):
        m = min(32, n - w)
        out[w + rng.permutation(m)[: min(per_warp, m)]] = status
    return out


@pytest.mark.parametrize("per_warp", [1, 12, 13, 32])
@pytest.mark.parametrize("n", [40, 1000])
def test_evolve(per_warp, n):
    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    scene = tracer.Scene(tris, fd)
    rays = random_rays(n, 7 + n, tris.shape[0])
    rays["status"] = _pick(n, per_warp, T.STATUS_ACTIVE, T.STATUS_INFINITY, 3)
    hit, _ = O.next_hit(rays, tris)
    draws = np.array([O.fresnel_draw(11, k, 1) for k in range(n)], np.float32)
    d = tracer.rays_to_device(rays)
    import torch

    tracer.evolve(scene, d, torch.from_numpy(hit).cuda(), S.CAUCHY_GLASS, seed=11)
    got = tracer.rays_to_host(d)
    assert_rays_equal(got, O.evolve(rays, hit, tris, draws, fd, S.CAUCHY_GLASS), "evolve")
    idle = rays["status"] != T.STATUS_ACTIVE
    # the records' own bytes, padding with them (indexing records would not copy that)
    raw = d.cpu().numpy().reshape(n, -1), np.ascontiguousarray(rays).view(np.uint8).reshape(n, -1)
    assert np.array_equal(raw[0][idle], raw[1][idle])
    assert scene.errors() == 0


@pytest.mark.parametrize("per_warp", [1, 4, 8, 9, 12, 13, 16, 17, 32])
@pytest.mark.parametrize("planes,upscale", [(0, 1), (1, 2), (3, 1), (8, 2), (64, 3)])
def test_light_map(per_warp, planes, upscale):
    import torch

    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    scene = tracer.Scene(tris, fd)
    n = 300
    rays = random_rays(n, 21, tris.shape[0], aim=1.0)
    rays["dp_dx"] *= 3.0
    rays["status"] = _pick(n, per_warp, T.STATUS_DIFFUSE, T.STATUS_INFINITY, per_warp)
    hit, _ = O.next_hit(rays, tris)
    spec = S.stratified_spectrum(planes) if planes else None
    tex = tracer.new_light_map(24, 16, max(planes, 1), "i32")
    d = tracer.rays_to_device(rays)
    tracer.continuum_light_map2(scene, d, torch.from_numpy(hit).cuda(), spec, upscale, tex)
    ref_tex = O.new_map(24, 16, max(planes, 1), "i32")
    ref = O.continuum_light_map(rays, hit, tris, spec, upscale, tex_i32=ref_tex)
    assert_rays_equal(tracer.rays_to_host(d), ref, "light map")
    assert np.array_equal(tex.cpu().numpy().ravel(), ref_tex.ravel(order="F")) and ref_tex.any()
    assert scene.errors() == 0
