"""The brute-force hitters' merged boxes: results equal the oracle's plain
search over every triangle, bit for bit, at the edges of groups (8), boxes
(32), tiles (32 / 64 / 128) and runs of tiles, for meshes in any order, and
for caller records whose boxes must not be trusted."""
import numpy as np
import pytest

from helpers import random_rays
from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu


def _mesh(n, shuffled, seed=3):
    """n triangles of a displaced sphere, in mesh order or shuffled."""
    k = next(k for k in range(1, 8) if 20 * 4 ** k >= n)
    g = S.sphere_tris(k, noise_amp=0.05, noise_seed=seed)[:n]
    if shuffled:
        g = g[np.random.default_rng(seed).permutation(n)]
    return np.concatenate([np.zeros((1, 10, 3), np.float32), g.astype(np.float32)], 0)


@pytest.mark.parametrize("tile", [32, 64, 128])
@pytest.mark.parametrize("n", [1, 7, 9, 33, 65, 257, 1000, 5000])
@pytest.mark.parametrize("shuffled", [False, True])
def test_resident_records(tile, n, shuffled):
    from splat_gb300 import _lib as L
    from splat_gb300 import tracer

    tris = _mesh(n, shuffled)
    rays = random_rays(777, 5 + n, tris.shape[0])
    rays["dir"][5] = np.nan
    rays["dir"][6] = 0.0
    rays["pos"][7] = np.inf
    o_hit, o_t = O.next_hit(rays, tris)
    d = tracer.rays_to_device(rays)
    scene = tracer.Scene(tris, tris.shape[0] + 1, bvh=False)
    lib = L.load()
    old = lib.splat_get_tuning(L.TUNE_BRUTE_TILE)
    try:
        L.check(lib.splat_set_tuning(L.TUNE_BRUTE_TILE, tile))
        hit, t = tracer.next_hit(scene, tracer.BRUTE, d, with_t=True)
        many = tracer.next_hit(scene, tracer.BRUTE, d.repeat(400)) if n == 1000 else None
    finally:
        L.check(lib.splat_set_tuning(L.TUNE_BRUTE_TILE, old))
    assert np.array_equal(hit.cpu().numpy(), o_hit)
    assert np.array_equal(t.cpu().numpy().view(np.uint32), o_t.view(np.uint32))
    if many is not None:
        assert np.array_equal(many.cpu().numpy(), np.tile(o_hit, 400))
    assert scene.errors() == 0


def test_more_tiles_than_a_run():
    """34,000 records are 1,063 tiles of 32: three runs of 512 in one range."""
    from splat_gb300 import _lib as L
    from splat_gb300 import tracer

    tris = _mesh(34000, False)
    rays = random_rays(300, 8, tris.shape[0])
    o_hit, _ = O.next_hit(rays, tris)
    # enough rays that the triangle range is not split
    d = tracer.rays_to_device(rays).repeat(1100)
    scene = tracer.Scene(tris, tris.shape[0] + 1, bvh=False)
    lib = L.load()
    old = lib.splat_get_tuning(L.TUNE_BRUTE_TILE)
    try:
        L.check(lib.splat_set_tuning(L.TUNE_BRUTE_TILE, 32))
        hit = tracer.next_hit(scene, tracer.BRUTE, d)
    finally:
        L.check(lib.splat_set_tuning(L.TUNE_BRUTE_TILE, old))
    assert np.array_equal(hit.cpu().numpy(), np.tile(o_hit, 1100))
    assert scene.errors() == 0


@pytest.mark.parametrize("n", [1, 9, 65, 1281])
@pytest.mark.parametrize("odd", ["plain", "normals", "slivers", "far", "degenerate", "shuffled"])
def test_caller_records(n, odd):
    from splat_gb300 import tracer

    tris = _mesh(n, odd == "shuffled", 11)
    rng = np.random.default_rng(n)
    rays = random_rays(1025, 9 + n, tris.shape[0])
    if odd == "normals":  # planes that are not the triangles' own
        tris[1::2, 0] = rng.normal(size=tris[1::2, 0].shape)
    elif odd == "slivers":
        w = rng.uniform(0.0, 1e-3, (len(tris[1::2]), 1)).astype(np.float32)
        tris[1::2, 3] = tris[1::2, 2] + w * (tris[1::2, 1] - tris[1::2, 2]) + 1e-6
        tris[1:, 0] = np.cross(tris[1:, 1] - tris[1:, 2], tris[1:, 2] - tris[1:, 3])
    elif odd == "far":
        far = rng.integers(0, len(rays), 300)
        rays["pos"][far] -= rays["dir"][far] * rng.uniform(50.0, 20000.0, (300, 1)).astype(np.float32)
    elif odd == "degenerate":
        tris[1::3, 3] = tris[1::3, 2]
        tris[2::5, 1:4] = 0.0
        tris[1:, 0] = np.cross(tris[1:, 1] - tris[1:, 2], tris[1:, 2] - tris[1:, 3])
        tris[1::7, 2] = np.nan
        rays["pos"][3] = np.nan
        rays["dir"][4] = 0.0
    o_hit, o_t = O.next_hit(rays, tris)
    hit, tmp = tracer.next_hit_brute(tracer.rays_to_device(rays), tracer.n_tris_array(tris))
    assert np.array_equal(hit.cpu().numpy(), o_hit)
    packed = tmp.cpu().numpy().view(np.uint64)
    dec = np.array([O.monotonic_f32(int(k >> np.uint64(32))) for k in packed], dtype=np.float32)
    assert np.array_equal(dec.view(np.uint32), o_t.view(np.uint32))
