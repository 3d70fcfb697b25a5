"""The brute-force hitters let every lane go over the groups of records its
own ray enters: rays that are strangers to one another, at the edges of
groups (8), tiles and the n_tris hitter's line between its two kernels (96),
with coincident records that tie.  Hits equal the oracle's plain search."""
import numpy as np
import pytest

from helpers import random_rays
from oracle import oracle as O
from splat_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _mesh(n, large, seed=4):
    """n triangles, some twice: of a sphere, or as large as the scene."""
    rng = np.random.default_rng(seed)
    if large:
        P = rng.uniform(-1.0, 1.0, (n, 3, 3))
        e = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
        N = np.repeat((e / np.linalg.norm(e, axis=1, keepdims=True))[:, None], 3, 1)
        g = S.ftri_records(P, N, np.zeros_like(P))
    else:
        k = next(k for k in range(1, 8) if 20 * 4 ** k >= n)
        g = S.sphere_tris(k, noise_amp=0.05, noise_seed=seed)
        g = g[rng.permutation(len(g))[:n]]
    g[n // 2: n // 2 + n // 10] = g[: n // 10]
    return np.concatenate([np.zeros((1, 10, 3), np.float32), np.asarray(g, np.float32)], 0)


@pytest.mark.parametrize("n", [7, 94, 95, 96, 97, 103, 255, 256, 300, 769])
@pytest.mark.parametrize("large", [False, True])
def test_strangers(n, large):
    from splat_gb300 import _lib as L
    from splat_gb300 import tracer

    tris = _mesh(n, large)
    rays = random_rays(1337, n, n + 1, aim=0.9)
    rays["dir"][::9] = np.eye(3, dtype=np.float32)[np.arange(len(rays[::9])) % 3]
    o_hit, o_t = O.next_hit(rays, tris)
    assert int((o_hit != 1).sum()) > 50
    d = tracer.rays_to_device(rays)
    hit, tmp = tracer.next_hit_brute(d, tracer.n_tris_array(tris))
    assert np.array_equal(hit.cpu().numpy(), o_hit)
    dec = np.array([O.monotonic_f32(int(k >> np.uint64(32))) for k in tmp.cpu().numpy().view(np.uint64)], np.float32)
    assert np.array_equal(dec.view(np.uint32), o_t.view(np.uint32))
    scene = tracer.Scene(tris, n + 2, bvh=False)
    lib = L.load()
    old = lib.splat_get_tuning(L.TUNE_BRUTE_TILE)
    try:
        for tile in (32, 64, 128):
            L.check(lib.splat_set_tuning(L.TUNE_BRUTE_TILE, tile))
            hit, t = tracer.next_hit(scene, tracer.BRUTE, d, with_t=True)
            assert np.array_equal(hit.cpu().numpy(), o_hit), tile
            assert np.array_equal(t.cpu().numpy().view(np.uint32), o_t.view(np.uint32)), tile
    finally:
        L.check(lib.splat_set_tuning(L.TUNE_BRUTE_TILE, old))
    assert scene.errors() == 0


def test_the_earlier_record_wins_on_both_sides_of_the_line():
    """Coincident records whose indices fall along the array: the earlier one
    is the hit, whichever kernel takes the array."""
    import torch

    from splat_gb300 import tracer

    for n in (60, 180):
        tris = _mesh(n, False)
        half = (n + 1) // 2
        tris[1 + half: 1 + 2 * half] = tris[1: 1 + half][: len(tris[1 + half: 1 + 2 * half])]
        rays = random_rays(900, 3, n + 1)
        rays["ignore_tri"] = 1
        nt = tracer.n_tris_array(tris).cpu().numpy().view(np.int32).reshape(-1, 13).copy()
        nt[1:, 0] = np.arange(len(nt), 1, -1)  # descending
        hit, _ = tracer.next_hit_brute(tracer.rays_to_device(rays), torch.from_numpy(nt.view(np.uint8).reshape(-1)).cuda())
        ref, _ = O.next_hit(rays, tris)  # ties take the smaller ascending index: the earlier record
        assert int((ref != 1).sum()) > 100
        assert np.array_equal(hit.cpu().numpy(), np.where(ref == 1, 1, len(nt) + 2 - ref))
