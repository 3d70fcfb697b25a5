"""GPU rebuilds at the edges of the sorted triangles' runs (32), groups of runs
(1,024) and sort tiles, and above the tiles a scatter block sums up itself:
hits by both BVHs equal the oracle's, the brute-force records follow, and a
step traces the rebuilt scene exactly."""
import numpy as np
import pytest

from helpers import random_rays
from oracle import oracle as O
from splat_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _tris(n, seed):
    """n triangles of a displaced sphere in shuffled order (some coincident)."""
    k = next(k for k in range(1, 9) if 20 * 4 ** k >= n)
    g = S.sphere_tris(k, noise_amp=0.08, noise_seed=seed)
    g = g[np.random.default_rng(seed).permutation(len(g))[:n]]
    g[n // 2: n // 2 + n // 20] = g[: n // 20]
    return np.concatenate([np.zeros((1, 10, 3), np.float32), g.astype(np.float32)], 0)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 32, 33, 63, 65, 1023, 1024, 1025, 1057, 2080, 5000])
def test_hits_after_a_rebuild(n):
    import torch

    from splat_gb300 import tracer

    scene = tracer.Scene(_tris(n, 3), n + 2)
    moved = _tris(n, 4)
    rays = random_rays(700, 5 + n, n + 1)
    rays["dir"][3] = np.nan
    rays["dir"][4] = (0.0, 1.0, 0.0)
    o_hit, o_t = O.next_hit(rays, moved)
    d = tracer.rays_to_device(rays)
    for _ in range(2):  # the first rebuild allocates, the second reuses
        scene.rebuild(torch.from_numpy(moved).cuda())
        for hitter in (tracer.BVH, tracer.BVH2, tracer.BRUTE):
            hit, t = tracer.next_hit(scene, hitter, d, with_t=True)
            assert np.array_equal(hit.cpu().numpy(), o_hit), hitter
            assert np.array_equal(t.cpu().numpy().view(np.uint32), o_t.view(np.uint32)), hitter
    assert scene.errors() == 0


@pytest.mark.parametrize("n", [262144, 262145, 300000])
def test_large_rebuild(n):
    """Either side of 256 sort tiles: the rebuilt tree against brute force."""
    import torch

    from splat_gb300 import tracer

    tris = _tris(n, 6)
    scene = tracer.Scene(tris, n + 2, bvh=False)
    scene.rebuild()
    d = tracer.rays_to_device(random_rays(20000, 9, n + 1))
    ref = tracer.next_hit(scene, tracer.BRUTE, d)
    assert int((ref != 1).sum()) > 5000
    assert torch.equal(tracer.next_hit(scene, tracer.BVH, d), ref)
    assert torch.equal(tracer.next_hit(scene, tracer.BVH2, d), ref)
    assert scene.errors() == 0
