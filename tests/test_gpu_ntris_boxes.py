"""The n_tris hitter's boxes where a record's own numbers do not bound what it
accepts: a needle whose plane contains its short edge's direction, and rays
with directions near the smallest number.  Hits equal the oracle's plain
search."""
import numpy as np
import pytest

from helpers import random_rays
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _both(rays, tris):
    from splat_gb300 import tracer

    o_hit, o_t = O.next_hit(rays, tris)
    hit, tmp = tracer.next_hit_brute(tracer.rays_to_device(rays), tracer.n_tris_array(tris))
    assert np.array_equal(hit.cpu().numpy(), o_hit)
    dec = np.array([O.monotonic_f32(int(k >> np.uint64(32))) for k in tmp.cpu().numpy().view(np.uint64)], np.float32)
    assert np.array_equal(dec.view(np.uint32), o_t.view(np.uint32))
    return o_hit


@pytest.mark.parametrize("short", [2.0 ** -16, 2.0 ** -13, 2.0 ** -12, 2.0 ** -10])
@pytest.mark.parametrize("swap", [False, True])
def test_needles(short, swap):
    """The corner at a is square, one leg is short, and the record's normal
    lies along it: accepted points are anywhere above the needle.  All numbers
    are exact, so the points' barycentrics are (0.5, 0)."""
    rng = np.random.default_rng(5)
    n = 40
    axes = np.eye(3)[np.array([rng.permutation(3) for _ in range(n)])]  # along the needle, its short leg, above
    a = rng.integers(-512, 513, (n, 3)) / 1024.0
    long_end, short_end = a + axes[:, 0], a + short * axes[:, 1]
    tris = np.zeros((n + 1, 10, 3), np.float32)
    tris[1:, 1] = a
    tris[1:, 2], tris[1:, 3] = (long_end, short_end) if swap else (short_end, long_end)
    tris[1:, 0] = axes[:, 1]
    rays = random_rays(n * 16, 3, n + 1)
    k = np.arange(len(rays)) % n
    rays["pos"] = (a[k] + 0.5 * axes[k, 0] + rng.integers(300, 3000, (len(k), 1)) / 1024.0 * axes[k, 2]
                   + axes[k, 1])
    rays["dir"] = -axes[k, 1]
    rays["ignore_tri"] = 1
    hit = _both(rays, tris)
    assert int((hit != 1).sum()) > len(rays) // 2


@pytest.mark.parametrize("scale", [1e-19, 1e-24, 1e-29, 1e-33])
def test_short_directions(scale):
    from splat_gb300 import scenes as S

    g = S.sphere_tris(2, noise_amp=0.05, noise_seed=3)
    tris = np.concatenate([np.zeros((1, 10, 3), np.float32), g.astype(np.float32)], 0)
    rays = random_rays(1500, 8, tris.shape[0])
    rays["dir"][::2] *= np.float32(scale)
    hit = _both(rays, tris)
    assert int((hit != 1).sum()) > 300
