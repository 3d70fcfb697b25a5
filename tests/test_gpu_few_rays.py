"""The four-wide BVH hitter's forms by ray count: a warp a ray, eight lanes a
ray, one lane a ray.  Hits equal brute force bit for bit at the edges between
them, on a soup of large overlapping triangles that fills the groups' stacks,
and with the count known on the device only."""
import numpy as np
import pytest

from helpers import assert_rays_equal, random_rays, small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    """n large triangles around the origin: every ray enters most boxes, and
    coincident copies tie on the distance."""
    rng = np.random.default_rng(seed)
    P = rng.uniform(-1.0, 1.0, (n, 3, 3))
    P[n // 2: n // 2 + n // 8] = P[: n // 8]
    e = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    N = np.repeat((e / np.linalg.norm(e, axis=1, keepdims=True))[:, None], 3, 1)
    return S.assemble(S.ftri_records(P, N, np.zeros_like(P)), S.floor_tris(-1.5, 4.0))


@pytest.mark.parametrize("n", [1, 9, 33, 4096, 4097, 16384, 16385, 40001])
@pytest.mark.parametrize("kind", ["sphere", "sponge", "soup"])
def test_hits_by_ray_count(n, kind):
    import torch

    from splat_gb300 import tracer

    if kind == "sphere":
        tris, fd = small_scene(4, 0.05)
    elif kind == "sponge":
        tris, fd = S.assemble(S.menger_tris(2, 2.0, 9), S.box_tris(3.0))
    else:
        tris, fd = _soup(3000, 5)
    scene = tracer.Scene(tris, fd)
    rays = random_rays(n, 3 + n, tris.shape[0])
    rays["dir"][::11] = np.eye(3, dtype=np.float32)[np.arange(len(rays[::11])) % 3]
    if n > 8:
        rays["dir"][3] = np.nan
        rays["dir"][4] = 0.0
        rays["pos"][5] = np.inf
    d = tracer.rays_to_device(rays)
    ref, tref = tracer.next_hit(scene, tracer.BRUTE, d, with_t=True)
    hit, t = tracer.next_hit(scene, tracer.BVH, d, with_t=True)
    assert torch.equal(hit, ref)
    assert torch.equal(t.view(torch.int32), tref.view(torch.int32))
    assert scene.errors() == 0


@pytest.mark.parametrize("active", [0, 1, 4096, 4097, 16384, 16385])
def test_hits_with_the_count_on_the_device(active):
    """More slots than active rays: the launch's bound is above every line,
    the count picks the form."""
    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    scene = tracer.Scene(tris, fd)
    n = 20000
    rays = random_rays(n, 77, tris.shape[0])
    rays["status"] = T.STATUS_INFINITY
    rays["status"][np.random.default_rng(2).permutation(n)[:active]] = T.STATUS_ACTIVE
    d = tracer.rays_to_device(rays)
    hit = tracer.run_evolution(tracer.BVH, scene, d, 2, S.CAUCHY_GLASS, None, seed=5)
    ref, _ = O.run_evolution(rays, tris, 2, fd, S.CAUCHY_GLASS, None, seed=5)
    ref_hit, _ = O.next_hit(ref, tris)
    assert_rays_equal(tracer.rays_to_host(d), ref, "device count")
    assert np.array_equal(hit.cpu().numpy(), ref_hit)
    assert scene.errors() == 0
