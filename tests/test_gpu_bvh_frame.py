"""The BVH's own frame (boxes axis-aligned in a rotated frame when the
scene's facets lie along it): hits equal brute force bit for bit whatever
the scene's rotation, also after a refit, and after a rebuild returns the
tree to the world frame."""
import numpy as np
import pytest

from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu


def _rays(R, n=4096, seed=5):
    """Scattered rays, and rays along and inside the facets' own directions
    (grazing and axis-parallel ones, where a box test rounds worst)."""
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, T.ADRAY)
    pos = rng.uniform(-2.5, 2.5, (n, 3))
    d = rng.normal(size=(n, 3))
    d[: n // 4] = (R @ np.eye(3)[rng.integers(0, 3, n // 4)].T).T * rng.choice([-1.0, 1.0], (n // 4, 1))
    d[n // 4: n // 2] = np.eye(3)[rng.integers(0, 3, n // 4)] * rng.choice([-1.0, 1.0], (n // 4, 1))
    k = rng.integers(0, 10, (n // 8, 3)) * (2.0 / 9.0) - 1.0  # on the cells' planes
    pos[: n // 8] = (R @ k.T).T
    d[n // 2] = 0.0
    d[n // 2 + 1] = np.nan
    d[n // 2 + 2] = (np.inf, 0.0, 1.0)
    d[n // 2 + 3] *= 1e-18
    d[n // 2 + 4] *= 1e18
    pos[n // 2 + 5] *= 1e3
    rays["pos"] = pos
    rays["dir"] = d
    rays["ignore_tri"] = 1
    rays["ignore_tri"][::7] = rng.integers(2, 4000, len(rays[::7]))
    rays["status"] = T.STATUS_ACTIVE
    return rays


@pytest.mark.parametrize("turn", ["none", "degree", "any", "other"])
def test_hits_equal_brute_force_in_any_frame(turn):
    import torch

    from splat_gb300 import _lib as L
    from splat_gb300 import tracer

    if turn == "none":
        R = np.eye(3)
    elif turn == "degree":
        c, s = np.cos(np.radians(3.0)), np.sin(np.radians(3.0))
        R = np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]])
    else:
        R = S.random_quaternion_matrix(11 if turn == "any" else 23)
    glass = S.rotate(S.menger_tris(2, 2.0, None), R)
    tris, fd = S.assemble(glass, S.box_tris(3.0))
    d_rays = tracer.rays_to_device(_rays(R))
    scene = tracer.Scene(tris, fd)

    def check(what):
        ref, tref = tracer.next_hit(scene, tracer.BRUTE, d_rays, with_t=True)
        assert int((ref != 1).sum()) > 1000
        lib = L.load()
        old = lib.splat_get_tuning(L.TUNE_BVH_PACKET)
        try:
            for hitter, packet in ((tracer.BVH2, 0), (tracer.BVH, 0), (tracer.BVH, 2)):
                L.check(lib.splat_set_tuning(L.TUNE_BVH_PACKET, packet))
                hit, t = tracer.next_hit(scene, hitter, d_rays, with_t=True)
                assert torch.equal(hit, ref), (what, hitter, packet)
                assert torch.equal(t.view(torch.int32), tref.view(torch.int32)), (what, hitter, packet)
                # enough rays for one lane a ray
                hit = tracer.next_hit(scene, hitter, d_rays.repeat(5))
                assert torch.equal(hit, ref.repeat(5)), (what, hitter, packet, "many")
        finally:
            L.check(lib.splat_set_tuning(L.TUNE_BVH_PACKET, old))

    check("built")
    moved = tris.copy()
    rng = np.random.default_rng(3)
    moved[1:, 1:4] += rng.normal(scale=0.02, size=moved[1:, 1:4].shape).astype(np.float32)
    a, b, c = moved[1:, 1], moved[1:, 2], moved[1:, 3]
    moved[1:, 0] = np.cross(a - b, b - c)
    d_moved = torch.from_numpy(moved).cuda()
    scene.update(d_moved)
    check("refit")
    scene.rebuild(d_moved)
    check("rebuilt")
    assert scene.errors() == 0
