"""First-bounce packets or one lane a ray, by rays per triangle: the drop-in
bounce loop and the fused camera pass give brute force's records and images on
both sides of their lines (5,132 records: 30,792 and 16,422.4 rays)."""
import numpy as np
import pytest

from helpers import assert_rays_equal
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    from splat_gb300 import tracer

    tris, fd = S.assemble(S.sphere_tris(4), S.box_tris(3.0))
    assert len(tris) == 5133
    return tracer.Scene(tris, fd)


@pytest.mark.parametrize("n", [30791, 30792, 30793])
def test_run_evolution(scene, n):
    from splat_gb300 import tracer

    light = T.rect_light((0.0, 2.6, 0.0), (0.0, -1.0, 0.0), (1.3, 0.0, 0.0), (0.0, 0.0, 1.3), n, 1)
    out = []
    for hitter in (tracer.BRUTE, tracer.BVH):
        rays = tracer.rays_from_light(light, 1, (T.LAMBDA_UNIFORM, 1, 400.0, 700.0), 3)
        hit = tracer.run_evolution(hitter, scene, rays, 3, S.CAUCHY_GLASS, seed=3)
        out.append((tracer.rays_to_host(rays), hit.cpu().numpy()))
    assert_rays_equal(out[1][0], out[0][0], f"{n} rays")
    assert np.array_equal(out[1][1], out[0][1])


@pytest.mark.parametrize("h,w", [(113, 145), (37, 443), (37, 444), (111, 148)])
def test_camera_pass(scene, h, w):
    import torch

    from splat_gb300 import tracer

    cam = S.realtime_camera()
    view = tracer.camera_look_at(cam["pos"], cam["look_at"], cam["up"], cam["fov"])
    spec = S.stratified_spectrum(2)
    shader = tracer.Shader(16, 16, 2)
    shader.set_light_map(torch.rand((2, 16, 16), device="cuda", generator=torch.Generator("cuda").manual_seed(1)))
    images = []
    for hitter in ("brute", "bvh"):
        P = tracer.render_params(view, h, w, 1, 3, S.CAUCHY_GLASS, spec, hitter, 5)
        images.append(tracer.image(tracer.CameraPass(scene, shader, P).run()))
    assert images[0].max() > 0 and np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
