"""Camera rays of grids with few rows, whose tiles have 8 rows or one instead
of 32: at the lines (4 and 16 rows) and around a tile's columns, records equal
the CPU restatement's, and the fused pass gives the records' image."""
import numpy as np
import pytest

from helpers import assert_rays_equal, small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1, 3, 4, 5, 8, 9, 16, 17, 24])
@pytest.mark.parametrize("w", [1, 63, 65, 513])
def test_camera_rays(h, w):
    import torch

    from splat_gb300 import tracer

    c = S.realtime_camera()
    args = (c["pos"], c["look_at"], c["up"], c["fov"])
    cam, ocam = tracer.camera_look_at(*args), O.camera_look_at(*args)
    rays = tracer.camera_rays(cam, h, w, 550.0, 7)
    assert_rays_equal(tracer.rays_to_host(rays), O.camera_rays(ocam, h, w, 550.0, 7), f"camera rays {h} x {w}")
    tris, fd = small_scene(2)
    scene = tracer.Scene(tris, fd)
    spec = S.stratified_spectrum(2)
    shader = tracer.Shader(16, 16, 2)
    shader.set_light_map(torch.rand((2, 16, 16), device="cuda", generator=torch.Generator("cuda").manual_seed(3)))
    P = tracer.render_params(cam, h, w, 1, 2, S.CAUCHY_GLASS, spec, "bvh", 7)
    fused = tracer.image(tracer.CameraPass(scene, shader, P).run())
    hit = tracer.run_evolution(tracer.BVH, scene, rays, 2, S.CAUCHY_GLASS, seed=7)
    plain = tracer.image(tracer.continuum_shade(scene, shader, rays, hit, spec, tracer.retina_factors(spec), 1, h, w))
    assert np.array_equal(fused.view(np.uint32), plain.view(np.uint32))
