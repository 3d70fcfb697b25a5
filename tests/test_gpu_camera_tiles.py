"""The camera pass at the edges of its kernels' tiles: camera rays of grids
around a 32 x 16 tile equal the CPU restatement's; a light map's texels reach
the texture whatever its width and alignment; shading through records and
through the fused pass agree for every sub-sample count."""
import numpy as np
import pytest

from helpers import assert_rays_equal, small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _cameras():
    from splat_gb300 import tracer

    cam = S.realtime_camera()
    args = (cam["pos"], cam["look_at"], cam["up"], cam["fov"])
    return tracer.camera_look_at(*args), O.camera_look_at(*args)


@pytest.mark.parametrize("h,w", [(1, 1), (31, 15), (32, 16), (33, 17), (64, 1), (1, 33), (97, 50)])
def test_camera_rays(h, w):
    from splat_gb300 import tracer

    cam, ocam = _cameras()
    got = tracer.rays_to_host(tracer.camera_rays(cam, h, w, 480.0, 7))
    assert_rays_equal(got, O.camera_rays(ocam, h, w, 480.0, 7), f"camera rays {h} x {w}")


@pytest.mark.parametrize("w,h,planes,offset", [(64, 33, 3, 0), (64, 33, 3, 1), (66, 16, 2, 0), (61, 17, 5, 0),
                                               (4, 1, 1, 0), (1, 1, 1, 0), (130, 40, 1, 2)])
@pytest.mark.parametrize("upscale", [1, 2, 3])
def test_light_map_and_sub_samples(w, h, planes, offset, upscale):
    """An int32 map (starting offset words into its buffer) shades like the
    float map of its values, which the library copies into the texture; the
    records' form and the fused form give the same image."""
    import torch

    from splat_gb300 import tracer

    cam, _ = _cameras()
    tris, fd = small_scene(2)
    scene = tracer.Scene(tris, fd)
    rng = np.random.default_rng(w * h + planes)
    buf = torch.from_numpy(rng.integers(0, 1 << 20, offset + planes * h * w, dtype=np.int32)).cuda()
    fixed = buf[offset:].view(planes, h, w)
    spec = S.stratified_spectrum(planes)
    height, width, depth, seed = 21 * upscale, 35 * upscale, 3, 5
    P = tracer.render_params(cam, height, width, upscale, depth, S.CAUCHY_GLASS, spec, "bvh", seed)
    rays = tracer.camera_rays(cam, 21, 35, 550.0, seed)
    hit = tracer.run_evolution(tracer.BVH, scene, rays, depth, S.CAUCHY_GLASS, seed=seed)
    images = []
    for tex in (fixed, fixed.float() * 2.0 ** -16):
        shader = tracer.Shader(w, h, planes, 0, 0)
        shader.set_light_map(tex)
        images.append(tracer.image(tracer.CameraPass(scene, shader, P).run()))
        images.append(tracer.image(tracer.continuum_shade(scene, shader, rays.clone(), hit, spec,
                                                          tracer.retina_factors(spec), upscale, height, width)))
    for im in images[1:]:
        assert np.array_equal(im.view(np.uint32), images[0].view(np.uint32))
    assert images[0].max() > 0
