"""Counting the traversal's work (SPLAT_TUNE_COUNT_WORK) leaves every result
as it is where few rays are left: bounces below the lines at which the plain
forms hand over to groups of lanes (4,096 and 16,384 rays), the final hit of
the records' bounce loop, and a small camera pass."""
import ctypes as C

import numpy as np
import pytest

from helpers import assert_rays_equal, random_rays, small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu


class _Counting:
    """The knob on, the counters cleared; work() reads them."""

    def __enter__(self):
        import torch

        from splat_gb300 import _lib as L

        self.L, self.lib = L, L.load()
        self.stream = torch.cuda.current_stream().cuda_stream
        self.work()
        self.old = self.lib.splat_get_tuning(L.TUNE_COUNT_WORK)
        L.check(self.lib.splat_set_tuning(L.TUNE_COUNT_WORK, 1))
        return self

    def __exit__(self, *exc):
        self.L.check(self.lib.splat_set_tuning(self.L.TUNE_COUNT_WORK, self.old))

    def work(self):
        """(nodes, pre-tests, full tests, rays) since the last read."""
        out = (C.c_int64 * 4)()
        self.L.check(self.lib.splat_hit_work(out, 1, self.stream))
        return [int(v) for v in out]


@pytest.mark.parametrize("res", [(60, 50), (128, 120), (160, 130)])
def test_steps(res):
    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    light = S.hemisphere_light(3, res[0], 1.05)
    light["res2"] = res[1]
    wl = S.Workload(name="count", tris=tris, first_diffuse=fd, light=light, upscale=1,
                    lambda_mode=(T.LAMBDA_STRATIFIED, 2, 400.0, 700.0), spectrum=S.stratified_spectrum(2), depth=4,
                    material=S.CAUCHY_GLASS, map_w=40, map_h=24, accum="i32", hitter="bvh", seed=9)
    scene = tracer.Scene(tris, fd)
    ref, st, _ = O.trace_forward(wl)
    bounces = [int(x) for x in st[: wl.depth]]
    assert min(bounces) < 4096
    with _Counting() as c:
        res = tracer.trace_forward(wl, scene)
        nodes, pre, full, rays = c.work()
    assert np.array_equal(res.tex.cpu().numpy().ravel(), ref.ravel(order="F")) and ref.any()
    assert res.stats["rays_per_bounce"] == bounces and res.stats["error"] == 0
    assert rays == sum(bounces) and nodes > rays and pre >= full > 0


@pytest.mark.parametrize("n", [700, 9000, 20000])
def test_run_evolution(n):
    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.05)
    scene = tracer.Scene(tris, fd)
    rays = random_rays(n, 41, tris.shape[0])
    rays["status"][::5] = T.STATUS_INFINITY
    ref, _ = O.run_evolution(rays, tris, 3, fd, S.CAUCHY_GLASS, None, seed=5)
    ref_hit, _ = O.next_hit(ref, tris)
    d = tracer.rays_to_device(rays)
    with _Counting():
        hit = tracer.run_evolution(tracer.BVH, scene, d, 3, S.CAUCHY_GLASS, None, seed=5)
    assert_rays_equal(tracer.rays_to_host(d), ref, "counted")
    assert np.array_equal(hit.cpu().numpy(), ref_hit)
    assert scene.errors() == 0


def test_camera_pass():
    import torch

    from splat_gb300 import tracer

    tris, fd = small_scene(3, 0.04)
    scene = tracer.Scene(tris, fd)
    cam = S.realtime_camera()
    cam = tracer.camera_look_at(cam["pos"], cam["look_at"], cam["up"], cam["fov"])
    shader = tracer.Shader(32, 32, 4)
    shader.set_light_map(torch.rand((4, 32, 32), device="cuda", generator=torch.Generator("cuda").manual_seed(3)))
    P = tracer.render_params(cam, 96, 128, 1, 4, S.CAUCHY_GLASS, S.stratified_spectrum(4), seed=7)
    ref = tracer.CameraPass(scene, shader, P).run().clone()
    with _Counting():
        got = tracer.CameraPass(scene, shader, P).run()
        torch.cuda.synchronize()
    assert torch.equal(got, ref) and bool(ref.any())
    assert scene.errors() == 0
