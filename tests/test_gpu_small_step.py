"""The trace step of few rays as one launch: maps and statistics equal the
CPU restatement's at group, block and range edges, for both hitters, every
material, footprint and accumulation, and at the line to the separate
launches."""
import numpy as np
import pytest

from helpers import small_scene
from oracle import oracle as O
from splat_gb300 import scenes as S
from splat_gb300 import types as T

pytestmark = pytest.mark.gpu

MATS = {"linear": (T.MATERIAL_LINEAR_REF, 0.0, 0.0), "cauchy": S.CAUCHY_GLASS,
        "sellmeier": (T.MATERIAL_SELLMEIER, 0.0, 0.0, (1.03961212, 0.231792344, 1.01046945),
                      (0.00600069867, 0.0200179144, 103.560653))}


def _check(wl, ray_begin=0, ray_end=0):
    from splat_gb300 import tracer

    scene = tracer.Scene(wl.tris, wl.first_diffuse, bvh=wl.hitter != "brute")
    res = tracer.trace_forward(wl, scene, ray_begin, ray_end)
    ref, st, _ = O.trace_forward(wl, ray_begin=ray_begin, ray_end=ray_end) if ray_end else O.trace_forward(wl)
    got, ref = res.tex.cpu().numpy().ravel(), ref.ravel(order="F")
    assert res.stats["error"] == 0
    assert res.stats["rays_per_bounce"] == [int(x) for x in st[: wl.depth]]
    if wl.accum == "i32":
        assert np.array_equal(got, ref)
    else:
        assert np.abs(got - ref).sum() <= 1e-5 * np.abs(ref).sum()
    assert ref.any()
    return res


@pytest.mark.parametrize("hitter", ["brute", "bvh"])
@pytest.mark.parametrize("mat", list(MATS))
@pytest.mark.parametrize("res,upscale,planes,accum", [((5, 3), 1, 1, "i32"), ((16, 16), 2, 9, "i32"),
                                                      ((33, 31), 1, 0, "f32"), ((70, 60), 3, 4, "i32")])
def test_small_steps(hitter, mat, res, upscale, planes, accum):
    tris, fd = small_scene(3, 0.05)
    light = S.hemisphere_light(3, res[0] * upscale, 1.05)
    light["res2"] = res[1] * upscale
    mode = (T.LAMBDA_STRATIFIED, planes, 400.0, 700.0) if planes else (T.LAMBDA_UNIFORM, 1, 400.0, 700.0)
    _check(S.Workload(name="small", tris=tris, first_diffuse=fd, light=light, upscale=upscale, lambda_mode=mode,
                      spectrum=S.stratified_spectrum(planes) if planes else None, depth=4, material=MATS[mat],
                      map_w=40, map_h=24, accum=accum, hitter=hitter, seed=9))


@pytest.mark.parametrize("n", [12287, 12288, 12289])
def test_at_the_line(n):
    tris, fd = S.assemble(S.menger_tris(1, 2.0, 5), S.box_tris(3.0))
    light = T.rect_light((0.0, 2.6, 0.0), (0.0, -1.0, 0.0), (1.3, 0.0, 0.0), (0.0, 0.0, 1.3), 128, 97)
    _check(S.Workload(name="line", tris=tris, first_diffuse=fd, light=light, upscale=1,
                      lambda_mode=(T.LAMBDA_STRATIFIED, 2, 400.0, 700.0), spectrum=S.stratified_spectrum(2), depth=3,
                      material=S.CAUCHY_GLASS, map_w=32, map_h=32, accum="i32", hitter="bvh", seed=4), 11, 11 + n)


def test_empty_scene_and_statistics_without_a_buffer():
    """A scene of the sentinel alone, and a step that wants no statistics."""
    import ctypes as C

    import torch

    from splat_gb300 import tracer

    tris, fd = small_scene(2)
    light = S.hemisphere_light(1, 24, 1.05)
    wl = S.Workload(name="empty", tris=tris, first_diffuse=fd, light=light, depth=2, map_w=16, map_h=16, accum="i32",
                    lambda_mode=(T.LAMBDA_UNIFORM, 1, 400.0, 700.0), spectrum=S.stratified_spectrum(2), hitter="bvh")
    step = tracer.TraceStep(wl)
    with_stats = step.run().clone()
    L = tracer.L
    L.check(L.load().splat_trace_forward(step.scene.handle, C.byref(step.params), step.tex.data_ptr(),
                                         step.ws.data_ptr(), step.ws.numel(), None, tracer._stream()))
    torch.cuda.synchronize()
    assert torch.equal(step.tex, with_stats) and bool(with_stats.any())
    none = wl.with_(tris=np.zeros((1, 10, 3), np.float32), first_diffuse=2)
    res = tracer.trace_forward(none)
    assert not res.tex.any() and res.stats["rays_per_bounce"] == [576, 0] and res.stats["error"] == 0
