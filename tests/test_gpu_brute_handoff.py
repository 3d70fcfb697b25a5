"""Brute force in a trace step hands its hits to the bounce kernel as packed
words and resets them for the next bounce: maps and statistics equal the CPU
restatement's with one and with several splits of the records, at block
edges, with ray ranges, several bounces and a splat beside them."""
import pytest

from splat_gb300 import scenes as S
from splat_gb300 import types as T
from test_gpu_small_step import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("depth", [1, 2, 5])
@pytest.mark.parametrize("begin,end", [(0, 12289), (7, 7 + 12800), (3, 12300)])
def test_handoff(order, depth, begin, end):
    tris, fd = S.assemble(S.sphere_tris(order), S.box_tris(3.0))
    light = T.rect_light((0.0, 2.6, 0.0), (0.0, -1.0, 0.0), (1.3, 0.0, 0.0), (0.0, 0.0, 1.3), 131, 103)
    wl = S.Workload(name="handoff", tris=tris, first_diffuse=fd, light=light, upscale=1,
                    lambda_mode=(T.LAMBDA_STRATIFIED, 3, 400.0, 700.0), spectrum=S.stratified_spectrum(3), depth=depth,
                    material=S.CAUCHY_GLASS, map_w=48, map_h=20, accum="i32", hitter="brute", seed=order + depth)
    _check(wl, begin, end)


def test_no_triangles():
    import numpy as np

    from splat_gb300 import tracer

    light = S.hemisphere_light(1, 120, 1.05)
    wl = S.Workload(name="empty", tris=np.zeros((1, 10, 3), np.float32), first_diffuse=2, light=light, depth=3,
                    map_w=16, map_h=16, accum="i32", lambda_mode=(T.LAMBDA_UNIFORM, 1, 400.0, 700.0),
                    spectrum=S.stratified_spectrum(2), hitter="brute")
    res = tracer.trace_forward(wl)
    assert not res.tex.any() and res.stats["rays_per_bounce"] == [14400, 0, 0] and res.stats["error"] == 0
