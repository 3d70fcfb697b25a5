"""The lines between one launch and separate launches for a brute-force step:
8,192 rays, or 12,288 for up to 128 records.  Maps and statistics equal the
CPU restatement's on both sides."""
import pytest

from splat_gb300 import scenes as S
from splat_gb300 import types as T
from test_gpu_small_step import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 8193, 12288, 12289])
@pytest.mark.parametrize("recs", [128, 129])
def test_at_the_lines(n, recs):
    tris, fd = S.assemble(S.sphere_tris(2)[: recs - 2], S.floor_tris(-1.5, 4.0))
    assert len(tris) - 1 == recs
    light = S.hemisphere_light(3, 128, 1.05)
    light["res2"] = 97
    _check(S.Workload(name="line", tris=tris, first_diffuse=fd, light=light, upscale=1,
                      lambda_mode=(T.LAMBDA_STRATIFIED, 2, 400.0, 700.0), spectrum=S.stratified_spectrum(2), depth=3,
                      material=S.CAUCHY_GLASS, map_w=32, map_h=32, accum="i32", hitter="brute", seed=4), 5, 5 + n)
