"""Single strategies of the bidirectional integrator, unweighted: each that can make the paths of one bounce
estimates the path tracer's direct light, the one that draws its own light point (s = 1) among them."""
import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_single_strategies_of_one_bounce(built_lib, tmp_path):
    """96 x 96, 256 spp.  The light seen directly (s = 0, t = 2) repeats whatever the path length; direct light by
    a sampled light point (1, 2), by light paths that reach the camera (2, 1) and by paths that hit the light
    (0, 3) is the path tracer's of one bounce less the light itself.  Image means: 2 % for the first two, as the
    image means of the whole estimator at twice the samples agree to 1 %; 5 % for hits on the light, whose
    variance is the inverse of its share of the hemisphere."""
    sc, sub = scenes.write_tri_light_box(str(tmp_path), level=2)
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 96, 96)

    def mean(strategy, bounces=4):
        ctx.set_option("bdpt_strategy", strategy)
        f = lts.PathTracingIntegrator(bounces, 1000, s, integrator=lts.INTEGRATOR_BDPT).render(256, 11)["film"]
        ctx.set_option("bdpt_strategy", 10000)
        return float(f.mean())

    seen = mean(2)
    assert seen > 0 and abs(mean(2, 8) - seen) <= 1e-6 * seen
    direct = float(lts.PathTracingIntegrator(1, 1000, s, integrator=lts.INTEGRATOR_WAVEFRONT).render(1024, 5)["film"].mean()) - seen
    got = {k: mean(k) for k in (102, 201, 3)}
    print(f"light {seen:.5f}, direct {direct:.5f}, strategies {got}")
    assert abs(got[102] - direct) <= 0.02 * direct
    assert abs(got[201] - direct) <= 0.02 * direct
    assert abs(got[3] - direct) <= 0.05 * direct
    ctx.close()
