"""Render metrics read without the film, and between renders of different integrators."""
import ctypes

import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_gather_time_belongs_to_its_render(tmp_path):
    """The film gather's time is in the metrics of an asynchronous render whose film nobody has fetched, and not
    in those of the render after it."""
    sc, sub = scenes.write_tri_light_box(str(tmp_path), level=2)
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 200, 120)
    wave = lts.PathTracingIntegrator(3, 3, s, integrator=lts.INTEGRATOR_WAVEFRONT)
    for other in (lts.INTEGRATOR_MEGAKERNEL, lts.INTEGRATOR_BDPT):
        d = wave.desc(4, 1)
        ctx.check(ctx.lib.lts_render_async(ctx.h, ctypes.byref(d)))
        first = ctx.metrics().render_stage_ms[5]
        assert 0 < first < 1000 and ctx.metrics().render_stage_ms[5] == first
        ctx.check(ctx.lib.lts_render_async(ctx.h, ctypes.byref(d)))
        lts.PathTracingIntegrator(3, 3, s, integrator=other).render(1, 1)
        assert list(ctx.metrics().render_stage_ms) == [0.0] * 6
    ctx.close()


@pytest.mark.parametrize("w,h,spp,chunks", [(40, 30, 1, 1), (256, 256, 5, 2)])
def test_bidirectional_launches(tmp_path, w, h, spp, chunks):
    """The bidirectional integrator launches five kernels per chunk of 2^18 samples."""
    sc, sub = scenes.write_tri_light_box(str(tmp_path), level=1)
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, w, h)
    lts.PathTracingIntegrator(3, 3, s, integrator=lts.INTEGRATOR_BDPT).render(spp, 1)
    assert ctx.metrics().render_launches == 5 * chunks
    lts.PathTracingIntegrator(3, 3, s, integrator=lts.INTEGRATOR_MEGAKERNEL).render(spp, 1)
    assert ctx.metrics().render_launches == 1
    ctx.close()
