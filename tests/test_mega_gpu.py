"""The megakernel without record mode (k_mega): its films against the wavefront's, whose samples it
draws bit for bit, at films that leave partial tiles, blocks of one to four tiles and sample
slices that do not divide the samples, for each kernel variant (matte, every lobe, general
traversal)."""
import numpy as np
import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,option", [("box", None), ("materials", None), ("materials", ("bvh_width", 2)),
                                          ("materials", ("watertight", 1)), ("inst", None)])
@pytest.mark.parametrize("w,h,spp,bounces,crop", [(2, 2, 1, 1, None), (17, 9, 3, 5, None), (61, 48, 2, 5, None),
                                                  (100, 75, 5, 4, (3, 2, 90, 70)), (160, 131, 17, 6, None)])
def test_film_equals_the_wavefronts(tmp_path, scene, option, w, h, spp, bounces, crop):
    d = str(tmp_path)
    sc, sub = {"box": lambda: scenes.write_box_sphere(d, level=2), "materials": lambda: scenes.write_materials_scene(d, level=2),
               "inst": lambda: scenes.write_stress_scene(d, rings=8, segs=16, instanced=True)}[scene]()
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, d, sc, sub, w, h)
    if option:
        ctx.set_option(*option)
    a, b = (lts.PathTracingIntegrator(bounces, 3, s, integrator=k).render(spp, 7, crop=crop, sums=True)
            for k in (lts.INTEGRATOR_MEGAKERNEL, lts.INTEGRATOR_WAVEFRONT))
    # the same sample values in sums of another order: FP32 compensated per slice, then FP64; 4e-7
    # relative to the sum of the terms' magnitudes covers both.  (Terms can be negative -- the
    # reference's dielectric Fresnel exceeds 1 -- so that is the sum of |L| over the pixels whose
    # samples reach a film pixel, filter weights below 1, not the sum itself.)
    r = lts.PathTracingIntegrator(bounces, 3, s, integrator=lts.INTEGRATOR_MEGAKERNEL).render(spp, 7, crop=crop, record=True,
                                                                                          film=False)
    x0, y0, x1, y1 = crop or (0, 0, w, h)
    mag = np.zeros((h + 2, w + 2, 4))
    per = np.abs(r["L"]).astype(np.float64).sum(axis=2)
    for dy in range(3):
        for dx in range(3):
            mag[y0 + dy:y1 + dy, x0 + dx:x1 + dx, :3] += per
            mag[y0 + dy:y1 + dy, x0 + dx:x1 + dx, 3] += spp
    mag = mag[:h, :w]
    fa, fb = a["film_sums"], b["film_sums"]
    assert np.all(np.abs(fa - fb) <= 4e-7 * mag + 1e-12)
    assert a["rays"] == b["rays"]
    ctx.close()


def test_no_bounces(tmp_path):
    sc, sub = scenes.write_box_sphere(str(tmp_path), level=2)
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 20, 12)
    r = lts.PathTracingIntegrator(0, 3, s).render(2, 1, sums=True)
    assert np.all(r["film"] == 0) and r["rays"] == 0 and r["film_sums"][5, 5, 3] > 0
    ctx.close()
