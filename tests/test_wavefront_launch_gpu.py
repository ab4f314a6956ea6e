"""The wavefront's launch structure: kept iteration graphs, list kernels that stride over lists
longer or shorter than their grids, and small ray lists spread over every warp of the trace grid.
Wavefront samples are the megakernel's bit for bit, so the recorded samples are compared exactly."""
import numpy as np
import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


def samples(scene, integrator, spp, seed, bounces, crop=None):
    r = lts.PathTracingIntegrator(bounces, 3, scene, integrator=integrator).render(spp, seed, crop=crop, record=True,
                                                                                  film=False)
    return r["L"], r["sig"]


# one path; fewer than a warp; around a classify tile (1,024 paths); around one list grid
# (152 SMs x 32 blocks x 128 threads = 622,592 paths), which the list kernels stride over
@pytest.mark.parametrize("w,h,spp", [(2, 2, 1), (5, 3, 1), (31, 33, 1), (32, 32, 1), (41, 25, 1), (64, 38, 256),
                                     (311, 143, 14), (320, 304, 7)])
def test_list_sizes(tmp_path, w, h, spp):
    sc, sub = scenes.write_materials_scene(str(tmp_path), level=2)
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, w, h)
    La, sa = samples(s, lts.INTEGRATOR_WAVEFRONT, spp, 5, 4)
    Lb, sb = samples(s, lts.INTEGRATOR_MEGAKERNEL, spp, 5, 4)
    assert np.array_equal(sa, sb) and np.array_equal(La, Lb)
    ctx.close()


def test_kept_graphs_follow_the_render(tmp_path):
    """One context, renders that change the seed, bounces, crop, pool, film size and scene: each film equals a
    fresh context's, whatever iteration graph the context kept from the render before."""
    files = {"m": scenes.write_materials_scene(str(tmp_path / "m"), level=2),
             "b": scenes.write_box_sphere(str(tmp_path / "b"), level=2)}
    steps = [("m", 48, 40, 4, 1, 5, 0), ("m", 48, 40, 4, 2, 5, 0), ("m", 48, 40, 4, 2, 9, 0), ("m", 48, 40, 2, 2, 9, 700),
             ("b", 48, 40, 4, 1, 5, 0), ("b", 33, 57, 4, 1, 5, 0), ("m", 33, 57, 4, 1, 20, 0), ("m", 48, 40, 4, 1, 5, 0)]

    def film(ctx, step):
        f, w, h, spp, seed, bounces, pool = step
        s = lts.Scene.parse(ctx, str(tmp_path / f), *files[f], w, h)
        ctx.set_option("wavefront_pool", pool)
        out = [lts.PathTracingIntegrator(bounces, 3, s, integrator=lts.INTEGRATOR_WAVEFRONT).render(spp, seed)["film"]
               for _ in range(2)]
        assert np.array_equal(out[0], out[1])
        return out[0]

    one = lts.Context(0)
    for step in steps:
        fresh = lts.Context(0)
        assert np.array_equal(film(one, step), film(fresh, step))
        fresh.close()
    one.close()
