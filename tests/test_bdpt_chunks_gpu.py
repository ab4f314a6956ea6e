"""The bidirectional integrator's chunks and strategies: the strategies rendered one at a time add
up, unweighted, to what each would give on any chunk split, and a film does not depend on how its
samples fall into chunks, blocks and partial tiles."""
import numpy as np
import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


def film(scene, spp, bounces, crop=None, strategy=10000, accumulate=False):
    ctx = scene.ctx
    ctx.set_option("bdpt_strategy", strategy)
    ctx.set_option("film_accumulate", 1 if accumulate else 0)
    r = lts.PathTracingIntegrator(bounces, 1000, scene, integrator=lts.INTEGRATOR_BDPT).render(spp, 3, crop=crop, sums=True)
    ctx.set_option("film_accumulate", 0)
    ctx.set_option("bdpt_strategy", 10000)
    return r


# one chunk is 2^18 samples: below a warp, ragged, exactly one chunk, one chunk and a sample row more
@pytest.mark.parametrize("matte", [True, False])
@pytest.mark.parametrize("w,h,spp,bounces", [(3, 2, 1, 0), (33, 17, 3, 8), (64, 64, 64, 2), (64, 65, 64, 2)])
def test_crops_partition_the_film(tmp_path, matte, w, h, spp, bounces):
    """The film of the whole image equals the accumulated films of its two halves (other chunks, other lanes; the
    samples are keyed by pixel): camera contributions and splats, up to FP64 summation order."""
    d = str(tmp_path)
    sc, sub = scenes.write_tri_light_box(d, level=2) if matte else scenes.write_point_lights(d, level=2)
    if not matte:  # a glossy and a mirror surface; the infinite light is refused
        text = (tmp_path / (sc + ".scene")).read_text().replace("1\t0.1 0.1 0.1\n", "0\n")
        (tmp_path / (sc + ".scene")).write_text(text)
        (tmp_path / (sub + ".subject")).write_text("0\n1\tsphere\n1\nC\tc\t3.9 2.4 1.8\tc\t0.2 0.4 1.4\t0.2\n")
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, d, sc, sub, w, h)
    whole = film(s, spp, bounces)["film_sums"]
    m = max(1, w // 2)
    film(s, spp, bounces, crop=(0, 0, m, h))
    parts = film(s, spp, bounces, crop=(m, 0, w, h), accumulate=True)["film_sums"]
    # identical products (radiance x filter weight, float) summed in FP64 in another order
    assert np.all(np.abs(whole - parts) <= 1e-12 * np.maximum(1.0, np.abs(whole).max()))
    assert np.isfinite(whole).all() and (bounces == 0 or whole[..., :3].sum() > 0)
    ctx.close()


def test_strategies_one_by_one(tmp_path):
    """Each strategy alone draws what it draws among the others, so strategies that sample no light point (s != 1)
    repeat exactly whatever the rest of the list is: s = 0 (hits on the light) over two path lengths."""
    sc, sub = scenes.write_tri_light_box(str(tmp_path), level=2)
    ctx = lts.Context(0)
    s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 40, 30)
    a = film(s, 8, 5, strategy=2)["film_sums"]   # s = 0, t = 2: the light seen directly
    b = film(s, 8, 1, strategy=2)["film_sums"]
    assert np.array_equal(a, b) and a[..., :3].max() > 0
    ctx.close()


@pytest.mark.parametrize("level,spp", [(0, 1), (2, 5)])
def test_shadow_rays_by_either_tree(tmp_path, level, spp):
    """The listed shadow rays through the 8-wide tree (fetched by persistent warps) and through the binary one (a
    stride loop) see the same, so the films are equal up to the splats' summation order."""
    sc, sub = scenes.write_tri_light_box(str(tmp_path), level=level)
    films = []
    for width in (8, 2):
        ctx = lts.Context(0)
        s = lts.Scene.parse(ctx, str(tmp_path), sc, sub, 37, 23)
        ctx.set_option("bvh_width", width)
        r = film(s, spp, 4)
        films.append((r["film_sums"], ctx.metrics().rays))
        ctx.close()
    (a, na), (b, nb) = films
    assert na == nb > 37 * 23 * spp and a[..., :3].max() > 0
    assert np.all(np.abs(a - b) <= 1e-12 * max(1.0, np.abs(a).max()))
