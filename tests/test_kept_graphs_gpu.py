"""Iteration graphs kept between renders that change what the wavefront runs: the radiance cache on and off and
with new weights, batched views, the two-level and the flat tree, and renders of a context after others.
Every film equals a fresh context's."""
import numpy as np
import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


def view(k):
    return dict(frm=(0.1 * k, 0.2, 0.8), at=(0, 0, -0.5), up=(0, 1, 0), vfov=60.0, focus=1.0, width=40 + 8 * k, height=33,
                spp=3, seed=k)


def step(ctx, files, s):
    """One film (or a list of views' films) of step s = (scene, option values, seed, weights' seed)."""
    scene, options, seed, weights = s
    sc = lts.Scene.parse(ctx, files[scene][0], *files[scene][1], 48, 36)
    if weights:
        net = lts.RadianceCacheMLP(ctx, seed=weights)  # inference only: the learning rate is 0
        ctx.set_option("radiance_cache_lr_micro", 0)
        assert net.params().any()
    for k, v in (("radiance_cache", 0), ("two_level_bvh", 1)) + options:
        if k != "views":
            ctx.set_option(k, v)
    if ("views", 1) in options:
        return np.concatenate([f.reshape(-1) for f in lts.render_views(sc, [view(1), view(2)], 4, 3)[0]])
    return lts.PathTracingIntegrator(4, 3, sc, integrator=lts.INTEGRATOR_WAVEFRONT).render(3, seed)["film"].reshape(-1)


def test_kept_graphs(built_lib, tmp_path):
    files = {}
    for name, write in (("m", lambda d: scenes.write_materials_scene(d, level=2)),
                        ("i", lambda d: scenes.write_stress_scene(d, rings=8, segs=16, instanced=True))):
        d = tmp_path / name
        d.mkdir()
        files[name] = (str(d), write(str(d)))
    cache = (("radiance_cache", 1),)
    steps = [("m", (), 1, 0), ("m", cache, 1, 5), ("m", cache, 2, 0), ("m", (), 2, 0), ("m", cache, 2, 6), ("m", (("views", 1),), 0, 0),
             ("m", (), 1, 0), ("i", (), 1, 0), ("i", (("two_level_bvh", 0),), 1, 0), ("i", cache, 1, 7), ("i", (), 3, 0),
             ("m", cache, 2, 6), ("i", (("views", 1),), 0, 0), ("m", (), 2, 0)]
    one = lts.Context(0)
    weights = 0
    for s in steps:
        weights = s[3] or weights
        fresh = lts.Context(0)
        want = step(fresh, files, s[:3] + (weights if ("radiance_cache", 1) in s[1] else 0,))
        got = step(one, files, s)
        assert np.array_equal(got, step(one, files, s[:3] + (0,)))
        assert np.array_equal(got, want) and np.isfinite(got).all() and got.any(), s
        fresh.close()
    one.close()
