"""Ray queries from separate arrays (Scene.intersect / simple_intersect, lts_intersect_arrays) against
the interleaved entry point and the binary tree, over batch sizes, strides, dtypes and tmax forms."""
import ctypes

import numpy as np
import pytest

import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("rays"))
    sc, sub = scenes.write_displaced(d, level=4)
    ctx = lts.Context(0)
    yield lts.Scene.parse(ctx, d, sc, sub, 64, 64)
    ctx.close()


def rays(n, seed):
    r = np.random.default_rng(seed)
    o = r.uniform(-0.95, 0.95, (n, 3)).astype(np.float32)
    d = (r.normal(0, 0.3, (n, 3)) - o).astype(np.float32)
    d[::7] = np.float32([0, 0, -1])  # axis-parallel: the slab form of the box test
    return o, d


def interleaved(scene, o, d, tmax, any_hit):
    n = len(o)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7] = o, tmax, d
    prim, t = np.empty(n, np.int32), np.empty(n, np.float32)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    scene.ctx.check(scene.ctx.lib.lts_intersect(scene.ctx.h, p(r), n, any_hit, p(prim), p(t)))
    return prim, t


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 5000])
def test_forms_agree(scene, n):
    o, d = rays(n, n)
    tmax = np.random.default_rng(n + 1).uniform(0.1, 2.0, n).astype(np.float32)
    for tm in (np.inf, 0.7, np.float32(0.7), np.full(1, 0.7), tmax):
        a, b = interleaved(scene, o, d, tm, 0), scene.intersect(o, d, tm)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        assert np.array_equal(interleaved(scene, o, d, tm, 1)[0] == 1, scene.simple_intersect(o, d, tm))
    # other dtypes and strides, one direction for all
    a = scene.intersect(o, d)
    b = scene.intersect(np.asfortranarray(o.astype(np.float64)), np.repeat(d, 2, axis=0)[::2])
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    a, b = scene.intersect(o, np.broadcast_to(d[:1], (n, 3))), scene.intersect(o, d[:1])
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    # the binary tree: the same hits by another traversal
    a = scene.intersect(o, d)
    scene.ctx.set_option("bvh_width", 2)
    b = scene.intersect(o, d)
    scene.ctx.set_option("bvh_width", 8)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_refused_and_empty(scene):
    o, d = rays(4, 0)
    with pytest.raises(ValueError):
        scene.intersect(o, d[:3])
    with pytest.raises(ValueError):
        scene.intersect(o, d, np.ones(3))
    with pytest.raises(ValueError):
        scene.intersect(o, d, np.ones((1, 1)))
    prim, t = scene.intersect(np.zeros((0, 3)), np.zeros((0, 3)))
    assert prim.shape == (0,) and t.shape == (0,)
    lib, h = scene.ctx.lib, scene.ctx.h
    assert lib.lts_intersect_arrays(h, None, None, None, 1, 1, 0, None, None) == 1
    p = ctypes.c_void_p(o.ctypes.data)
    assert lib.lts_intersect_arrays(h, p, p, p, 2, 4, 0, p, None) == 1
