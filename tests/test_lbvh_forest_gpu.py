"""The LBVH build's one-block sort, sort tiles and group merging at the sizes where they change, and
trees whose forests are as long as they can be (all codes equal: ranges by position alone)."""
import numpy as np
import pytest

from oracle import lbvh_np

pytestmark = pytest.mark.gpu


def check(lts, ctx, tris, mode, code_limit):
    out = lts.build_bvh_triangles(ctx, tris, mode, code_limit)
    codes, ids = lbvh_np.stable_sort(*lbvh_np.morton_codes(tris, code_limit))
    n = len(tris)
    assert np.array_equal(out["sorted_codes"], codes) and np.array_equal(out["sorted_ids"], ids)
    left, right = lbvh_np.karras_topology(codes)
    assert np.array_equal(out["node_left"][: n - 1], left) and np.array_equal(out["node_right"][: n - 1], right)
    assert np.all(out["node_left"][n - 1:] == -1) and np.all(out["node_right"][n - 1:] == -1)
    assert np.array_equal(out["node_key"], np.concatenate([np.full(n - 1, -1), np.arange(n)]).astype(np.int32))
    mn, mx = lbvh_np.tri_bounds(tris)
    leaf = np.concatenate([mn, mx], 1)
    lbvh_np.check_tree(out["node_left"], out["node_right"], out["node_bounds"],
                       leaf if mode == lts.BVH_REFERENCE else leaf[ids])


# the one-block sort ends at 4,096; tree blocks of 512 in groups of 24 (12,288 leaves): one block,
# one short group, a group and one leaf, two levels of groups (294,912 leaves and one); small sort
# tiles of 2,048 keys end at 500,000
@pytest.mark.parametrize("n", [2, 33, 4095, 4096, 4097, 12287, 12288, 12289, 294913, 500000, 500001])
@pytest.mark.parametrize("mode,part", [(1, 0.0), (0, 0.6)])
def test_sizes(built_lib, n, mode, part):
    import lighttransportsimulation_gb300 as lts
    from lighttransportsimulation_gb300 import scenes
    ctx = lts.Context(0)
    check(lts, ctx, scenes.random_triangles(n, seed=n), mode, int(n * part) if part else -1)
    ctx.close()


@pytest.mark.parametrize("n", [1000, 4096, 30011])
@pytest.mark.parametrize("kind", ["equal", "line", "clusters"])
def test_degenerate_codes(built_lib, n, kind):
    """Equal triangles (every delta from the positions), a line (deep, one-sided codes), and a few
    clusters of equal triangles; the context is used again for a smaller build in between."""
    import lighttransportsimulation_gb300 as lts
    rng = np.random.default_rng(n)
    base = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32) * np.float32(1e-3)
    if kind == "equal":
        at = np.zeros((n, 3), np.float32)
    elif kind == "line":
        at = np.zeros((n, 3), np.float32)
        at[:, 0] = np.float32(0.5) ** (np.arange(n) % 24).astype(np.float32)
    else:
        at = rng.random((7, 3)).astype(np.float32)[rng.integers(0, 7, n)]
    tris = (base[None] + at[:, None]).astype(np.float32)
    ctx = lts.Context(0)
    check(lts, ctx, tris, 1, -1)
    check(lts, ctx, tris[: n // 3], 1, -1)
    check(lts, ctx, tris, 0, n // 2)
    ctx.close()
