"""Trees whose blocks leave long forests: at every edge between blocks of 512 leaves the codes close in on each
other, so that many subtrees of either block have their parents beyond it, and a group of 24 blocks
hands more subtrees to one block than it has threads (the merge then runs in chunks, and again over the chunks)."""
import numpy as np
import pytest

from oracle import lbvh_np

BLOCK, GROUP = 512, 24


def chain_codes(blocks):
    """Sorted codes of 512 leaves a block.  Around the edge before block b every code has b + 1 on top and the
    bits below alternate: clearing a set bit of that middle gives a neighbour to its left, setting a clear one to
    its right, the nearer the lower the bit.  What is left of a block repeats a code between two edges."""
    top = int(blocks + 1).bit_length()
    low = 30 - top
    middle = sum(1 << k for k in range(0, low, 2))
    codes = np.zeros((blocks, BLOCK), np.int64)

    def right_of(edge):  # decreasing deltas: the neighbours after the middle, nearest first
        base = edge << low
        keep = lambda k: (middle >> k) << k  # noqa: E731  the bits from k up
        return [base | middle] + [base | keep(k) | (1 << k) for k in range(1, low, 2)]

    def left_of(edge):
        base = edge << low
        return [base | (((middle >> (k + 1)) << (k + 1))) | ((1 << k) - 1 if k else 0) for k in range(low - 1 - (low - 1) % 2, -1, -2)]

    for b in range(blocks):
        head, tail = right_of(b), left_of(b + 1)
        fill = BLOCK - len(head) - len(tail)
        codes[b] = head + [head[-1]] * fill + tail
    codes = codes.reshape(-1)
    codes[0], codes[-1] = 0, (1 << 30) - 1  # the scene box's corners
    assert np.all(np.diff(codes) >= 0) and codes[-1] < 1 << 30
    return codes.astype(np.uint32)


def triangles(codes):
    """Point-sized triangles whose centroids quantise to the codes (exact in binary: (q + 1/2) / 1024)."""
    q = np.zeros((len(codes), 3), np.int64)
    for bit in range(10):
        for axis in range(3):
            q[:, axis] |= ((codes.astype(np.int64) >> (3 * bit + axis)) & 1) << bit
    p = ((q + 0.5) / 1024).astype(np.float32)
    p[0], p[-1] = 0.0, 1.0
    return np.repeat(p[:, None, :], 3, axis=1)


def deltas(codes):
    i = np.arange(len(codes) - 1)
    x = codes[:-1] ^ codes[1:]
    clz = lambda v: 31 - np.floor(np.log2(np.maximum(v, 1).astype(np.float64))).astype(np.int64)  # noqa: E731
    return np.where(x == 0, 40 + clz(i ^ (i + 1)), clz(x.astype(np.int64)))


def forest_sizes(codes):
    """Subtrees that every block leaves: its leaves less the nodes whose range lies inside it (a node split at
    boundary g reaches as far as the deltas around g are larger)."""
    d = np.concatenate([[-1], deltas(codes), [-1]])  # boundary i lies before leaf i
    n = len(codes)
    out = []
    for b0 in range(0, n, BLOCK):
        b1 = min(b0 + BLOCK, n)
        inside = 0
        for g in range(b0 + 1, b1):
            lo, hi = d[b0:g], d[g + 1:b1 + 1]
            inside += bool(np.any(lo < d[g])) and bool(np.any(hi < d[g]))
        out.append(b1 - b0 - inside)
    return np.array(out)


def test_the_codes_make_long_forests():
    codes = chain_codes(GROUP)
    t = triangles(codes)
    got, _ = lbvh_np.morton_codes(t, -1)
    assert np.array_equal(got, codes)
    sizes = forest_sizes(codes)
    assert sizes.max() <= 127 and sizes.sum() > BLOCK, sizes


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [GROUP, GROUP + 1, 3 * GROUP])
@pytest.mark.parametrize("mode", [1, 0])
def test_long_forests(built_lib, blocks, mode):
    import lighttransportsimulation_gb300 as lts
    codes = chain_codes(blocks)
    t = triangles(codes)
    if mode == 1:
        t = t[np.random.default_rng(blocks).permutation(len(t))]
    ctx = lts.Context(0)
    out = lts.build_bvh_triangles(ctx, t, mode, -1)
    want, ids = lbvh_np.stable_sort(*lbvh_np.morton_codes(t, -1))
    n = len(t)
    assert np.array_equal(out["sorted_codes"], want) and np.array_equal(out["sorted_ids"], ids) and np.array_equal(want, codes)
    left, right = lbvh_np.karras_topology(want)
    assert np.array_equal(out["node_left"][: n - 1], left) and np.array_equal(out["node_right"][: n - 1], right)
    mn, mx = lbvh_np.tri_bounds(t)
    leaf = np.concatenate([mn, mx], 1)
    lbvh_np.check_tree(out["node_left"], out["node_right"], out["node_bounds"], leaf if mode == 0 else leaf[ids])
    ctx.close()
