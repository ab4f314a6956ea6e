"""Radiance-cache inference over tiles, groups and partial tiles, through both feature paths (row
order by TMA, listed rows by cp.async are the renderer's), against the oracle."""
import numpy as np
import pytest

from oracle import mlp_np

pytestmark = pytest.mark.gpu


# one row; around a 128-row tile; around one tile on each of 152 SMs; around five tiles in flight per
# SM (97,280 rows), which makes a warpgroup take a second tile
@pytest.mark.parametrize("n", [1, 127, 128, 129, 19455, 19457, 97280, 97281, 100003])
def test_rows(built_lib, n):
    import lighttransportsimulation_gb300 as lts
    ctx = lts.Context(0)
    net = lts.RadianceCacheMLP(ctx, seed=3)
    rng = np.random.default_rng(n)
    params = mlp_np.he_init(n)
    net.set_params(params)
    feat = mlp_np.bf16_bits(rng.uniform(-1, 1, (n, 96)).astype(np.float32))
    out = net.forward(feat)
    ref = mlp_np.forward(params, feat)
    # the oracle rounds to bf16 where the kernel does; FP32 sums in another order can move an
    # activation to its other bf16 neighbour (2^-8 relative), a few of 64 inputs of later layers
    assert np.allclose(out, ref, rtol=2e-2, atol=1e-4)
    assert np.sqrt(np.mean((out - ref) ** 2)) <= 2e-3 * np.sqrt(np.mean(ref ** 2))
    ctx.close()


def test_nan_and_infinite_features(built_lib):
    """A NaN pre-activation leaves ReLU as 0, as fmaxf gives; rows beside it are not touched."""
    import lighttransportsimulation_gb300 as lts
    ctx = lts.Context(0)
    net = lts.RadianceCacheMLP(ctx, seed=3)
    rng = np.random.default_rng(0)
    feat = mlp_np.bf16_bits(rng.uniform(-1, 1, (256, 96)).astype(np.float32))
    clean = net.forward(feat)
    feat[130, 5] = 0x7FC0
    feat[200, 7] = 0x7F80
    out = net.forward(feat)
    keep = np.ones(256, bool)
    keep[[130, 200]] = False
    assert np.array_equal(out[keep], clean[keep])
    assert np.array_equal(out[130], np.ones(3, np.float32))  # every hidden unit 0: exp(0)
    ctx.close()


# training: one row; around a 128-row tile; around one tile on each of 152 SMs, which makes a CTA take a second
# tile (the other feature buffer) and a third (the first one again)
@pytest.mark.parametrize("n", [1, 127, 129, 19455, 19457, 38913])
def test_gradients(built_lib, n):
    import lighttransportsimulation_gb300 as lts
    ctx = lts.Context(0)
    net = lts.RadianceCacheMLP(ctx, seed=3)
    rng = np.random.default_rng(n)
    params = mlp_np.he_init(n)
    net.set_params(params)
    feat = mlp_np.bf16_bits(rng.uniform(-1, 1, (n, 96)).astype(np.float32))
    target = rng.uniform(0, 2, (n, 3)).astype(np.float32)
    loss, g = net.train_step(feat, target, lr=0.0, want_grad=True)
    loss_ref, g_ref = mlp_np.loss_and_grad(params, feat, target)
    # the repository's own bounds: bf16 rounding points are the oracle's, sums come in another order
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref)
    for off, (o, i) in zip(mlp_np.OFFSETS, mlp_np.LAYERS):
        a, b = g[off:off + o * i], g_ref[off:off + o * i]
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b)
    ctx.close()
