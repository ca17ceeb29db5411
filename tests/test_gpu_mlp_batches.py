"""The fused training batch at the edges of its 16-row tiles, its 256-row K
passes and the hidden product's 128-row tiles, against the numpy oracle with
the tolerances of the other gradient tests (the oracle rounds to BF16 at the
kernels' points; what is left is FP32 summation order and the flips of a
BF16 rounding it causes)."""
import numpy as np
import pytest

from oracle import mlp_ref
from test_gpu_mlp import BLOCKS, H, N_IN, N_OUT, blocks, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 127, 129, 255, 256, 257, 513])
def test_gradient_at_tile_edges(boids_lib, rows):
    net = boids_lib.Surrogate(N_IN, H, N_OUT, seed=4)
    rng = np.random.default_rng(rows)
    p = net.params()
    p[N_IN * H:N_IN * H + H] = rng.normal(0, 0.1, H)
    net.set_params(p)
    x = rng.random((rows, N_IN), dtype=np.float32)
    t = rng.normal(0, 1, (rows, N_OUT)).astype(np.float32)
    g, loss = net.gradient(x, t)
    gr, lr_ = mlp_ref.gradient(p, x, t, N_IN, H, N_OUT)
    assert loss == pytest.approx(lr_, rel=2e-3)
    gb, grb = blocks(g), blocks(gr)
    for name in BLOCKS:
        assert rel(gb[name], grb[name]) < 5e-3, name
    net.close()


def test_one_batch_of_training_is_the_gradient_and_adam(boids_lib):
    """One epoch of one batch equals Adam's first step on the gradient."""
    net = boids_lib.Surrogate(N_IN, H, N_OUT, seed=4)
    rng = np.random.default_rng(1)
    x = rng.random((100, N_IN), dtype=np.float32)
    t = rng.normal(0, 1, (100, N_OUT)).astype(np.float32)
    p = net.params()
    g, _ = net.gradient(x, t)
    net.train(x, t, epochs=1, batch=100, lr=1e-3, seed=3)
    # m / c1 = g and v / c2 = g^2 up to a few FP32 roundings of each (1e-5
    # relative); the shuffled rows change g by its own summation order
    want = p - 1e-3 * g / (np.abs(g) + 1e-8)
    moved = np.abs(g) > 1e-4 * np.abs(g).max()
    assert np.abs((net.params() - want)[moved]).max() < 1e-3 * 2e-2
    net.close()
