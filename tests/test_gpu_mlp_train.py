"""The training kernels at the edges of their tiles: 32-sample CTAs, 128-sample dot products, 32 of those in shared
memory at a time and 8,192 samples per launch, against the FP64 oracle with the same BF16 roundings."""
import numpy as np
import pytest

from multigridsoftbody_b200.learned import MLP
from oracle.binding import mlp_loss_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 4095, 4097, 8192, 8193, 20001])
def test_gradient_at_tile_edges(lib, oracle_built, n):
    rng = np.random.default_rng(n)
    net = MLP(seed=11)
    x = rng.normal(size=(n, 9)).astype(np.float32)
    t = rng.normal(size=(n, 3)).astype(np.float32)
    loss, g = net.loss_grad(x, t)
    lo, go = mlp_loss_grad(net.params.astype(np.float64), x.astype(np.float64), t.astype(np.float64), bf16=True)
    # FP32 sums over n samples, and hidden activations that round to the other BF16 neighbour
    assert abs(loss - lo) <= 1e-3 * lo
    for a, b in ((0, 576), (576, 640), (640, 4736), (4736, 4800), (4800, 4992), (4992, 4995)):
        assert np.linalg.norm(g[a:b] - go[a:b]) <= 1e-2 * np.linalg.norm(go[a:b]) + 1e-6, (a, b)
    net.close()


@pytest.mark.parametrize("batch", [77, 9000])
def test_training_step_is_the_gradient_step(lib, batch):
    """One Adam step from zero moments moves every parameter by lr * sign(gradient) (the bias corrections cancel):
    the sampled minibatch's loss and step come from the same sums as loss_grad on those samples."""
    rng = np.random.default_rng(3)
    x = rng.normal(size=(1, 9)).astype(np.float32)   # one pair: every sample is it
    t = rng.normal(size=(1, 3)).astype(np.float32)
    net = MLP(seed=5)
    before = net.params
    loss, g = net.loss_grad(np.repeat(x, batch, 0), np.repeat(t, batch, 0))
    losses = net.train(x, t, steps=1, batch=batch, lr=1e-3, seed=1)
    assert losses[0] == np.float32(loss)
    moved = net.params - before
    clear = np.abs(g) > 1e-5   # eps = 1e-8 against sqrt(g^2): within 1e-3 of lr; FP32 parameters up to 0.5: 6e-8
    assert np.allclose(moved[clear], -1e-3 * np.sign(g[clear]), rtol=2e-3, atol=1e-7)
    net.close()
