"""The network kernels at the edges of their tiles and grids.

Every sample's outputs depend on its inputs alone, so a call with more samples
than one wave of CTAs holds must return exactly what calls on its pieces return.
One Adam step on 1, 33 and 63 samples (a lone sample, a second tile of one, a
last tile one short) must follow the update rule at the oracle's gradient: the
first step moves each parameter by lr g / (|g| + eps), so by lr to 1 % wherever
|g| > 1e-5 (the FP32 gradient is within 1e-4 of the oracle's there).
"""
import numpy as np
import pytest

from oracle import mlp_oracle as O

pytestmark = pytest.mark.gpu


def states(n, seed):
    return np.random.default_rng(seed).uniform(-1.5, 1.5, size=(n, 4)).astype(np.float32)


@pytest.mark.parametrize("bf16,path", [(True, 2), (True, 1), (False, 1)])
def test_forward_beyond_one_wave(bf16, path):
    from lbm_solver_3d_b200.mlp import MLP
    n = 1024 * 128 + 129   # more tiles of 128, and of 32, than CTAs of any wave
    x = states(n, 5)
    net = MLP(bf16=bf16, params=O.init_params(3).astype(np.float32))
    y = net.forward(x, path=path)
    for a, b in ((0, 1), (100, 228), (n - 130, n), (n // 2, n // 2 + 1000)):
        assert np.array_equal(y[a:b], net.forward(x[a:b], path=path))
    net.close()


@pytest.mark.parametrize("n", [1, 33, 63])
def test_adam_step_on_partial_tiles(n):
    from lbm_solver_3d_b200.mlp import MLP
    x, th, lr = states(n, 8), O.init_params(9).astype(np.float32), 1e-3
    y = np.stack([np.cos(x[:, 0]), np.sin(x[:, 1]), x[:, 2] * x[:, 3]], 1).astype(np.float32)
    net = MLP(bf16=False, params=th)
    net.set_data(x, y)
    net.train_epoch(np.arange(n)[::-1], batch=64, lr=lr)
    _, g = O.loss_grad(th.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    big = np.abs(g) > 1e-5
    want = th - lr * g / (np.abs(g) + 1e-8)
    assert np.abs(net.params()[big] - want[big]).max() <= lr * 1e-2
    net.close()
