"""Losses, gradients and Adam steps of the network on ragged batches.

loss_grad on 1, 33, 63 and 65 samples (a lone sample, a second tile of one, a
last tile one short, a third tile of one) against the FP64 oracle: a value is
the end of at most nine chained products of 64 or fewer FP32 terms, 64 * 6e-8 =
4e-6 relative each in the worst case, 3.5e-5 in all, so 1e-4 in norm.

Six Adam steps in one stream of programmatic launches, batches of 64, 64 and 22
twice over, against an FP64 Adam loop over the oracle's gradients, with eps =
1e-2 so that a step is a smooth function of the gradients (a step of lr times
m / (sqrt(v) + eps) moves by at most 2 lr / eps times a gradient's error). Those
errors are 3.5e-5 of gradients of at most 0.6, 2.1e-5, hence 4.2e-3 lr a step
and 2.5e-2 lr in all; 4e-2 lr is allowed. (Dividing the batch of 22 by 32 moves
parameters by 0.15 lr.)
"""
import ctypes

import numpy as np
import pytest

from oracle import mlp_oracle as O

pytestmark = pytest.mark.gpu


def data(n, seed):
    x = np.random.default_rng(seed).uniform(-1.5, 1.5, size=(n, 4)).astype(np.float32)
    y = np.stack([np.cos(x[:, 0]), np.sin(x[:, 1]), x[:, 2] * x[:, 3]], 1).astype(np.float32)
    return x, y


@pytest.mark.parametrize("n", [1, 33, 63, 65])
def test_loss_and_gradient_on_partial_tiles(n):
    from lbm_solver_3d_b200.mlp import MLP
    x, y = data(n, 31)
    th = O.init_params(4).astype(np.float32)
    net = MLP(bf16=False, params=th)
    net.set_data(x, y)
    loss, g = net.loss_grad()
    lo, go = O.loss_grad(th.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    assert abs(loss - lo) <= 1e-4 * lo
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)
    net.close()


def test_adam_steps_follow_the_rule():
    from lbm_solver_3d_b200.mlp import MLP
    n, batch, lr, b1, b2, eps = 150, 64, 2e-3, 0.9, 0.999, 1e-2
    x, y = data(n, 32)
    th = O.init_params(5).astype(np.float32)
    net = MLP(bf16=False, params=th)
    assert net.lib.lbmgpu_mlp_set_adam(net.h, ctypes.c_float(b1), ctypes.c_float(b2), ctypes.c_float(eps)) == 0
    net.set_data(x, y)
    want, m, v, t = th.astype(np.float64), 0.0, 0.0, 0
    for epoch in range(2):
        order = np.random.default_rng([33, epoch]).permutation(n).astype(np.int32)
        net.train_epoch(order, batch=batch, lr=lr)
        for k in range(0, n, batch):
            i = order[k:k + batch]
            _, g = O.loss_grad(want, x[i].astype(np.float64), y[i].astype(np.float64))
            assert np.abs(g).max() <= 0.6
            t += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            want = want - lr * (m / (1 - b1 ** t)) / (np.sqrt(v / (1 - b2 ** t)) + eps)
    assert np.abs(net.params() - want).max() <= 4e-2 * lr
    net.close()
