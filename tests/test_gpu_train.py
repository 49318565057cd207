"""GPU: the training kernel (dr_mlp_train) step by step.

One Adam update from a known state depends only on the gradient, which dr_mlp_grad gives at
the same weights: after each single step the weights are compared with the update computed
in float64 from that gradient.  Batch sizes around the 16 CTAs x 8 examples of the kernel
and its chunks of 320 examples.  Tolerance: 1 - powf(0.999, t) loses up to 2^-25 / 1e-3 =
3e-5 relative at t = 1, half of it after the square root, so 1e-4 of the learning rate plus
the rounding of the weight itself.  Many steps in one call equal as many single steps.
"""
import numpy as np
import pytest

import dr_b200

pytestmark = pytest.mark.gpu
LR = 3e-3


def _data(B, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (B, 4)).astype(np.float32), rng.normal(0, 1, (B, 4)).astype(np.float32)


@pytest.mark.parametrize("B", [1, 15, 16, 17, 128, 129, 319, 320, 321, 705, 4096])
def test_single_steps(engine, B):
    x, t = _data(B, B)
    mlp = dr_b200.MLP(engine, seed=3)
    w = np.random.default_rng(B + 1).normal(0, 0.2, mlp.n_params).astype(np.float32)
    mlp.set_weights(w)
    m = v = np.zeros(mlp.n_params)
    b1, b2 = np.float32(0.9), np.float32(0.999)
    for step in range(1, 5):
        g, loss = mlp.grad(x, t)
        assert abs(mlp.train(x, t, 1, LR) - loss) <= 1e-6 * loss
        g = g.astype(np.float64)
        m = float(b1) * m + float(np.float32(1) - b1) * g
        v = float(b2) * v + float(np.float32(1) - b2) * g * g
        want = w - LR * (m / (1 - float(b1) ** step)) / (np.sqrt(v / (1 - float(b2) ** step)) + 1e-8)
        w = mlp.get_weights()
        assert np.all(np.abs(w - want) <= 1e-4 * LR + 2.0**-23 * np.abs(want)), (B, step)


def test_steps_in_one_call(engine):
    x, t = _data(305, 9)
    a, b = dr_b200.MLP(engine, seed=5), dr_b200.MLP(engine, seed=5)
    la = a.train(x, t, 12, LR)
    for _ in range(12):
        lb = b.train(x, t, 1, LR)
    assert la == lb and np.array_equal(a.get_weights(), b.get_weights())
    assert a.train(x, t, 0, LR) == la and np.array_equal(a.get_weights(), b.get_weights())
