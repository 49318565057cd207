"""GPU: training step by step, the route of a device without room for a 16-CTA cluster.

Its sums run in the cluster kernel's order, so weights, loss and the optimiser's state (further
steps from there) are the same bit for bit, also where the two routes alternate."""
import ctypes

import numpy as np
import pytest

import dr_b200

pytestmark = pytest.mark.gpu


def _steps(mlp, x, t, steps, lr=3e-3):
    f = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))  # noqa: E731
    loss = ctypes.c_float()
    assert dr_b200.lib().dr_debug_mlp_train_steps(mlp._h, f(x), f(t), len(x), steps, lr, ctypes.byref(loss)) == 0
    return loss.value


@pytest.mark.parametrize("B", [1, 16, 305, 1000])
def test_routes_agree(engine, B):
    rng = np.random.default_rng(B)
    x, t = rng.normal(0, 1, (B, 4)).astype(np.float32), rng.normal(0, 1, (B, 4)).astype(np.float32)
    a, b = dr_b200.MLP(engine, seed=5), dr_b200.MLP(engine, seed=5)
    for n in (1, 7, 0, 20):
        assert _steps(b, x, t, n) == a.train(x, t, n)
        assert np.array_equal(a.get_weights(), b.get_weights()), n
    assert _steps(a, x, t, 5) == b.train(x, t, 5)
    assert np.array_equal(a.get_weights(), b.get_weights())
