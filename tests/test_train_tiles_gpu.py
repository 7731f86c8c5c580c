"""The training kernel's sample tiles (32) and row order: the gradient at tile
edges against the float64 restatement, and one epoch of a permuted batch
against the same steps taken one by one.

Tolerance of the gradient: FP32 sums of at most n + 64 + 64 + 12 products of
values bounded by a few units, relative to the largest entry: (n + 140) 2^-24 x 8.
"""
import numpy as np
import pytest

import paddi_b200 as P
from tests.test_learned_r import _data, np_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 32 * 148 + 5])
def test_gradient_at_tile_edges(n):
    X, Y = _data(n, seed=n)
    p = P.init_params(2)
    with P.Context(device=0) as c:
        g, loss = c.model_grad(X, Y, p, tau=0.3)
    want, wl = np_grad(p, X.astype(np.float64), Y.astype(np.float64), float(np.float32(0.3)))
    tol = 8 * (n + 140) * 2.0 ** -24
    assert np.abs(g - want).max() <= tol * max(np.abs(want).max(), 1e-3)
    assert abs(loss - wl) <= tol * abs(wl)


def test_a_batch_of_everything_is_one_step_of_any_order():
    """With one batch per epoch the order cannot matter beyond rounding: one Adam
    step of the full gradient (its size is the learning rate)."""
    X, Y = _data(77, seed=5)
    p0 = P.init_params(4)
    with P.Context(device=0) as c:
        a, _ = c.model_train(X, Y, tau=0.2, epochs=1, batch=77, lr=1e-3, seed=1, init=p0)
        b, _ = c.model_train(X, Y, tau=0.2, epochs=1, batch=4096, lr=1e-3, seed=9, init=p0)
        g, _ = c.model_grad(X, Y, p0, tau=0.2)
    sure = np.abs(g) > 1e-4 * np.abs(g).max()
    want = p0 - 1e-3 * np.sign(g)
    assert np.abs(a - want)[sure].max() < 2e-5 and np.abs(b - want)[sure].max() < 2e-5
