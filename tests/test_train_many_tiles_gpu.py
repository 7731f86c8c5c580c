"""The training kernel with several tiles per CTA: the gradient kept in
registers from tile to tile.

n = 3 * 32 * 148 + 5: every CTA of a 148-SM GPU takes three full tiles and one a
fourth of 5 samples, whose features and targets are large enough to carry 7 % of
the largest entry.  Leaving out any tile moves the gradient by far more than
the tolerance, which does not grow with n: a CTA sums at most 128 samples in
FP32 (with 140 terms of the layers' sums), CTAs are added in FP64, so 8 (128 +
140) 2^-24 of the largest entry.  (The loss's slope has a sign per sample: none of
the samples' errors is near zero, so rounding cannot turn it.)
"""
import numpy as np
import pytest

import paddi_b200 as P
from tests.test_learned_r import _data, np_forward, np_grad

pytestmark = pytest.mark.gpu

N = 3 * 32 * 148 + 5
TOL = 8 * (128 + 140) * 2.0 ** -24


def _samples():
    X, Y = _data(N, seed=11)
    p = P.init_params(2)
    X[-5:] *= 20
    Y[-5:] -= 400
    y, _ = np_forward(p, X.astype(np.float64))
    e = Y - y
    keep = np.abs(e) < 1e-4  # moved away from the kink
    Y[keep] += 0.01
    return p, X, Y


def test_gradient_over_several_tiles_per_block():
    p, X, Y = _samples()
    tau = float(np.float32(0.3))
    X64, Y64 = X.astype(np.float64), Y.astype(np.float64)
    want, wl = np_grad(p, X64, Y64, tau)
    # what is left without the last tile, and without any block's third
    for cut in (slice(0, N - 5), slice(0, 2 * 32 * 148)):
        part, _ = np_grad(p, X64[cut], Y64[cut], tau)
        part *= len(X64[cut]) / N
        assert np.abs(part - want).max() > 100 * TOL * np.abs(want).max()
    with P.Context(device=0) as c:
        g, loss = c.model_grad(X, Y, p, tau=0.3)
    assert np.abs(g - want).max() <= TOL * np.abs(want).max()
    assert abs(loss - wl) <= TOL * abs(wl)
