"""Witnesses taken back to a length (k_witness.cu) when the next length's new
value is a spike.

A missed attempt whose next length was already queued steps every pair's dot
product back.  Where the value taken away is a spike (here 1e7 to 1e9 beside
windows of unit size), what is left of the shorter windows' dot product is the
rounding of the spike's: it must prove nothing.  The series: eight beats of
2048 values, zero at their ends, a spike at 2000 of each, one beat altered just
before it, and a bump 64 values before it, at which the top distance drops (at
length 64 the schedule misses several times).  A run and the same attempts
alone, without witnesses, must agree in every discord and count.
"""
import numpy as np
import pytest

import paddi_b200 as P
from paddi_b200 import datagen

pytestmark = pytest.mark.gpu


def _series(seed, spike, beats=8):
    rng = np.random.default_rng(seed)
    base = np.cumsum(rng.normal(0, 1, 1920))
    base -= np.linspace(base[0], base[-1], 1920)
    base = base / base.std() + 8.0
    x = np.zeros((beats, 2048), np.float32)
    for b in range(beats):
        x[b, 80:2000] = base + rng.normal(0, 0.004, 1920)
        x[b, 2000] = spike * (1 + 0.01 * rng.random())
        x[b, 2000 - 64] += 12.0
    x[beats // 2, 1999] += 3.0
    x[beats // 2, 1990] -= 1.0
    return x.reshape(-1)


@pytest.mark.parametrize("spike", [1e7, 1e8, 1e9])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_a_value_taken_back_leaves_no_false_proof(seed, spike):
    x = _series(seed, spike)
    with P.Context(device=0, r_policy=P.R_BOUND) as ctx, \
            P.Context(device=0, r_policy=P.R_BOUND) as one:
        got, log = ctx.palmad(x, 60, 68)
        assert sum(a["m"] == 64 for a in log) > 1  # steps back happened
        for k, d in enumerate(got):
            (e,), _ = one.palmad(x, 60 + k, 60 + k)
            assert (d.ind, d.dist) == (e.ind, e.dist), 60 + k
        for a in log:  # (the schedule's r may be negative; its square is the threshold)
            _, rows = one.pd3(x, a["m"], r=abs(a["r"]))
            assert [(b["n_cand"], b["n_disc"]) for b in rows] == [(a["n_cand"], a["n_disc"])], a


@pytest.mark.parametrize("guided", [True, False])
def test_the_bound_counts_every_step(guided):
    """The rounding bound of a carried pair scales with the steps taken over each
    value: one per length, and two more per attempt that missed with the next length
    queued (the guided policies queue it, for all lengths but the last).  (The
    reference's schedule runs on noise anomalies: it can stand still on others.)"""
    if guided:
        x, lo = _series(0, 10.0), 60
    else:
        x, _ = datagen.palmad_series(n=30000, seed=2, n_anom=4, min_len=64, max_len=96,
                                     kinds_cycle=("noise",))
        lo = 64
    with P.Context(device=0, r_policy=P.R_BOUND if guided else P.R_MERLIN) as ctx:
        _, log = ctx.palmad(x, lo, lo + 8)
        steps2 = ctx.debug_get(P.DEBUG_WITNESS_STEPS)
    tries = [sum(a["m"] == m for a in log) for m in range(lo, lo + 8)]
    assert tries[0] > 1
    assert steps2 == sum((2 * t - 1 if guided else 1) ** 2 for t in tries)
