"""Worker contexts of batched calls: what they keep, what a failure inside one does.

Every result is compared with the series' own runs on a fresh context.
"""
import numpy as np
import pytest

import paddi_b200 as P
from paddi_b200 import datagen
from tests.test_witness_back_gpu import _series as spiky_series

pytestmark = pytest.mark.gpu


def _walks(lens, seed):
    return [datagen.random_walk_sine(n, np.random.default_rng(seed + k)).astype(np.float32)
            for k, n in enumerate(lens)]


def _alone(xs, lo, hi, **kw):
    out = []
    for x in xs:
        with P.Context(device=0, **kw) as c:
            out.append(c.palmad(x, lo, hi)[0])
    return out


@pytest.mark.parametrize("k", [1, 9, 20])
def test_a_series_that_does_not_fit_beside_the_others_runs_alone(k):
    """The first worker's k-th allocation is refused (of its series' buffers, then the
    bound's dot products after them): the series runs again on a single worker."""
    xs = _walks([9000, 7000, 5000, 3000], 1)
    with P.Context(device=0, r_policy=P.R_BOUND) as ctx:
        ctx.debug_set(P.DEBUG_FAIL_ALLOC, k)
        got, _ = ctx.palmad_batched(xs, 20, 28, streams=3)
        assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0
    assert got == _alone(xs, 20, 28, r_policy=P.R_BOUND)


def test_idle_workers_are_dropped_for_an_allocation_of_their_context():
    xs = _walks([9000, 7000, 5000], 2)
    with P.Context(device=0, r_policy=P.R_BOUND) as ctx:
        ctx.palmad_batched(xs, 20, 28, streams=3)
        assert ctx.debug_get(P.DEBUG_WORKERS) == 3
        ctx.debug_set(P.DEBUG_FAIL_ALLOC, 4)
        got, _ = ctx.palmad(xs[0], 20, 28)
        assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0 and ctx.debug_get(P.DEBUG_WORKERS) == 0
        again, _ = ctx.palmad_batched(xs, 20, 28, streams=2)
        assert ctx.debug_get(P.DEBUG_WORKERS) == 2
    want = _alone(xs, 20, 28, r_policy=P.R_BOUND)
    assert got == want[0] and again == want


def test_workers_of_long_series_are_not_kept():
    """At most 2^23 points in all are kept between calls."""
    xs = _walks([1 << 22, 1 << 22, 1 << 22], 3)
    with P.Context(device=0, r_policy=P.R_BOUND) as ctx:
        ctx.palmad_batched(xs, 64, 64, streams=3)
        assert ctx.debug_get(P.DEBUG_WORKERS) == 2
        ctx.palmad_batched([x[:4000] for x in xs], 20, 22, streams=3)
        assert ctx.debug_get(P.DEBUG_WORKERS) <= 2


def test_a_failure_inside_a_worker_leaves_the_next_batch_alone():
    """One series needs more attempts than allowed: its status is returned, the others'
    results are there, and a batch of the others works as before."""
    lo, hi = 60, 68
    xs = _walks([6000, 4000, 5000], 3)
    hard = spiky_series(0, 1e8)
    logs = []
    for x in xs + [hard]:
        with P.Context(device=0, r_policy=P.R_BOUND) as c:
            _, log = c.palmad(x, lo, hi)
            logs.append(max(sum(a["m"] == m for a in log) for m in range(lo, hi + 1)))
    cap = max(logs[:3])
    assert logs[3] > cap  # the fourth alone exceeds it
    with P.Context(device=0, r_policy=P.R_BOUND, iter_cap=cap) as ctx:
        first, _ = ctx.palmad_batched(xs, lo, hi, streams=2)
        with pytest.raises(P.PaddiError) as e:
            ctx.palmad_batched(xs + [hard], lo, hi, streams=2)
        assert e.value.status == P.PADDI_ERR_ITER_CAP
        assert ctx.debug_get(P.DEBUG_WORKERS) == 0
        again, _ = ctx.palmad_batched(xs, lo, hi, streams=2)
    want = _alone(xs, lo, hi, r_policy=P.R_BOUND)
    assert first == want and again == want


def test_kept_workers_take_the_model_of_the_call():
    """Two models that need different numbers of attempts on the same series: a worker
    kept from a call with the first must run the second.  (A margin far above 1 puts the
    first model's r above every top distance where it is used at all.)"""
    xs = []
    for seed in range(6):
        x, _ = datagen.palmad_series(n=20000, seed=seed, n_anom=3, min_len=30, max_len=36,
                                     kinds_cycle=("flat", "noise"))
        xs.append(x)
    lo, hi = 30, 44
    with P.Context(device=0, r_policy=P.R_LEARNED) as ctx:
        d1, a1 = ctx.palmad_batched(xs, lo, hi, streams=2)
        ctx.set_model(P.init_params(5), margin=4.0)
        d2, a2 = ctx.palmad_batched(xs, lo, hi, streams=2)
    with P.Context(device=0, r_policy=P.R_LEARNED, model=P.init_params(5),
                   model_margin=4.0) as other:
        d3, a3 = other.palmad_batched(xs, lo, hi, streams=2)
    assert list(a1) != list(a2) and list(a2) == list(a3)
    assert d1 == d2 == d3
