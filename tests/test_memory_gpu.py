"""Memory that a context can do without is given up before a call fails.

A refused allocation is made on the host (PADDI_DEBUG_FAIL_ALLOC refuses the
k-th next one once).  The buffers of the series are reserved before, so the
count starts at the run's own allocations.
"""
import numpy as np
import pytest

import paddi_b200 as P
from paddi_b200 import datagen

pytestmark = pytest.mark.gpu


def _noise_series(n=30000):
    x, _ = datagen.palmad_series(n=n, seed=2, n_anom=4, min_len=64, max_len=96,
                                 kinds_cycle=("noise",))
    return x


def _give_up_block_maxima(ctx):
    """A refused allocation takes the block maxima's memory first, and fails only then."""
    ctx.debug_set(P.DEBUG_FAIL_ALLOC, 1)
    ctx.debug_set(P.DEBUG_RECHECK_CAP, 1024)
    assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0


def _rows(log):
    return [(a["m"], a["r"], a["n_cand"], a["n_disc"]) for a in log]


@pytest.mark.parametrize("policy,k", [(P.R_MERLIN, 1), (P.R_BOUND, 2)])
def test_a_run_goes_on_without_memory_for_the_witnesses(policy, k):
    """(the bound's dot products are allocated before the witnesses)"""
    x = _noise_series()
    with P.Context(device=0, r_policy=policy) as ctx:
        ctx.reserve(len(x), 80)
        _give_up_block_maxima(ctx)
        ctx.debug_set(P.DEBUG_FAIL_ALLOC, k)
        got, log = ctx.palmad(x, 64, 80)
        assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0
        assert ctx.debug_get(P.DEBUG_WITNESS_STEPS) == 0  # none carried
        want, wlog = ctx.palmad(x, 64, 80)
        assert ctx.debug_get(P.DEBUG_WITNESS_STEPS) > 0
    assert got == want and _rows(log) == _rows(wlog)


@pytest.mark.parametrize("policy,k", [(P.R_MERLIN, 2), (P.R_BOUND, 3), (P.R_BOUND, 4)])
def test_witnesses_are_given_up_for_memory_needed_later(policy, k):
    """The profile's buffers are allocated after the first length's attempts: refused
    once, they take the witnesses' memory, and the lengths after run without."""
    x = _noise_series()
    with P.Context(device=0, r_policy=policy) as ctx:
        ctx.reserve(len(x), 80)
        ctx.debug_set(P.DEBUG_FAIL_ALLOC, k)
        got, log, prof = ctx.palmad_profiled(x, 64, 70)
        assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0
        assert ctx.debug_get(P.DEBUG_WITNESS_STEPS) == 0
        want, wlog, wprof = ctx.palmad_profiled(x, 64, 70)
    assert got == want and _rows(log) == _rows(wlog)
    # a distance is known to the guard band (2e-4 in correlation) on each side
    for j, (a, b) in enumerate(zip(prof, wprof)):
        np.testing.assert_array_equal(a > 0, b > 0)
        assert np.abs(a - b)[a > 0].max() <= 2 * 2 * (64 + j) * 2e-4


@pytest.mark.parametrize("policy", [P.R_MERLIN, P.R_BOUND])
def test_witnesses_are_given_up_for_the_recheck_queue(policy):
    """A recheck queue of one window overflows (with a wide guard band) while the
    run's witnesses are in use; its growth, refused once, takes their memory."""
    x = _noise_series()
    with P.Context(device=0, r_policy=policy, guard=0.01) as ctx:
        want, wlog = ctx.palmad(x, 64, 80)  # all buffers are there from now on
        assert max(a["n_recheck"] for a in wlog) > 1
        ctx.debug_set(P.DEBUG_RECHECK_CAP, 1)
        ctx.debug_set(P.DEBUG_FAIL_ALLOC, 1)
        got, log = ctx.palmad(x, 64, 80)
        assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0
        assert ctx.debug_get(P.DEBUG_WITNESS_STEPS) < 16
    assert got == want and _rows(log) == _rows(wlog)


@pytest.mark.parametrize("k", [1, 2])
def test_a_refused_growth_leaves_the_recheck_queue(k):
    """Either buffer of the larger queue refused: the call fails, the queue stays as it
    was and the next call, which grows it, is a good one."""
    x = _noise_series(8192)
    with P.Context(device=0) as ctx:
        want, _ = ctx.pd3(x, 64, top_k=4)
        _give_up_block_maxima(ctx)
        ctx.debug_set(P.DEBUG_RECHECK_CAP, 1)
        ctx.debug_set(P.DEBUG_FAIL_ALLOC, k)
        with pytest.raises(P.PaddiError) as e:
            ctx.pd3(x, 64, top_k=4)
        assert e.value.status == P.PADDI_ERR_OUT_OF_MEMORY
        assert ctx.debug_get(P.DEBUG_RECHECK_CAP) == 1
        got, _ = ctx.pd3(x, 64, top_k=4)
        assert ctx.debug_get(P.DEBUG_RECHECK_CAP) > 1
    assert got == want


@pytest.mark.parametrize("dist", [P.DIST_SPLIT_FP16, P.DIST_SPLIT_BF16])
@pytest.mark.parametrize("when", ["at the start", "in use"])
def test_searches_run_without_memory_for_the_block_maxima(dist, when):
    """Refused at the start (the last of the 18 buffers of a series), or given up for a
    growing recheck queue: the recheck then scans the whole series."""
    x = _noise_series()
    with P.Context(device=0, distance_kernel=dist) as ctx:
        want, wlog = ctx.pd3(x, 64, top_k=4)
    with P.Context(device=0, distance_kernel=dist) as ctx:
        if when == "at the start":
            ctx.debug_set(P.DEBUG_FAIL_ALLOC, 18)
        else:
            ctx.reserve(len(x), 64)
            ctx.debug_set(P.DEBUG_RECHECK_CAP, 1)
            ctx.debug_set(P.DEBUG_FAIL_ALLOC, 1)
        got, log = ctx.pd3(x, 64, top_k=4)
        assert ctx.debug_get(P.DEBUG_FAIL_ALLOC) == 0
        again, _ = ctx.pd3(x, 64, top_k=4)
    assert got == want and again == want and _rows(log) == _rows(wlog)
