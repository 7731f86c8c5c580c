"""A refine wait that runs out reaches the caller of every entry point that refines.

As in test_failures.py nothing faults: the tensor-core refine withholds a
stage (wait limit about 0.1 s); the FP32 refine, whose only waits are those
between its rounds, gets a limit of one cycle.  Either records the timeout
and returns; the pairs not met are missing, so the call must fail.
"""
import numpy as np
import pytest

import paddi_b200 as P
from oracle import oracle as O
from paddi_b200 import datagen, sharded

pytestmark = pytest.mark.gpu


def _threshold(x, m):
    nn, _ = O.nn_profile(x, m)
    return float(np.float32(np.quantile(nn, 0.99)))  # some candidates reach the refine


@pytest.mark.parametrize("dist", [P.DIST_SPLIT_FP16, P.DIST_SPLIT_BF16])
def test_sharded_refine_reports_a_timeout(dist):
    x, _ = datagen.palmad_series(n=1 << 13, seed=21, n_anom=4, min_len=32, max_len=96)
    m, N = 80, (1 << 13) - 79
    r2 = _threshold(x, m)
    with P.Context(device=0, distance_kernel=dist) as ctx:
        be = sharded.GpuBackend(ctx, x, device=0)
        alive = be.phase1(m, r2, 0, N)
        ind, rho, pr = be.refine(m, r2, alive, 0, N)
        assert len(ind) > 0
        want, _ = be.select(m, r2, ind, rho, pr, 1)
        ctx.debug_set(P.DEBUG_WAIT_CYCLES, 200_000_000)
        ctx.debug_set(P.DEBUG_WITHHOLD_STAGE, 1)
        with pytest.raises(P.PaddiError) as e:
            be.refine(m, r2, alive, 0, N)
        assert e.value.status == P.PADDI_ERR_CUDA and "timed out" in str(e.value)
        ctx.debug_set(P.DEBUG_WITHHOLD_STAGE, 0)
        ctx.debug_set(P.DEBUG_WAIT_CYCLES, 0)
        ind, rho, pr = be.refine(m, r2, alive, 0, N)
        again, _ = be.select(m, r2, ind, rho, pr, 1)
        assert again == want


def test_the_message_names_the_refine_that_gave_up():
    """n above 65536 windows: four rounds.  The FP32 refine's blocks without work in a
    round wait for the others', here at most one cycle."""
    x, _ = datagen.palmad_series(n=1 << 17, seed=4, n_anom=8, min_len=32, max_len=96)
    m = 80
    with P.Context(device=0, distance_kernel=P.DIST_FP32) as ctx:
        (top,), _ = ctx.pd3(x, m)
        r = 0.7 * float(np.sqrt(top.dist))
        want, (row,) = ctx.pd3(x, m, r=r)
        assert row["n_cand"] > 8  # more than one tile: the rounds go on
        ctx.debug_set(P.DEBUG_WAIT_CYCLES, 1)
        with pytest.raises(P.PaddiError) as e:
            ctx.pd3(x, m, r=r)
        assert e.value.status == P.PADDI_ERR_CUDA
        assert "FP32 refine" in str(e.value) and "timed out" in str(e.value)
        ctx.debug_set(P.DEBUG_WAIT_CYCLES, 0)
        again, _ = ctx.pd3(x, m, r=r)
        assert again == want
