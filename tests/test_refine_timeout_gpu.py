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
