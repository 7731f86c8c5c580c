"""The refines' rounds in one launch, and phase 1's split segments.

Rounds start at 65536 windows; a candidate tile holds 16 (tensor cores, 8 for
64-row tiles) or 8 (FP32) candidates.  Thresholds are taken from the FP64 nn
profile so that a chosen number of candidates survives: none, one, a tile's
worth and one more, many.  Counts must equal the profile's exactly.
"""
import numpy as np
import pytest

from oracle import oracle as O
from paddi_b200 import datagen

pytestmark = pytest.mark.gpu

# windows, length (K' = 48: all products at once; 128, 416: tiles are screened
# where a work item has four or more, i.e. with thousands of candidates)
@pytest.fixture(scope="module", params=[(65536 - 1, 40), (65536, 40), (65536 + 2048 + 7, 40),
                                        (65536 + 2048 + 7, 120), (66001, 400)])
def case(request):
    N, m = request.param
    x, _ = datagen.pd3_series(n=N + m - 1, seed=11, n_anom=4, anom_len=100)
    return x, m, np.sort(O.nn_profile_fast(x, m).astype(np.float32))


@pytest.mark.parametrize("dist,rows", [("fp32", 0), ("fp16", 0), ("fp16", 64), ("bf16", 0)])
def test_survivor_counts_across_rounds(case, dist, rows):
    import paddi_b200 as P
    x, M, nn = case
    k = {"fp32": P.DIST_FP32, "fp16": P.DIST_SPLIT_FP16, "bf16": P.DIST_SPLIT_BF16}[dist]
    with P.Context(device=0, distance_kernel=k, tile_rows=rows) as ctx:
        for keep in (0, 1, 8, 9, 16, 17, 300, 5000):
            v = float(nn[-1]) * 1.01 if keep == 0 else 0.5 * (float(nn[-keep]) + float(nn[-keep - 1]))
            r = float(np.sqrt(np.float32(v)))
            r2 = float(np.float32(r) * np.float32(r))
            _, (a,) = ctx.pd3(x, M, r=r)
            assert a["n_cand"] == int((nn >= r2).sum()), keep
            assert a["n_disc"] == int((nn > r2).sum()), keep


@pytest.mark.parametrize("n,m", [(300, 20), (64 * 15 * 148 // 8, 30), (64 * 15 * 148 + 40, 40)])
@pytest.mark.parametrize("seg", [64, 72, 256, 520, 4096])
def test_phase1_tasks_do_not_change_results(n, m, seg):
    """Every split of the rows gives the same candidates (the last n has more rows
    than one 64-row task per resident warp covers)."""
    import paddi_b200 as P
    x, _ = datagen.pd3_series(n=n, seed=5, n_anom=2, anom_len=max(10, min(100, n // 40)))
    with P.Context(device=0) as ctx:
        ref, rl = ctx.pd3(x, m, segment_len=256)
        got, gl = ctx.pd3(x, m, segment_len=seg)
    assert [(d.ind, d.dist) for d in got] == [(d.ind, d.dist) for d in ref]
    assert [(a["n_cand"], a["n_disc"]) for a in gl] == [(a["n_cand"], a["n_disc"]) for a in rl]
