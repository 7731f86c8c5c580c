"""Witnesses carried between the lengths of a PALMAD run (k_witness.cu).

A run of several lengths selects candidates from the witnesses of the length
before; a run of one length, or a single PD3 attempt, has none.  Both must give
the same discords and, per attempt, the same candidate and discord counts
(every prune is exact).  Distances are FP64 values rounded to float on both
sides, so they are compared for equality.
"""
import numpy as np
import pytest

from paddi_b200 import datagen

pytestmark = pytest.mark.gpu


def _check(x, minL, maxL, **kw):
    import paddi_b200 as P
    with P.Context(device=0, **kw) as ctx, P.Context(device=0, **kw) as one:
        got, log = ctx.palmad(x, minL, maxL)
        for k, d in enumerate(got):
            (e,), _ = one.palmad(x, minL + k, minL + k)
            assert (d.ind, d.dist) == (e.ind, e.dist), minL + k
        for a in log:
            _, (b,) = one.pd3(x, a["m"], r=a["r"])
            assert (a["n_cand"], a["n_disc"]) == (b["n_cand"], b["n_disc"]), (a["m"], a["r"])
    return log


# tile edges of the step (1024 windows) and the check (2048), and short series (from 4 maxL
# on: every window then has a neighbour)
@pytest.mark.parametrize("n,minL,maxL", [
    (150, 3, 32), (420, 16, 100), (1024 + 31, 30, 40), (2048 + 40, 38, 45), (2049 + 40, 40, 70),
    (9001, 20, 120), (40000, 64, 200), (20000, 725, 735),
])
@pytest.mark.parametrize("policy", ["bound", "learned"])
def test_lengths_with_and_without_witnesses_agree(n, minL, maxL, policy):
    import paddi_b200 as P
    pol = {"bound": P.R_BOUND, "learned": P.R_LEARNED}[policy]
    x = datagen.random_walk_sine(n, np.random.default_rng(n + minL)).astype(np.float32)
    _check(x, minL, maxL, r_policy=pol)


def test_merlin_schedule_with_witnesses():
    """The reference's schedule (noise anomalies only: its decrement can vanish on
    other series and then never ends)."""
    import paddi_b200 as P
    x, _ = datagen.palmad_series(n=30000, seed=2, n_anom=4, min_len=64, max_len=96,
                                 kinds_cycle=("noise",))
    _check(x, 64, 80, r_policy=P.R_MERLIN)


@pytest.mark.parametrize("kind", ["near_flat", "offset", "quantised", "ecg_flat"])
@pytest.mark.parametrize("dist", ["fp16", "bf16", "fp32"])
def test_hostile_series_with_witnesses(kind, dist):
    import paddi_b200 as P
    k = {"fp16": P.DIST_SPLIT_FP16, "bf16": P.DIST_SPLIT_BF16, "fp32": P.DIST_FP32}[dist]
    x, _ = datagen.hostile_series(kind, n=1 << 14, seed=3)
    _check(x, 50, 62, r_policy=P.R_BOUND, distance_kernel=k)


def test_repeated_attempts_step_the_witnesses_back():
    """Anomalies of one short length: the top distance drops where they stop to be
    discords, the guided schedule misses there, and the next length's statistics
    and witnesses, queued ahead, are taken back."""
    import paddi_b200 as P
    missed = 0
    for seed in range(4):
        x, _ = datagen.palmad_series(n=30000, seed=seed, n_anom=3, min_len=70, max_len=80,
                                     kinds_cycle=("flat", "noise"))
        log = _check(x, 60, 90, r_policy=P.R_BOUND)
        per = {}
        for a in log:
            per[a["m"]] = per.get(a["m"], 0) + 1
        missed += sum(1 for m, c in per.items() if m > 60 and c > 1)
    assert missed > 0
