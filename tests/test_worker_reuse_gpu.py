"""Worker contexts kept between batched calls: every call must see the options,
the model and the series of that call only."""
import numpy as np
import pytest

from paddi_b200 import datagen

pytestmark = pytest.mark.gpu


def _series(lens, seed):
    return [datagen.random_walk_sine(n, np.random.default_rng(seed + k)).astype(np.float32)
            for k, n in enumerate(lens)]


def test_repeated_batches_equal_single_runs():
    import paddi_b200 as P
    with P.Context(device=0, r_policy=P.R_BOUND) as ctx:
        # growing and shrinking batches and stream counts on one context
        for lens, lo, hi, streams in (([3000, 9000], 20, 30, 2), ([2000] * 5, 40, 44, 4),
                                      ([30000, 1500, 700], 25, 35, 1), ([9000, 3000], 20, 30, 3)):
            xs = _series(lens, sum(lens))
            got, att = ctx.palmad_batched(xs, lo, hi, streams=streams)
            for x, d, a in zip(xs, got, att):
                want, log = P.Context(device=0, r_policy=P.R_BOUND).palmad(x, lo, hi)
                assert [(q.ind, q.dist) for q in d] == [(q.ind, q.dist) for q in want]
                assert a == len(log)


def test_workers_follow_the_model_and_survive_a_failed_batch():
    import paddi_b200 as P
    xs = _series([6000, 4000], 3)
    with P.Context(device=0, r_policy=P.R_LEARNED, iter_cap=200) as ctx:
        first, a1 = ctx.palmad_batched(xs, 30, 40, streams=2)
        ctx.set_model(P.init_params(5))
        with P.Context(device=0, r_policy=P.R_LEARNED, model=P.init_params(5)) as other:
            _, a2 = ctx.palmad_batched(xs, 30, 40, streams=2)
            _, a3 = other.palmad_batched(xs, 30, 40, streams=2)
        assert a2 == a3
        with pytest.raises(P.PaddiError):
            ctx.palmad_batched([xs[0], xs[1][:50]], 30, 40, streams=2)  # too short: refused
        again, _ = ctx.palmad_batched(xs, 30, 40, streams=2)
    assert [[(q.ind, q.dist) for q in d] for d in again] == \
        [[(q.ind, q.dist) for q in d] for d in first]
