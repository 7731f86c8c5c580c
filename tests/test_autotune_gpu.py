"""The autotuner on a series too short for its segment lengths to differ.

Phase 1 splits a segment where a series is too short to fill the GPU, so 256,
384 and 512 rows are then one program.  It is timed once: the three entries
are equal, and the first of them is taken.
"""
import pytest

import paddi_b200 as P
from paddi_b200 import datagen

pytestmark = pytest.mark.gpu


def test_equal_programs_are_timed_once():
    x, _ = datagen.palmad_series(n=1 << 14, seed=2, n_anom=4, min_len=32, max_len=96,
                                 kinds_cycle=("noise",))
    with P.Context(device=0, r_policy=P.R_BOUND) as ctx:
        got = ctx.autotune(x, 48, 60)
    ms = got["probe_ms"]
    assert len(ms) == 18 and min(ms.values()) > 0
    for tr in (0, 64):
        for ch in (8, 12, 16):
            assert ms[tr, 256, ch] == ms[tr, 384, ch] == ms[tr, 512, ch]
    assert got["segment_len"] == 256
