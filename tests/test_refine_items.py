"""The refine's work items (CPU only).

The CTAs of a refine wait for one another between rounds with a limit of
about 4e9 clock cycles, so no item may come near it: at the lowest rates that
the kernels reach (38 FMA a cycle and CTA for the FP32 refine, 4e4 cycles for
a tile of 2048 windows on the tensor cores) an item stays below a tenth of
the limit for every length and series length, up to four million candidates
(beyond, the item counter's 31 bits decide; a round then takes days).  Small
rounds are split as the number of CTAs alone would have it.
"""
import ctypes as C

import pytest

import paddi_b200 as P

LIMIT = 4e9


def _item(kernel, m, cand, windows, ctas):
    n = C.c_int64(0)
    span = P.lib().paddi_debug_refine_item(kernel, m, cand, windows, ctas, C.byref(n))
    return span, n.value


@pytest.mark.parametrize("windows", [4096, 99999, 1 << 22, 1 << 25, (1 << 29) + 77, (1 << 31) - 5000])
@pytest.mark.parametrize("cand", [1, 9, 5000, 300000, 1 << 22])
@pytest.mark.parametrize("m", [3, 300, 729, 730, 1024])
def test_items_stay_far_below_the_wait_limit(m, cand, windows):
    for kernel, ctas in ((P.DIST_FP32, 296), (P.DIST_SPLIT_FP16, 148)):
        span, n = _item(kernel, m, cand, windows, ctas)
        assert span * n >= windows and (n - 1) * span < windows + 2048 * n
        fp32 = kernel == P.DIST_FP32 or m > 729
        cycles = 8.0 * span * m / 38 if fp32 else span / 2048 * 4e4
        assert cycles < LIMIT / 10, (kernel, span, n)
        tiles = -(-cand // 8)
        assert tiles * n < 2 ** 31


@pytest.mark.parametrize("windows,cand", [(2048, 1), (65536, 100), (131072, 3000), (1 << 21, 40)])
def test_small_rounds_are_split_by_the_ctas(windows, cand):
    span, n = _item(P.DIST_FP32, 400, cand, windows, 296)
    tiles = -(-cand // 8)
    want = max(1, min((592 + tiles - 1) // tiles, windows // 1024))
    assert n == want and span == -(-(-(-windows // want)) // 1024) * 1024
    span, n = _item(P.DIST_SPLIT_FP16, 300, cand, windows, 148)
    want = max(1, min(windows // 2048, 148 // (-(-cand // 16))))
    assert n == want and span == -(-(-(-windows // want)) // 2048) * 2048


def test_arguments_outside_the_ranges_are_refused():
    for a in ((1, 2, 5, 5, 5), (1, 1025, 5, 5, 5), (1, 64, 0, 5, 5), (1, 64, 5, 0, 5),
              (1, 64, 5, 5, 0), (1, 64, 5, 2 ** 32 - 1, 5)):
        assert P.lib().paddi_debug_refine_item(*a, None) == -1
