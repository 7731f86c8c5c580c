"""Room for attempt rows in the Python binding (CPU only).

The library takes the number of rows as an unsigned 32-bit value: what does
not fit in that, a negative number above all, must be refused before the call,
or the library would write past the rows.
"""
import numpy as np
import pytest

import paddi_b200 as P


@pytest.mark.parametrize("cap", [-1, -100000, 2 ** 32])
def test_row_counts_outside_the_librarys_range_are_refused(cap):
    with pytest.raises(ValueError):
        P._LogRows(cap)


def test_no_rows_are_a_valid_choice():
    rows = P._LogRows(0)
    rows.n.value = 7  # attempts made, none recorded
    assert rows.dicts() == []


def test_rows_come_back_as_the_struct_has_them():
    rows = P._LogRows(3)
    a = P._Log.from_buffer(rows.buf[1:2])
    a.m, a.r, a.n_cand, a.top.ind, a.top.dist, a.n_fragile = 77, 0.5, 1 << 40, -3, 2.25, 9
    rows.n.value = 2
    got = rows.dicts()[1]
    assert got == a.as_dict() and list(got) == list(a.as_dict())
    assert (got["m"], got["r"], got["n_cand"], got["top_ind"], got["top_dist"],
            got["n_fragile"]) == (77, 0.5, 1 << 40, -3, 2.25, 9)
    assert all(type(v) in (int, float) for v in got.values())
    assert np.dtype(P._Log).itemsize == rows.buf.itemsize
