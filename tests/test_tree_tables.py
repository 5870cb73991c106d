"""Widths of the flat tables a tree is walked from on the device."""

import numpy as np
import pytest


@pytest.mark.parametrize("columns", list(range(1, 40)) + [45, 65, 153])
def test_rows_are_padded_by_a_third_at_most(columns):
    from art.tree import _sector_rows

    a = _sector_rows(5, columns)
    whole = a.base
    assert a.shape == (5, columns) and whole.shape[0] == 5 and whole.flags.c_contiguous
    assert columns <= whole.shape[1] and 3 * whole.shape[1] <= 4 * columns
    if columns >= 9:  # from here on whole sectors always fit that
        assert whole.shape[1] % 4 == 0
    a[:] = np.arange(columns)
    assert np.array_equal(whole[:, :columns], a) and not whole[:, columns:].any()
