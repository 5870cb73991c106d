"""Workspace sizes of the batched ridge, from the built library (no GPU)."""

import pytest


@pytest.mark.parametrize("count", [1, 2, 100, 300, 16384, 16385, 100000])
@pytest.mark.parametrize("features", [1, 9, 45, 47, 153])
def test_size_by_rows(lib, count, features):
    full = lib.art_ridge_workspace_size(count, features)
    sizes = [lib.art_ridge_workspace_size_rows(count, features, n) for n in (0, 256, 10_000, 1_000_000, 10**12)]
    assert sizes == sorted(sizes) and sizes[-1] == full and sizes[0] <= full
    if count > 16384:  # never split
        assert sizes[0] == full
        return
    # every unit Gram of the worst batch of that many rows has room: systems of 257
    # rows (two units each), or units of 256 rows in long systems
    pa = min(features, 47) + 1
    for rows, size in ((10_000, sizes[2]), (1_000_000, sizes[3])):
        units = max(min(count, rows // 257) * 2, min(count * 256, rows // 256))
        assert size == full or size - sizes[0] >= units * pa * (pa + 1) // 2 * 8
    # a hundred small systems do not ask for the 256 MiB that a hundred large ones may use
    if count == 100 and features == 45:
        assert full > 200 << 20 and lib.art_ridge_workspace_size_rows(100, 45, 100_000) < 10 << 20
