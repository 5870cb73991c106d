"""Copies by pinned chunks: whole arrays at the edges of a chunk and of the ring."""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("chunks", [1, 2, 3, 7])
def test_round_trip(chunks, extra):
    import torch

    from art import _device as D

    n = chunks * D._CHUNK // 8 + extra
    a = np.random.default_rng(chunks).integers(0, 2 ** 60, n).astype(np.float64)
    keep = a.copy()
    for src in (a, keep[::-1][::-1]):
        dev = D.upload_rows(src, torch.float64)
        if src is a:
            a[:] = 0.0  # the host array is free when the call returns
        np.testing.assert_array_equal(dev.cpu().numpy(), keep)
    ro = keep.view()
    ro.flags.writeable = False
    np.testing.assert_array_equal(D.upload_rows(ro, torch.float64).cpu().numpy(), keep)
    small = np.arange(n, dtype=np.int32)
    back = D.download(dev, torch.from_numpy(small).cuda())
    np.testing.assert_array_equal(back[0], keep)
    np.testing.assert_array_equal(back[1], small)
    assert all(b.flags.writeable for b in back)


def test_pack():
    from art import _device as D

    rng = np.random.default_rng(0)
    arrays = [np.arange(14, dtype=np.int32).reshape(7, 2), rng.normal(size=(7, 12)), rng.normal(size=(7, 4)),
              np.arange(7, dtype=np.int32)]
    for a, t in zip(arrays, D.pack(arrays)):
        np.testing.assert_array_equal(t.cpu().numpy(), a)
        assert t.cpu().numpy().dtype == a.dtype and t.data_ptr() % 256 == 0
