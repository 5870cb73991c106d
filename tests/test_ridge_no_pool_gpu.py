"""Large systems without room to split them: a whole CTA's, with the split's bits.

A batch whose workspace holds the lists alone, one with a part of the pool, and
one too long to be split (16,385 systems) must give the results of the split
batch to the bit, bad inputs included.
"""

import ctypes as C

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

AFFINE, POLY1, POLY2, POLY1_NOBIAS, POLY2_NOBIAS = range(5)


def _solve(X, y, w, ro, d, kind, p, share):
    """Results with a workspace of the lists and `share` of the rest; None: no workspace."""
    import torch

    from art import _native as N
    from art._device import ptr, stream_handle

    K = len(ro) - 1
    lib = N.load_library()
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    keep = [t(X.reshape(-1)), t(y), None if w is None else t(w), t(np.asarray(ro, np.int64)), t(np.asarray(ro[:-1], np.int64) * d),
            t(np.full(K, d, np.int32)), t(np.full(K, kind, np.int32)), t(np.full(K, 1e-6))]
    x, yt, wt, rot, xo, dt, kt, rt = keep
    seg = N.ArtSegments(K, ptr(rot), ptr(xo), ptr(dt), ptr(kt))
    prob = N.ArtRidgeProblem(seg, ptr(x), ptr(yt), ptr(wt), ptr(rt), 0.0, 0, 0, 1e-12, p, d, 0, 0)
    beta = torch.full((K, p), float("nan"), dtype=torch.float64, device="cuda")
    lam, status = torch.empty(K, dtype=torch.float64, device="cuda"), torch.empty(K, dtype=torch.int32, device="cuda")
    res = N.ArtRidgeResult(ptr(beta), p, ptr(lam), None, ptr(status), None)
    if share is None:
        N.check(lib.art_ridge_batched_noalloc(C.byref(prob), C.byref(res), stream_handle()), "noalloc")
    else:
        full, lists = lib.art_ridge_workspace_size(K, p), lib.art_ridge_workspace_size(1 << 20, p) // (1 << 20) * K + 8192
        ws = torch.empty(int(lists + share * max(full - lists, 0)), dtype=torch.uint8, device="cuda")
        N.check(lib.art_ridge_batched(C.byref(prob), C.byref(res), ptr(ws), ws.numel(), stream_handle()), "batched")
    return beta.cpu().numpy(), lam.cpu().numpy(), status.cpu().numpy()


@pytest.mark.parametrize("kind,d", [(AFFINE, 23), (POLY2, 6), (AFFINE, 32), (POLY2_NOBIAS, 8), (POLY1_NOBIAS, 47), (AFFINE, 9)])
@pytest.mark.parametrize("bad", [None, "x", "weight"])
def test_without_a_pool(kind, d, bad):
    from art.models import kind_feature_count

    rng = np.random.default_rng(d + kind)
    p = kind_feature_count(d, kind)
    ns = [257, 70001, 300, 1025, 20000, 512, 3001, 64, 1024, 5000]
    ro = np.concatenate([[0], np.cumsum(ns)])
    X, y, w = rng.uniform(-1.0, 1.0, (ro[-1], d)), rng.normal(size=ro[-1]), rng.uniform(0.0, 1.0, ro[-1])
    if bad == "x":
        X[ro[1] + 60000, d - 1] = np.nan
    elif bad == "weight":
        w[ro[4] + 12345] = -1.0
    split = _solve(X, y, w, ro, d, kind, p, 1.0)
    failed = {None: [], "x": [1], "weight": [4]}[bad]
    want = np.zeros(len(ns), np.int32)
    want[failed] = -2 if bad == "x" else -1
    np.testing.assert_array_equal(split[2], want)
    for share in (None, 0.0, 0.02):
        for got, ref in zip(_solve(X, y, w, ro, d, kind, p, share), split):
            np.testing.assert_array_equal(got, ref, err_msg=str(share))
    many = 16385 - len(ns)
    ro2 = np.concatenate([ro, ro[-1] + np.arange(1, many + 1)])
    long = _solve(np.concatenate([X, rng.uniform(-1.0, 1.0, (many, d))]), np.concatenate([y, rng.normal(size=many)]),
                  np.concatenate([w, np.ones(many)]), ro2, d, kind, p, 1.0)
    for got, ref in zip(long, split):
        np.testing.assert_array_equal(got[: len(ns)], ref)
