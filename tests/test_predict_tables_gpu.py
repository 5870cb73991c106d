"""Tree prediction: table strides, alignments, model kinds and staged copies.

The walk gives the same bits for every table stride and alignment; leaves are
the numpy walk's (no score here is within rounding of its threshold, by a
margin that the test checks), and a prediction of p products meets numpy's in
double double of 4 p eps of its absolute terms.
"""

import numpy as np
import pytest

from conftest import gpu_available
from oracle import ridge as O

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


def _tree(d, kind, rng, depth=5):
    n = 2 ** (depth + 1) - 1
    child = np.full((n, 2), -1, dtype=np.int32)
    inner = 2 ** depth - 1
    child[:inner, 0] = 2 * np.arange(inner) + 1
    child[:inner, 1] = 2 * np.arange(inner) + 2
    theta = rng.normal(size=(n, d + 1)) * np.r_[np.ones(d), 0.1]
    coef = rng.normal(size=(n, O.feature_count(d, kind)))
    return child, theta, coef, np.full(n, kind, dtype=np.int32)


def _wide(a, stride, lead):
    """Rows of `stride` doubles behind `lead` others; what lies between is NaN."""
    buf = np.full(lead + len(a) * stride, np.nan)
    buf[lead:].reshape(len(a), stride)[:, : a.shape[1]] = a
    return buf


def _call(tree, X, ts, cs, lead):
    import torch

    from art import _native as N

    child, theta, coef, kinds = tree
    d = X.shape[1]
    dev = [torch.from_numpy(a).cuda() for a in (child, _wide(theta, ts, lead), _wide(coef, cs, lead), kinds, X)]
    leaf = torch.empty(len(X), dtype=torch.int32, device="cuda")
    pred = torch.empty(len(X), dtype=torch.float64, device="cuda")
    p = [t.data_ptr() for t in dev]
    N.check(N.load_library().art_tree_predict(d, len(child), p[0], p[1] + 8 * lead, ts, p[2] + 8 * lead, cs, p[3],
                                              len(X), p[4], leaf.data_ptr(), pred.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream), "art_tree_predict")
    return leaf.cpu().numpy(), pred.cpu().numpy()


@pytest.mark.parametrize("d,kind", [(1, O.POLY2), (3, O.AFFINE), (4, O.POLY2_NOBIAS), (7, O.POLY1), (8, O.POLY2),
                                    (8, O.AFFINE), (9, O.POLY1_NOBIAS), (16, O.POLY2), (49, O.AFFINE), (64, O.AFFINE)])
def test_strides_kinds_and_the_numpy_walk(d, kind):
    rng = np.random.default_rng(10 * d + kind)
    X = rng.uniform(-1, 1, (777, d))
    tree = child, theta, coef, _ = _tree(d, kind, rng)
    leaf, pred = _call(tree, X, d + 1, coef.shape[1], 0)
    at, gap = np.zeros(len(X), dtype=int), np.inf
    while (child[at, 0] >= 0).any():
        s = (X * theta[at, :d]).sum(1) - theta[at, d]
        inner = child[at, 0] >= 0
        gap = min(gap, np.abs(s[inner]).min())
        at = np.where(inner, child[at, (s >= 0).astype(int)], at)
    assert gap > 1e-10
    np.testing.assert_array_equal(leaf, at)
    Phi = O.features(X, kind)
    terms = Phi * coef[at]
    bound = 4 * terms.shape[1] * np.finfo(float).eps * np.abs(terms).sum(1)
    assert (np.abs(pred - terms.sum(1)) <= bound).all()
    up = lambda v, m: -(-v // m) * m  # noqa: E731
    for ts, cs, lead in ((up(d + 1, 4), up(coef.shape[1], 4), 0), (up(d + 1, 2), up(coef.shape[1], 2), 2),
                         (up(d + 1, 4) + 4, up(coef.shape[1], 4) + 4, 4), (d + 2, coef.shape[1] + 3, 1)):
        again = _call(tree, X, ts, cs, lead)
        np.testing.assert_array_equal(again[0], leaf)
        np.testing.assert_array_equal(again[1], pred)
