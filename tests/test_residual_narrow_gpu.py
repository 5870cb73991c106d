"""Residual sums of levels with few features: their first launch is a kernel of its
own, chosen by the stride of the coefficients.  Its sums are the general
kernel's to the bit, so that a node's result does not depend on its level."""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

# below, at and above a warp's tile, a CTA's, a node's ranges and the joint sizes
ROWS = [0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 513, 1023, 1024, 1025, 2047, 2048, 2049, 3000, 8191, 8193, 20000]


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("count", [33, 700, 3500])
@pytest.mark.parametrize("d,kind", [(1, 0), (5, 0), (5, 1), (1, 2), (2, 2), (6, 3), (1, 4), (2, 4)])
def test_narrow_sums_are_the_general_ones(d, kind, count, odd):
    import torch

    from art.models import kind_feature_count, segment_residuals

    p = kind_feature_count(d, kind)
    assert p <= 6
    rng = np.random.default_rng(count + d)
    ns = np.concatenate([ROWS, rng.integers(0, 400, count - len(ROWS))]).astype(np.int64)
    rng.shuffle(ns)
    ro = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    n = int(ro[-1])
    X, y = rng.normal(size=(n, d)), rng.normal(size=n)
    beta = np.zeros((count, 8))
    beta[:, :p] = rng.normal(size=(count, p))
    if odd:
        at = rng.integers(0, n, 40)
        X[at, rng.integers(0, d, 40)] = rng.choice([np.inf, -np.inf, np.nan, 1e200, 1e-200], 40)
        beta[rng.integers(0, count, 5), rng.integers(0, p, 5)] = [np.inf, np.nan, 0.0, 1e200, 1e-200]
    args = (X.reshape(-1), y, ro, [d] * count, [kind] * count)
    narrow = segment_residuals(*args, np.ascontiguousarray(beta[:, :p]))
    general = segment_residuals(*args, beta)
    for a, b in zip(narrow, general):
        a, b = a.cpu(), b.cpu()
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        assert torch.equal(a.nan_to_num(0.0, 1.0, -1.0), b.nan_to_num(0.0, 1.0, -1.0))
    if odd:
        return
    i, j = np.triu_indices(d)
    one, cross = np.ones((n, 1)), X[:, i] * X[:, j]
    phi = {0: [X, one], 1: [one, X], 2: [one, X, cross], 3: [X], 4: [X, cross]}[kind]
    err = y - np.sum(np.hstack(phi) * np.repeat(beta[:, :p], ns, axis=0), axis=1)
    for got, v in ((narrow[0], err), (narrow[1], y)):
        want = np.array([np.dot(v[a:b], v[a:b]) for a, b in zip(ro[:-1], ro[1:])])
        # positive terms: the sum's relative error is below rows x 2^-53, the
        # error of a residual (p + 2 roundings of its terms) is far below 1e-13
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-10, atol=1e-24)
