"""Residual sums of rows at the ends of the number range.

The products of a quadratic model are formed before they meet their
coefficients, as numpy's features are: a coefficient times one input may
overflow where the products do not.  Where an input is not finite, neither the
zero padding nor another feature may change what numpy gives.
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("d,kind", [(2, 2), (3, 4), (8, 2), (11, 2), (16, 4), (5, 0), (7, 1), (6, 3)])
def test_one_row_at_a_time(d, kind):
    from art.models import kind_feature_count, segment_residuals

    inf, nan = np.inf, np.nan
    p = kind_feature_count(d, kind)
    rng = np.random.default_rng(d)
    rows = []
    for lo, hi, c in [(0.0, 1e200, 1e200), (1e-200, 1e200, 1e150), (1e-160, 1e180, 1e140), (inf, 1.0, 1.0), (inf, 0.0, 1.0),
                      (-inf, -2.0, 0.0), (nan, 1.0, 1.0), (1e200, 1e200, 1e-200), (inf, inf, 1.0)]:
        x, b = np.zeros(d), np.zeros(p)
        x[0], x[d - 1] = lo, hi
        b[-1] = 0.25
        i, j = np.triu_indices(d)
        first = p - len(i) if kind in (2, 4) else 0
        at = first + int(np.flatnonzero((i == 0) & (j == d - 1))[0]) if kind in (2, 4) else rng.integers(0, p)
        b[at] = c
        rows.append((x, b))
    X, beta = np.array([r[0] for r in rows]), np.array([r[1] for r in rows])
    K = len(rows)
    y = np.full(K, 0.5)
    sse, _ = segment_residuals(X.reshape(-1), y, np.arange(K + 1), [d] * K, [kind] * K, beta)
    one = np.ones((K, 1))
    i, j = np.triu_indices(d)
    with np.errstate(all="ignore"):
        phi = {0: lambda: np.hstack([X, one]), 1: lambda: np.hstack([one, X]), 2: lambda: np.hstack([one, X, X[:, i] * X[:, j]]),
               3: lambda: X, 4: lambda: np.hstack([X, X[:, i] * X[:, j]])}[kind]()
        pred = np.zeros(K)
        for f in range(p):  # in feature order
            pred = pred + phi[:, f] * beta[:, f]
        want = (y - pred) ** 2
    np.testing.assert_allclose(sse.cpu().numpy(), want, rtol=1e-12)
