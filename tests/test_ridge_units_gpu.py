"""FP64 MMA ridge kernel: unit and tile boundaries, every block count, split systems.

A system's Gram is the sum of fixed units of its rows, whoever forms them, so a
system split over many warps (a few large systems on the device) must equal,
bit for bit, the same system formed by one warp (a batch of many systems, or no
scratch to split into), and both must solve the normal equations to FP64
accuracy.  The tolerance is 1e-14 times the 2-norm condition number of the
regularised Gram, at least 1e-12: two FP64 solvers with different summation
orders agree to about that number times the unit roundoff.
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

AFFINE, POLY1, POLY2, POLY1_NOBIAS, POLY2_NOBIAS = range(5)


def _phi(X, kind):
    one = np.ones((X.shape[0], 1))
    i, j = np.triu_indices(X.shape[1])
    return {AFFINE: lambda: np.hstack([X, one]), POLY1: lambda: np.hstack([one, X]),
            POLY2: lambda: np.hstack([one, X, X[:, i] * X[:, j]]), POLY1_NOBIAS: lambda: X,
            POLY2_NOBIAS: lambda: np.hstack([X, X[:, i] * X[:, j]])}[kind]()


# one to six 8-column blocks, even and odd row lengths (16- and 8-byte copies),
# tiles of 32 rows and fewer
@pytest.mark.parametrize("kind,d", [(AFFINE, 1), (POLY2, 2), (AFFINE, 7), (POLY2, 4), (POLY1, 15), (AFFINE, 16),
                                    (POLY1_NOBIAS, 23), (POLY2_NOBIAS, 6), (AFFINE, 32), (AFFINE, 39),
                                    (POLY2, 8), (POLY1_NOBIAS, 47)])
@pytest.mark.parametrize("weighted", [True, False])
def test_units_and_tiles(kind, d, weighted):
    from art.models import kind_feature_count, solve_weighted_ridge_batched

    rng = np.random.default_rng(100 * kind + d)
    p = kind_feature_count(d, kind)
    ns = [max(p, 31) + 4, 255, 256, 257, 511, 2049, 70001]
    ro = np.concatenate([[0], np.cumsum(ns)])
    X = rng.uniform(-1.0, 1.0, (ro[-1], d))
    y = rng.normal(size=ro[-1])
    w = rng.uniform(0.0, 1.0, ro[-1]) if weighted else None
    kw = dict(weight_floor=0.0, max_features=p, max_dim=d)
    K = len(ns)
    out = solve_weighted_ridge_batched(X.reshape(-1), y, w, ro, [d] * K, [kind] * K, [1e-6] * K, **kw)
    beta, lam = out.beta.cpu().numpy(), out.ridge_effective.cpu().numpy()
    assert np.all(out.status.cpu().numpy() == 0)
    for k in range(K):
        rows = slice(ro[k], ro[k + 1])
        phi = _phi(X[rows], kind)
        q = np.ones(ns[k]) if w is None else w[rows]
        G = phi.T @ (phi * q[:, None])
        lk = 1e-6 * np.trace(G) / p
        A = G + lk * np.eye(p)
        ref = np.linalg.solve(A, phi.T @ (q * y[rows]))
        assert abs(lam[k] - lk) <= 1e-12 * lk
        tol = max(1e-12, 1e-14 * np.linalg.cond(A))
        assert np.linalg.norm(beta[k, :p] - ref) <= tol * np.linalg.norm(ref), (k, ns[k])
    # the last two systems alone (split), and every system in a batch too large
    # to split any (16,385 systems, most of them tiny)
    for k in (K - 2, K - 1):
        rows = slice(ro[k], ro[k + 1])
        one = solve_weighted_ridge_batched(X[rows].reshape(-1), y[rows], None if w is None else w[rows], [0, ns[k]],
                                           [d], [kind], [1e-6], **kw)
        np.testing.assert_array_equal(one.beta.cpu().numpy()[0, :p], beta[k, :p])
    many = 16385 - K
    ro2 = np.concatenate([ro, ro[-1] + np.arange(1, many + 1)])
    X2 = np.concatenate([X, rng.uniform(-1.0, 1.0, (many, d))])
    y2 = np.concatenate([y, rng.normal(size=many)])
    w2 = None if w is None else np.concatenate([w, np.ones(many)])
    big = solve_weighted_ridge_batched(X2.reshape(-1), y2, w2, ro2, [d] * (K + many), [kind] * (K + many),
                                       [1e-6] * (K + many), **kw)
    np.testing.assert_array_equal(big.beta.cpu().numpy()[:K, :p], beta[:, :p])


@pytest.mark.parametrize("bad", ["x", "y", "inf", "weight", "nan_weight"])
def test_bad_input_in_a_split_system(bad):
    """A non-finite or negative input anywhere in a split system fails that system only."""

    from art.models import solve_weighted_ridge_batched

    rng = np.random.default_rng(3)
    d, ns = 8, [40000, 30011]
    ro = np.concatenate([[0], np.cumsum(ns)])
    X, y, w = rng.uniform(-1, 1, (ro[-1], d)), rng.normal(size=ro[-1]), rng.uniform(0, 1, ro[-1])
    at = 33333
    if bad == "x":
        X[at, 3] = np.nan
        w[at] = 0.0
    elif bad == "inf":
        X[at, 0] = -np.inf
    elif bad == "y":
        y[at] = np.inf
        w[at] = 0.0
    elif bad == "weight":
        w[at] = -1e-300
    else:
        w[at] = np.nan
    out = solve_weighted_ridge_batched(X.reshape(-1), y, w, ro, [d] * 2, [POLY2] * 2, [1e-6] * 2, weight_floor=0.0,
                                       max_features=45, max_dim=d)
    st = out.status.cpu().numpy()
    assert st[0] == (-1 if "weight" in bad else -2) and st[1] == 0
    assert np.all(np.isnan(out.beta.cpu().numpy()[0])) and np.all(np.isfinite(out.beta.cpu().numpy()[1]))


# the wide kernel: group rows of one to five, several warps a group, the widest
# model (its right-hand side apart), rows of 16- and 8-byte copies, long and
# short chunks (d > 64 takes chunks of 16 rows)
@pytest.mark.parametrize("kind,d", [(AFFINE, 47), (POLY2, 9), (AFFINE, 63), (POLY1_NOBIAS, 64), (AFFINE, 96), (POLY1_NOBIAS, 97),
                                    (POLY2, 14), (POLY1_NOBIAS, 127), (POLY1_NOBIAS, 128), (POLY2, 16), (AFFINE, 158),
                                    (POLY1_NOBIAS, 160)])
@pytest.mark.parametrize("weighted", [True, False])
def test_wide_systems(kind, d, weighted):
    from art.models import kind_feature_count, solve_weighted_ridge_batched

    rng = np.random.default_rng(7 * d + kind)
    p = kind_feature_count(d, kind)
    ns = [0, 3, p + 5, 2 * p + 1, 1024, 1091]
    ro = np.concatenate([[0], np.cumsum(ns)])
    X = rng.uniform(-1.0, 1.0, (ro[-1], d))
    y = rng.normal(size=ro[-1])
    w = rng.uniform(0.0, 1.0, ro[-1]) if weighted else None
    K = len(ns)
    out = solve_weighted_ridge_batched(X.reshape(-1), y, w, ro, [d] * K, [kind] * K, [1e-4] * K, weight_floor=0.0,
                                       max_features=p, max_dim=d, condition=True)
    beta, st = out.beta.cpu().numpy(), out.status.cpu().numpy()
    assert st[0] == 1 and np.all(st[1:] == 0)
    for k in range(1, K):
        rows = slice(ro[k], ro[k + 1])
        phi = _phi(X[rows], kind)
        q = np.ones(ns[k]) if w is None else w[rows]
        G = phi.T @ (phi * q[:, None])
        A = G + 1e-4 * np.trace(G) / p * np.eye(p)
        ref = np.linalg.solve(A, phi.T @ (q * y[rows]))
        cond = np.linalg.cond(A)
        assert np.linalg.norm(beta[k, :p] - ref) <= max(1e-12, 1e-14 * cond) * np.linalg.norm(ref), (k, ns[k])
        # the estimate is of the 1-norm condition number's square root, from below, rarely by more than 3
        est = float(out.cond_estimate[k])
        c1 = np.sqrt(np.linalg.cond(A, 1))
        assert c1 / 3 <= est <= c1 * (1 + 1e-6)


@pytest.mark.parametrize("bad", ["x", "y", "weight"])
def test_bad_input_in_a_wide_system(bad):
    from art.models import solve_weighted_ridge_batched

    rng = np.random.default_rng(4)
    d, ns = 16, [700, 500]
    ro = np.concatenate([[0], np.cumsum(ns)])
    X, y, w = rng.uniform(-1, 1, (ro[-1], d)), rng.normal(size=ro[-1]), rng.uniform(0, 1, ro[-1])
    if bad == "x":
        X[690, 15] = np.inf
        w[690] = 0.0
    elif bad == "y":
        y[3] = np.nan
    else:
        w[699] = -1.0
    for precision in ("fp64", "mixed"):
        out = solve_weighted_ridge_batched(X.reshape(-1), y, w, ro, [d] * 2, [POLY2] * 2, [1e-6] * 2, precision=precision,
                                           max_features=153, max_dim=d)
        st = out.status.cpu().numpy()
        assert st[0] == (-1 if bad == "weight" else -2) and st[1] == 0
