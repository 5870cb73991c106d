"""The tensor-core ridge kernel, asked for by its threshold.

The mixed form's default sends no system to it, so its oracle tolerance, its
determinism and its statuses are checked with ``tensor_min_features=33``; the
refinement passes a system carries show that it was solved there.
"""

import numpy as np
import pytest

from conftest import gpu_available
from oracle import ridge as O
from test_ridge_gpu import _oracle_check, make_batch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


def _solve(wl, **kw):
    from art.models import solve_weighted_ridge_batched

    return solve_weighted_ridge_batched(wl.x, wl.y, wl.w, wl.row_offsets, wl.dims, wl.kinds, wl.ridge, x_offsets=wl.x_offsets,
                                        precision="mixed", max_features=wl.max_features, max_dim=wl.max_dim,
                                        tensor_min_features=33, **kw)


def _tensor(wl):
    return np.array([O.feature_count(int(d), int(k)) for d, k in zip(wl.dims, wl.kinds)]) >= 33


@pytest.mark.parametrize("factor", [False, True])
@pytest.mark.parametrize("seed,K,n_max", [(7, 96, 700), (8, 24, 5000)])
def test_matches_the_oracle(seed, K, n_max, factor):
    from art import _native as N

    wl = make_batch(K=K, seed=seed, n_max=n_max)
    out = _solve(wl, fp64_factor=factor)
    _oracle_check(wl, out)
    info, tensor = out.info.cpu().numpy(), _tensor(wl)
    there = (((info >> N.INFO_REFINE_SHIFT) & 255) > 0) | ((info & N.INFO_FP64_RESOLVE) != 0)
    solved = out.status.cpu().numpy() == 0
    assert tensor.any() and np.all(there[tensor & solved]) and not np.any(there[~tensor])


def test_is_deterministic_and_alone_equals_batched():
    wl = make_batch(K=40, seed=12)
    a, b = _solve(wl), _solve(wl)
    np.testing.assert_array_equal(np.nan_to_num(a.beta.cpu().numpy()), np.nan_to_num(b.beta.cpu().numpy()))
    for k in np.flatnonzero(_tensor(wl))[:4]:
        sub = wl.subset([k])
        c = _solve(sub)
        p = O.feature_count(int(wl.dims[k]), int(wl.kinds[k]))
        np.testing.assert_array_equal(c.beta.cpu().numpy()[0, :p], a.beta.cpu().numpy()[k, :p])


@pytest.mark.parametrize("kind,d", [(2, 8), (2, 16)])
def test_bad_inputs_and_empty_systems(kind, d):
    from art.models import kind_feature_count, solve_weighted_ridge_batched

    rng = np.random.default_rng(9)
    p = kind_feature_count(d, kind)
    n = [0, 400, 400, 400, 400, 401]
    ro = np.concatenate([[0], np.cumsum(n)])
    X, y, w = rng.uniform(-1, 1, (ro[-1], d)), rng.normal(size=ro[-1]), rng.uniform(0.1, 1.0, ro[-1])
    X[ro[1] + 399, d - 1] = np.inf
    w[ro[2] + 200] = -2.0
    y[ro[3]] = np.nan
    w[ro[4] + 1] = np.inf
    out = solve_weighted_ridge_batched(X.reshape(-1), y, w, ro, [d] * 6, [kind] * 6, [1e-4] * 6, precision="mixed",
                                       max_features=p, max_dim=d, tensor_min_features=33)
    assert out.status.cpu().numpy().tolist() == [1, -2, -1, -2, -1, 0]
    assert np.isfinite(out.beta.cpu().numpy()[5]).all() and np.isnan(out.beta.cpu().numpy()[1:5]).all()
