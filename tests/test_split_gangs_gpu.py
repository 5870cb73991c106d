"""Warp form of the split search: gang sizes, block counts, row layouts.

With one restart a node is searched by a warp (below 1,023 rows), a CTA or a
cluster (from 4,095 rows); models of more than 23 features keep one side per
warp and always take a gang.  Every size and width must meet the oracle's
search (theta at 1e-9 relative, as the other split tests) and give the same
bits alone, in a batch, and in a batch whose widest model is wider.
"""

import numpy as np
import pytest

from conftest import gpu_available
from oracle import ridge as O
from oracle import split as S
from test_split_gpu import splitter_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

NS = [150, 1022, 1023, 4094, 4095, 9001, 20011]


def _nodes(d, seed, ns):
    rng = np.random.default_rng(seed)
    Xs = [rng.uniform(-1, 1, (n, d)) for n in ns]
    u = rng.normal(size=d)
    ys = [np.sin(2 * X[:, 0]) + np.tanh(4 * (X @ (u / np.linalg.norm(u)))) + 0.3 * (X ** 2).sum(1) / d for X in Xs]
    return Xs, ys


def _call(s, Xs, ys, dims, kinds, T, lam, th0, lead=0, **kw):
    from art.splitters import split_level

    n = np.array([len(y) for y in ys])
    ro = np.concatenate([[0], np.cumsum(n)])
    xo = np.concatenate([[0], np.cumsum(n * np.asarray(dims))])[:-1] + lead
    x = np.concatenate([np.zeros(lead)] + [X.reshape(-1) for X in Xs])
    return split_level(s, x, np.concatenate(ys), ro, dims, kinds, T, lam, x_offsets=xo, theta0=th0,
                       parent_loss=[1.0] * len(ys), **kw)


# one to six 8-column blocks; last blocks of up to four columns and more; odd,
# even and power-of-two row lengths; a lead element takes the 8-byte copies
@pytest.mark.parametrize("kind,d,lead", [(O.AFFINE, 1, 0), (O.POLY2, 2, 0), (O.AFFINE, 5, 0), (O.AFFINE, 8, 1),
                                         (O.AFFINE, 16, 0), (O.POLY2, 5, 0), (O.AFFINE, 22, 0), (O.AFFINE, 27, 0),
                                         (O.AFFINE, 32, 0), (O.POLY2, 8, 0), (O.AFFINE, 46, 0), (O.AFFINE, 40, 1)])
def test_gang_sizes_match_the_oracle(kind, d, lead):
    Xs, ys = _nodes(d, 10 * d + kind, NS)
    init = np.random.default_rng(3)
    th0 = np.array([[S.initialize_theta(X, init)] for X in Xs])
    T, lam, iters = 0.2, 1e-6, 6
    s = splitter_for(kind, T, lam, 1, iters, {"min_side_points": 1})
    K = len(NS)
    res = _call(s, Xs, ys, [d] * K, [kind] * K, T, lam, th0, lead, traces=True)
    get = lambda r, name: getattr(r, name).cpu().numpy()  # noqa: E731
    p = S.Params(max_iters=iters, n_restarts=1, min_side_points=1)
    features = 1 + d if kind == O.AFFINE else 1 + d + d * (d + 1) // 2
    for k in range(K):
        if NS[k] < 4 * features:
            continue  # sides of fewer rows than features: the fits are not determined to 1e-9
        opt = S.optimize(Xs[k], ys[k], th0[k][0], T, kind, lam, p)
        try:
            hard = S.hard_result(Xs[k], ys[k], opt["theta"], kind, lam, 1.0, p, True)
        except ValueError:  # a side below the minimum
            assert get(res, "failure")[k] == 2
            continue
        assert get(res, "failure")[k] == 0
        np.testing.assert_allclose(get(res, "theta")[k], np.r_[hard["w"], hard["z"]], rtol=1e-9, atol=1e-10)
        assert get(res, "n_iters")[k] == opt["n_iters"] and get(res, "n_right")[k] == hard["n_right"]
        np.testing.assert_allclose(get(res, "trace_loss")[k, 0, : opt["n_iters"] + 1], opt["losses"], rtol=1e-9)
        np.testing.assert_array_equal(get(res, "trace_backtracks")[k, 0, : opt["n_iters"]], opt["backtracks"])
        np.testing.assert_allclose(get(res, "loss")[k], hard["loss"], rtol=1e-9)
    # alone, and beside a wider model
    names = ("theta", "loss", "n_right", "n_iters", "beta", "final_alpha")
    wide_X, wide_y = _nodes(46, 5, [700])
    for k in range(K):
        one = _call(s, Xs[k:k + 1], ys[k:k + 1], [d], [kind], T, lam, th0[k:k + 1])
        for name in names:
            np.testing.assert_array_equal(get(one, name)[0], get(res, name)[k], err_msg=f"{name} {k}")
    if kind == O.AFFINE and d < 46:
        th = np.zeros((K + 1, 1, 47))
        th[:K, :, : d + 1] = th0
        th[K, 0] = S.initialize_theta(wide_X[0], init)
        both = _call(s, Xs + wide_X, ys + wide_y, [d] * K + [46], [kind] * (K + 1), T, lam, th)
        for k in range(K):
            np.testing.assert_array_equal(get(both, "theta")[k, : d + 1], get(res, "theta")[k])
            np.testing.assert_array_equal(get(both, "loss")[k], get(res, "loss")[k])


@pytest.mark.parametrize("n", [800, 3000, 12000])
@pytest.mark.parametrize("d,kind", [(4, O.POLY2), (32, O.AFFINE)])
def test_gang_long_line_searches_and_fallback(n, d, kind):
    """More backtracks than candidates of a pass, failed attempts, min-side
    failure and fallback, and the geometry-only result of every gang."""
    Xs, ys = _nodes(d, 77, [n])
    th0 = np.array([[S.initialize_theta(Xs[0], np.random.default_rng(1))]])
    T, lam = 0.05, 1e-6
    for extra in ({"alpha0": 1e3, "min_side_points": 1}, {"alpha0": 1e3, "max_backtracks": 1, "min_side_points": 1},
                  {"min_side_points": n // 2 - 1, "min_side_fallback": True},
                  {"adaptive_alpha": False, "alpha0": 50.0, "max_backtracks": 2, "min_side_points": 1}):
        s = splitter_for(kind, T, lam, 1, 5, extra)
        res = _call(s, Xs, ys, [d], [kind], T, lam, th0, traces=True)
        p = S.Params(max_iters=5, n_restarts=1, **extra)
        opt = S.optimize(Xs[0], ys[0], th0[0][0], T, kind, lam, p)
        from art import _native as N

        assert N.STOP_REASONS[int(res.stop_reason[0])] == opt["stop_reason"]
        assert int(res.n_iters[0]) == opt["n_iters"]
        np.testing.assert_array_equal(res.trace_backtracks.cpu().numpy()[0, 0, : opt["n_iters"]], opt["backtracks"])
        np.testing.assert_allclose(float(res.final_alpha[0]), opt["final_alpha"], rtol=1e-12)
        geo = _call(s, Xs, ys, [d], [kind], T, lam, th0, hard_refit=False)
        assert int(geo.failure[0]) == int(res.failure[0])
        if int(res.failure[0]) == 0:
            np.testing.assert_array_equal(geo.theta.cpu().numpy(), res.theta.cpu().numpy())
            assert int(geo.n_right[0]) == int(res.n_right[0])
