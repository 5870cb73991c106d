"""The CTA form of the split search with one and two restarts a node.

Levels of at most two restarts take the warp form where their declared widest
node fits it (46 inputs, 47 features); a declared width of 50 inputs keeps them on
the CTA form, whose gangs span CTAs through global scratch and whose rows stream
through a ring.  Tolerances as in test_split_gpu.py.
"""

import ast

import numpy as np
import pytest

from conftest import GOLDEN, gpu_available
from oracle import ridge as O
from oracle import split as S
from test_split_gpu import splitter_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]
SG = np.load(GOLDEN / "split_golden.npz")
WIDE = dict(max_dim=50, max_features=51, group_restarts=0, trial_steps=0, restart_warps=0)


def _starts(rows, d):
    th = np.zeros((*rows.shape[:-1], 51))
    th[..., : d + 1] = rows
    return th


@pytest.mark.parametrize("ctas_per_sm", [1, 2])
@pytest.mark.parametrize("i", [0, 1, 3, 4, 5])  # the fixtures of one and two restarts
def test_golden_splits(i, ctas_per_sm):
    from art.splitters import level_result_to_split, split_level

    kind, T, lam, R, iters, parent_loss = SG[f"s{i}_meta"]
    s = splitter_for(int(kind), T, lam, R, iters, ast.literal_eval(str(SG[f"s{i}_extra"])))
    X, y = SG[f"s{i}_X"], SG[f"s{i}_y"]
    d = X.shape[1]
    res = split_level(s, X.reshape(-1), y, [0, len(y)], [d], [int(kind)], T, lam, parent_loss=[parent_loss],
                      theta0=_starts(SG[f"s{i}_theta0"][None], d), traces=True, ctas_per_sm=ctas_per_sm, **WIDE)
    out = level_result_to_split(s, res, 0, len(y), parent_loss, True)
    np.testing.assert_allclose(out.loss, float(SG[f"s{i}_loss"]), rtol=1e-9)
    if int(R) == 1 or np.allclose(np.r_[out.w, out.z], SG[f"s{i}_theta"], rtol=1e-9, atol=1e-11):
        np.testing.assert_allclose(np.r_[out.w, out.z], SG[f"s{i}_theta"], rtol=1e-9, atol=1e-11)
        assert out.n_iters == int(SG[f"s{i}_n_iters"]) and out.n_right == int(SG[f"s{i}_n_right"])
        np.testing.assert_allclose(out.metadata["soft_loss_history"], SG[f"s{i}_soft_losses"], rtol=1e-9, atol=1e-13)


@pytest.mark.parametrize("ctas_per_sm", [1, 2])
@pytest.mark.parametrize("d,ns", [(3, [150_000, 700, 70_000, 3001]), (50, [40_000, 900, 17_000, 2048])])
def test_gangs_match_the_oracle_and_are_batch_independent(d, ns, ctas_per_sm):
    """Nodes above 16,384 rows are split by gangs of CTAs, the others stream through the ring."""

    from art.splitters import level_result_to_split, split_level

    rng = np.random.default_rng(d)
    K = len(ns)
    Xs = [rng.uniform(-1, 1, (n, d)) for n in ns]
    ys = [np.sin(2 * X[:, 0]) + 0.5 * np.tanh(4 * (X[:, 1] - X[:, 2])) for X in Xs]
    start = np.zeros(d + 1)
    start[:2] = 0.6, 0.8
    th0 = _starts(np.broadcast_to(start, (K, 1, d + 1)), d)
    T, lam, iters = 0.2, 1e-6, 5
    s = splitter_for(O.AFFINE, T, lam, 1, iters, {"min_side_points": 1, "min_side_fraction": 0.0})
    ro = np.concatenate([[0], np.cumsum(ns)])
    kw = dict(ctas_per_sm=ctas_per_sm, **WIDE)
    res = split_level(s, np.concatenate([X.reshape(-1) for X in Xs]), np.concatenate(ys), ro, [d] * K, [O.AFFINE] * K, T, lam,
                      parent_loss=[1.0] * K, theta0=th0, **kw)
    p = S.Params(max_iters=iters, n_restarts=1, min_side_points=1, min_side_fraction=0.0)
    for k in range(K):
        opt = S.optimize(Xs[k], ys[k], start, T, O.AFFINE, lam, p)
        out = level_result_to_split(s, res, k, ns[k], 1.0, True)
        np.testing.assert_allclose(np.r_[out.w, out.z], opt["theta"], rtol=1e-8, atol=1e-10)
        assert out.n_iters == opt["n_iters"]
        alone = split_level(s, Xs[k].reshape(-1), ys[k], [0, ns[k]], [d], [O.AFFINE], T, lam, parent_loss=[1.0],
                            theta0=th0[k:k + 1], **kw)
        for name in ("theta", "loss", "n_right", "n_iters", "beta"):
            np.testing.assert_array_equal(getattr(alone, name).cpu().numpy()[0], getattr(res, name).cpu().numpy()[k],
                                          err_msg=f"{name} {k}")
