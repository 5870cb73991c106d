"""Limits of backtracks up to the largest: the same searches as with a few thousand.

A step that has underflowed to zero cannot become acceptable, so an attempt ends
there whatever the limit; until then the limit must not be reached or overflow.
"""

import numpy as np
import pytest

from conftest import gpu_available
from oracle import ridge as O
from test_split_gpu import splitter_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


# warp form alone and in a gang, the CTA form, each with searches that mostly
# fail (a slope that the objective cannot meet) and that succeed
@pytest.mark.parametrize("R,warps,n", [(1, 1, 300), (2, 1, 5000), (4, 1, 300), (4, 0, 300)])
@pytest.mark.parametrize("armijo", [1e-4, 0.99])
def test_any_limit_of_backtracks(R, warps, n, armijo):
    from art.splitters import split_level

    rng = np.random.default_rng(n + R)
    d = 3
    X = rng.uniform(-1, 1, (n, d))
    y = np.tanh(5 * (X[:, 0] - 0.3 * X[:, 1])) + 0.1 * rng.normal(size=n)
    th0 = np.concatenate([rng.normal(size=(1, R, d)), np.zeros((1, R, 1))], axis=2)
    got = []
    for limit in (2000, 2**31 - 1):
        s = splitter_for(O.AFFINE, 0.1, 1e-6, R, 6, {"max_backtracks": limit, "armijo_c": armijo, "min_side_points": 2})
        r = split_level(s, X.reshape(-1), y, [0, n], [d], [O.AFFINE], 0.1, 1e-6, theta0=th0, traces=True, restart_warps=warps,
                        group_restarts=0, trial_steps=0, ctas_per_sm=0)
        got.append({k: getattr(r, k).cpu().numpy() for k in ("theta", "loss", "n_iters", "stop_reason", "final_alpha",
                                                              "trace_loss", "trace_step", "trace_backtracks")})
    for name, v in got[0].items():
        np.testing.assert_array_equal(got[1][name], v, err_msg=name)
    assert got[0]["n_iters"][0] >= 0
