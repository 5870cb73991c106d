"""Wide systems give the same bits alone and beside others.

The rows a CTA stages at a time follow the batch's widest system; which warp adds
which rows must not.
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

AFFINE, POLY2 = 0, 2


@pytest.mark.parametrize("d,kind", [(48, AFFINE), (55, AFFINE), (62, AFFINE), (9, POLY2), (64, AFFINE), (12, POLY2), (16, POLY2)])
@pytest.mark.parametrize("beside", [(16, POLY2), (64, AFFINE), (120, AFFINE), (158, AFFINE)])
def test_alone_and_beside_a_wider_system(d, kind, beside):
    from art.models import kind_feature_count, solve_weighted_ridge_batched

    rng = np.random.default_rng(d)
    dims, kinds, ns = [d, beside[0], 64], [kind, beside[1], AFFINE], [777, 400, 300]
    xs = [rng.uniform(-1.0, 1.0, (n, k)) for n, k in zip(ns, dims)]
    ro = np.concatenate([[0], np.cumsum(ns)])
    xo = np.concatenate([[0], np.cumsum([x.size for x in xs])])[:-1]
    y, w = rng.normal(size=ro[-1]), rng.uniform(0.0, 1.0, ro[-1])
    p = kind_feature_count(d, kind)
    kw = dict(weight_floor=0.0)
    both = solve_weighted_ridge_batched(np.concatenate([x.reshape(-1) for x in xs]), y, w, ro, dims, kinds, [1e-6] * 3,
                                        x_offsets=xo, max_features=max(kind_feature_count(a, b) for a, b in zip(dims, kinds)),
                                        max_dim=max(dims), **kw)
    one = solve_weighted_ridge_batched(xs[0].reshape(-1), y[: ns[0]], w[: ns[0]], [0, ns[0]], [d], [kind], [1e-6], max_features=p,
                                       max_dim=d, **kw)
    assert int(both.status[0]) == 0 and int(one.status[0]) == 0
    np.testing.assert_array_equal(both.beta.cpu().numpy()[0, :p], one.beta.cpu().numpy()[0, :p])
