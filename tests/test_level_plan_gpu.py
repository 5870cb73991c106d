"""Level routing by the number of nodes: nodes of a warp, of a CTA, of a cluster.

How a level's nodes are dealt out follows their number; a node's residual sums
must keep their bits, and its partition is the same list, whatever stands beside
it.  The sides are compared with the sign of the score in extended precision.
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

SIZES = [0, 1, 33, 255, 257, 449, 1000, 1024, 1025, 3000, 9001, 40000, 70001]


@pytest.mark.parametrize("d,kind", [(2, 2), (5, 0), (16, 2)])
@pytest.mark.parametrize("pads", [140, 500, 700, 2500, 9000, 30000])
def test_a_node_is_routed_the_same_in_any_level(d, kind, pads):
    from art.models import kind_feature_count, segment_residuals
    from art.tree import partition_rows

    rng = np.random.default_rng(pads + d)
    ns = rng.permutation(np.concatenate([np.tile(SIZES, 2), rng.integers(0, 8, pads)])).astype(np.int64)
    K = ns.size
    ro = np.concatenate([[0], np.cumsum(ns)])
    X, y = rng.uniform(-1.0, 1.0, (ro[-1], d)), rng.normal(size=ro[-1])
    p = kind_feature_count(d, kind)
    beta = rng.normal(size=(K, p))
    th = np.zeros((K, d + 1))
    th[:, :d] = rng.normal(size=(K, d))
    th[:, d] = rng.uniform(-0.3, 0.3, K)
    split = (rng.uniform(size=K) < 0.9).astype(np.int8)
    perm, nr = (t.cpu().numpy() for t in partition_rows(X.reshape(-1), ro, [d] * K, th, split=split))
    owner = np.repeat(np.arange(K), ns)
    right = (X.astype(np.longdouble) * th[owner, :d]).sum(1) - th[owner, d] >= 0
    right &= split[owner] != 0
    np.testing.assert_array_equal(nr, np.bincount(owner, weights=right, minlength=K).astype(np.int64))
    np.testing.assert_array_equal(perm, np.lexsort((np.arange(owner.size), right, owner)))
    sse, ssy = (t.cpu().numpy() for t in segment_residuals(X.reshape(-1), y, ro, [d] * K, [kind] * K, beta))
    assert np.all(sse[ns == 0] == 0.0)
    np.testing.assert_allclose(ssy, np.bincount(owner, weights=y * y, minlength=K), rtol=4e-13, atol=0)
    for k in np.flatnonzero(np.isin(ns, SIZES[1:]))[:40]:  # alone
        a, b = ro[k], ro[k + 1]
        s, q = segment_residuals(X[a:b].reshape(-1), y[a:b], [0, b - a], [d], [kind], beta[k:k + 1])
        assert s.item() == sse[k] and q.item() == ssy[k], ns[k]
