"""Residual sums and partitions of a level: cluster sizes, range edges, row layouts.

Partitions are compared exactly with the sign of the score in extended
precision (the drawn rows are never within rounding of their planes); residual
sums with numpy in FP64, to n_terms * eps relative of the sum of absolute
terms (4e-13 covers 4e5 rows in any order of pairwise partial sums), and bit for
bit between a node alone and the same node in a batch.
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


def _features(X, kind):
    one = np.ones((X.shape[0], 1))
    i, j = np.triu_indices(X.shape[1])
    return {0: lambda: np.hstack([X, one]), 1: lambda: np.hstack([one, X]), 2: lambda: np.hstack([one, X, X[:, i] * X[:, j]]),
            3: lambda: X, 4: lambda: np.hstack([X, X[:, i] * X[:, j]])}[kind]()


# rows of whole sectors, of 16-byte pairs and of single doubles; an odd lead
# element shifts every row off its alignment
@pytest.mark.parametrize("d,kind,lead", [(1, 0, 0), (2, 2, 0), (3, 2, 0), (4, 2, 0), (4, 2, 1), (6, 4, 0), (8, 2, 0), (8, 2, 2),
                                         (13, 0, 0), (16, 2, 0), (32, 0, 0), (33, 3, 0), (64, 1, 0)])
@pytest.mark.parametrize("pad_nodes", [0, 600])
def test_level_routing(d, kind, lead, pad_nodes):
    from art.models import kind_feature_count, segment_residuals
    from art.tree import partition_rows

    rng = np.random.default_rng(10 * d + kind)
    ns = np.array([0, 1, 31, 255, 256, 257, 1023, 1024, 1025, 4097, 20011, 70000] + [3] * pad_nodes)
    K = ns.size
    ro = np.concatenate([[0], np.cumsum(ns)])
    X = rng.uniform(-1.0, 1.0, (ro[-1], d))
    y = rng.normal(size=ro[-1])
    p = kind_feature_count(d, kind)
    beta = rng.normal(size=(K, p))
    th = np.zeros((K, d + 1))
    th[:, :d] = rng.normal(size=(K, d))
    th[:, :d] /= np.linalg.norm(th[:, :d], axis=1, keepdims=True)
    th[:, d] = rng.uniform(-0.3, 0.3, K)
    split = np.ones(K, np.int8)
    split[4] = 0
    flat = np.concatenate([np.zeros(lead), X.reshape(-1)])
    xo = ro[:-1] * d + lead
    sse, ssy = segment_residuals(flat, y, ro, [d] * K, [kind] * K, beta, x_offsets=xo)
    perm, nr = partition_rows(flat, ro, [d] * K, th, split=split, x_offsets=xo)
    sse, ssy, perm, nr = (t.cpu().numpy() for t in (sse, ssy, perm, nr))
    for k in range(12):
        a, b = ro[k], ro[k + 1]
        r2 = (y[a:b] - _features(X[a:b], kind) @ beta[k]) ** 2
        assert abs(sse[k] - r2.sum()) <= 4e-13 * max(r2.sum(), 1e-300)
        assert abs(ssy[k] - (y[a:b] ** 2).sum()) <= 4e-13 * max((y[a:b] ** 2).sum(), 1e-300)
        right = (X[a:b].astype(np.longdouble) @ th[k, :d].astype(np.longdouble) - th[k, d]) >= 0 if split[k] else np.zeros(b - a, bool)
        assert nr[k] == right.sum()
        np.testing.assert_array_equal(perm[a:b], a + np.concatenate([np.flatnonzero(~right), np.flatnonzero(right)]))
    for k in (9, 11):  # alone: another cluster size when the batch is long
        a, b = ro[k], ro[k + 1]
        s1, y1 = segment_residuals(X[a:b].reshape(-1), y[a:b], [0, b - a], [d], [kind], beta[k:k + 1])
        assert s1.cpu().numpy()[0] == sse[k] and y1.cpu().numpy()[0] == ssy[k]


def test_partition_past_the_mask_capacity():
    """A node of more rows than its cluster's bit masks hold."""
    import torch

    from art.tree import partition_rows

    n = 16 * (1 << 18) + 12345
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x = torch.rand((n, 2), generator=g, device="cuda", dtype=torch.float64) - 0.5
    th = torch.tensor([[0.6, 0.8, 0.01]], device="cuda", dtype=torch.float64)
    perm, nr = partition_rows(x.reshape(-1), torch.tensor([0, n], device="cuda"), [2], th)
    s = x[:, 0] * 0.6 + x[:, 1] * 0.8 - 0.01
    assert s.abs().min() > 1e-14  # no row within rounding of the plane
    right = s >= 0
    assert int(nr[0]) == int(right.sum())
    assert torch.equal(perm, torch.cat([torch.nonzero(~right)[:, 0], torch.nonzero(right)[:, 0]]))
