"""Device-drawn starts: z is the median of the node's scores at every size.

With a first step far below rounding the search returns its start, so z is the
start's and w differs from it by the last renormalisation (1e-15).  The median
of n scores moves by no more than |x| times that, and the next order statistic
is 1 / (n density) away, at least 1e-6 here: 1e-12 tells them apart.
"""

import numpy as np
import pytest

from conftest import gpu_available
from oracle import ridge as O
from test_split_gangs_gpu import _call
from test_split_gpu import splitter_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


def _starts(d, ns, lead, repeat=1):
    rng = np.random.default_rng(100 * d + len(ns))
    Xs = [np.repeat(rng.uniform(-1, 1, (-(-n // repeat), d)), repeat, axis=0)[:n] for n in ns]
    ys = [np.sin(2 * X[:, 0]) + 0.1 * rng.normal(size=len(X)) for X in Xs]
    K = len(ns)
    s = splitter_for(O.AFFINE, 0.2, 1e-6, 1, 1, {"alpha0": 1e-300, "min_side_points": 1})
    res = _call(s, Xs, ys, [d] * K, [O.AFFINE] * K, 0.2, 1e-6, None, lead)
    theta = res.theta.cpu().numpy()
    assert not res.failure.cpu().numpy().any()
    for X, t in zip(Xs, theta):
        assert np.linalg.norm(t[:d]) == pytest.approx(1.0, rel=1e-14)
        assert abs(t[d] - np.median(X @ t[:d])) <= 1e-12
    return theta


# ranks of 1,024 rows; eight ranks keep 65,536 keys and recompute the rest;
# rows of 8-byte, 16-byte and 32-byte loads
@pytest.mark.parametrize("d,lead", [(1, 0), (3, 0), (4, 0), (4, 1), (6, 0), (8, 2), (22, 0), (40, 0)])
def test_start_is_the_median(d, lead):
    _starts(d, [201, 1024, 1025, 2049, 30000, 65536, 65537, 140002], lead)


def test_single_blocks_and_ties():
    """More starts than are given clusters (blocks past their keys among them),
    and tied middle values."""
    _starts(4, [8193, 300, 20000, 8192, 777] + [64] * 1100, 0)
    _starts(4, [1000, 1002, 70000], 0, repeat=4)
