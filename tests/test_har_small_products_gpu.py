"""Hit-and-run steps whose products or slacks are tiny: every nonzero product bounds.

The quotients of a step come from a reciprocal where the divisor and the slack
allow it, and from the division elsewhere: denormal products (unnormalised
directions with components of 1e-310, and starts on a face, where a dropped
bound would leave the polytope), and slacks far below the coordinates' scale
(from 2^-900 on the quotients are correctly rounded).
The polytopes are boxes and one row that is half a coordinate, so that numpy's
products, and with them its states, are exact to the bit.
"""

import numpy as np
import pytest

from conftest import gpu_available
from oracle import sampling as H

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

STEPS = 4


def _case(d, C, small, rng):
    """Box, row bound, starts and draws of C chains."""

    lo, hi = np.full((C, d), -2.0**-10), np.full((C, d), 2.0**-10)
    x0 = rng.uniform(-0.7, 0.7, (C, d)) * 2.0**-10
    face = rng.integers(0, d, C)
    dirs = rng.normal(size=(C, STEPS, d))
    unif = rng.uniform(size=(C, STEPS))
    if small == "products":  # on a face, with a denormal component there and others; some steps all denormal
        x0[np.arange(C), face] = np.where(rng.uniform(size=C) < 0.5, lo[:, 0], hi[:, 0])
        tiny = rng.choice([-1.0, 1.0], dirs.shape) * rng.uniform(1e-310, 2e-309, dirs.shape)
        swap = rng.uniform(size=dirs.shape) < 0.3
        swap[np.arange(C), 0, face] = True
        swap[::3, 1] = True
        dirs = np.where(swap, tiny, dirs)
    else:  # slacks of 1e-270 to 1e-200 on one face; half of the steps end on the chord's lower end
        lo[np.arange(C), face] = 0.0
        x0[np.arange(C), face] = 10.0 ** rng.uniform(-270, -200, C)
        unif[::2] = 0.0
    return lo, hi, x0, dirs, unif


@pytest.mark.parametrize("d,C", [(1, 37), (2, 37), (2, 2400), (5, 2400), (8, 37), (8, 2400), (12, 2400), (24, 37), (40, 37)])
@pytest.mark.parametrize("small", ["products", "slacks"])
def test_tiny_products_and_slacks_bound_the_step(d, C, small):
    import torch

    from art.sampling import DevicePolytopes, hit_and_run_device

    rng = np.random.default_rng(1000 * d + C)
    lo, hi, x0, dirs, unif = _case(d, C, small, rng)
    row = np.zeros((C, d))
    row[:, 0] = 0.5
    b = 0.5 * hi[:, 0]
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    polys = DevicePolytopes(d, t(lo), t(hi), t(np.arange(C + 1)), t(row), t(b), 1)
    samples, last, status = hit_and_run_device(polys, np.arange(C, dtype=np.int32), x0, burn_in=0, thinning=1,
                                               n_rounds=STEPS, mode="batched", directions=dirs, uniforms=unif)
    assert int(status.abs().sum()) == 0
    samples = samples.cpu().numpy()
    eye = np.eye(d)
    for c in range(C):
        A = np.vstack([row[c], eye, -eye])
        bound = np.concatenate([[b[c]], hi[c], -lo[c]])
        want, _ = H.chains_batched(A, bound, x0[c:c + 1], dirs[c:c + 1], unif[c:c + 1], 0, 1, STEPS)
        assert np.isfinite(want).all()
        np.testing.assert_array_equal(samples[:, c], want[:, 0])
    np.testing.assert_array_equal(last.cpu().numpy(), samples[-1])
