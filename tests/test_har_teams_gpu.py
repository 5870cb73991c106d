"""Hit-and-run teams: a chain's states do not depend on how many chains run.

Many chains run in teams of 8 or 16 lanes where the dimension allows, few in a
warp each; both must give the same bits (a chain amplifies a rounding, so the
comparison is exact).  A reference chain in numpy with the same injected draws
checks the arithmetic of the team paths over a length too short for roundings
to grow past the tolerance (ten steps amplify a rounding by less than 100).
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]

MANY, FEW = 2400, 37


def _polytopes(d, k, C, rng, box=True):
    import torch

    from art.sampling import DevicePolytopes

    rows = rng.integers(max(0, k - 2), k + 1, C)
    ro = np.concatenate([[0], np.cumsum(rows)])
    A = rng.normal(size=(max(ro[-1], 1), d))
    A /= np.linalg.norm(A, axis=1, keepdims=True)
    c = rng.uniform(-0.4, 0.4, (C, d))
    owner = np.repeat(np.arange(C), rows)
    b = np.einsum("ij,ij->i", A[: ro[-1]], c[owner]) + rng.uniform(0.1, 0.4, ro[-1])
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    lo = np.full((C, d), -1.0)
    if not box:  # a coordinate open on one side
        lo[:, 0] = -np.inf
    polys = DevicePolytopes(d, t(lo), t(np.ones((C, d))), t(ro), t(A), t(b if b.size else np.zeros(1)), k)
    return polys, c, ro, A, b, lo


@pytest.mark.parametrize("d,k", [(1, 0), (2, 4), (3, 9), (4, 20), (7, 8), (8, 16), (8, 32), (11, 12), (16, 17), (24, 5),
                                 (33, 12), (64, 12)])
@pytest.mark.parametrize("mode", ["batched", "scalar"])
@pytest.mark.parametrize("injected", [False, True])
def test_teams_give_the_same_bits(d, k, mode, injected):
    from art.sampling import DevicePolytopes, hit_and_run_device

    rng = np.random.default_rng(100 * d + k)
    polys, c, ro, A, b, lo = _polytopes(d, k, MANY, rng, box=(d % 2 == 0 or d == 1))
    steps = 7 * 11 + 3
    kw = dict(burn_in=3, thinning=7, n_rounds=11, mode=mode)
    draws = {}
    if injected:
        dirs, unif = rng.normal(size=(MANY, steps, d)), rng.uniform(size=(MANY, steps))
        dirs[::5, 4] = 0.0 if mode == "scalar" else dirs[::5, 4]  # skipped steps in some teams of a warp
        draws = dict(directions=dirs, uniforms=unif)
    else:
        draws = dict(seeds=np.arange(MANY, dtype=np.uint64) * np.uint64(7919))
    chain = np.arange(MANY, dtype=np.int32)
    s, x, st = hit_and_run_device(polys, chain, c, **draws, **kw)
    assert int(st.abs().sum()) == 0
    some = np.sort(rng.choice(MANY, FEW, replace=False))
    few = {n: v[some] for n, v in draws.items()}
    s2, x2, st2 = hit_and_run_device(polys, chain[some], c[some], **few, **kw)
    # (a sample slot whose step was skipped is not written)
    got, want = s.cpu().numpy()[:, some], s2.cpu().numpy()
    if not (injected and mode == "scalar"):
        np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(x.cpu().numpy()[some], x2.cpu().numpy())
    if not injected or mode != "batched":
        return
    first, _, _ = hit_and_run_device(polys, chain, c, burn_in=0, thinning=1, n_rounds=10, mode=mode,
                                     directions=dirs[:, :10].copy(), uniforms=unif[:, :10].copy())
    first = first.cpu().numpy()
    for j in some[:5]:
        Aj, bj = A[ro[j]:ro[j + 1]], b[ro[j]:ro[j + 1]]
        rows = np.vstack([Aj, np.eye(d), -np.eye(d)])
        xj = c[j].copy()
        slack = np.concatenate([bj - Aj @ xj, 1.0 - xj, xj - lo[j]])
        for step in range(10):
            u = dirs[j, step]
            au = rows @ u
            with np.errstate(divide="ignore", invalid="ignore"):
                q = slack / au
            hi, low = np.min(q[au > 0]), np.max(q[au < 0], initial=-np.inf)
            t = low + unif[j, step] * (hi - low)
            xj = xj + t * u
            slack = slack - t * au
            np.testing.assert_allclose(first[step, j], xj, rtol=0, atol=1e-12)


def test_direction_maps_give_the_same_bits():
    import torch

    from art.sampling import DevicePolytopes, hit_and_run_device

    rng = np.random.default_rng(8)
    for d in (2, 5, 12, 40):
        polys, c, *_ = _polytopes(d, 6, MANY, rng)
        polys.maps = torch.from_numpy(rng.normal(size=(MANY, d, d))).cuda()
        seeds = np.arange(MANY, dtype=np.uint64) + np.uint64(5)
        chain = np.arange(MANY, dtype=np.int32)
        kw = dict(burn_in=0, thinning=4, n_rounds=9, mode="scalar")
        s, x, st = hit_and_run_device(polys, chain, c, seeds=seeds, **kw)
        s2, x2, _ = hit_and_run_device(polys, chain[:FEW], c[:FEW], seeds=seeds[:FEW], **kw)
        assert int(st.abs().sum()) == 0
        np.testing.assert_array_equal(s.cpu().numpy()[:, :FEW], s2.cpu().numpy())
        np.testing.assert_array_equal(x.cpu().numpy()[:FEW], x2.cpu().numpy())
