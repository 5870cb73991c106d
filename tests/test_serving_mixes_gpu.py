"""Jobs of every split form in one tick: each is identical alone and in the mix.

Dimensions above 46 take another form of the split search than the others, and
nodes of more than 65,536 rows another launch than small ones.
"""

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


def test_wide_and_large_jobs_beside_narrow_ones():
    from art.serving import ServingEngine, SurrogateJob

    spec = [(2, 70000, 2), (8, 3000, 4), (32, 3000, 4), (48, 4000, 3), (60, 3000, 3), (4, 68000, 2), (2, 2000, 4), (24, 3500, 3)]
    jobs = [SurrogateJob(job_id=i, dim=d, n_initial=n, seed=50 + i, max_depth=depth, rounds=1, max_iters=12)
            for i, (d, n, depth) in enumerate(spec)]
    mixed = ServingEngine(precision="fp64").run(jobs)
    for job, res in zip(jobs, mixed):
        alone = ServingEngine(precision="fp64").build_alone(job)
        assert [p for p, *_ in res.splits] == [p for p, *_ in alone.splits] and len(res.splits) > 0
        for (path, t1), (_, t2) in zip(res.splits, alone.splits):
            np.testing.assert_array_equal(t1, t2, err_msg=f"d={job.dim} {path}")
        for l1, l2 in zip(res.leaves, alone.leaves):
            np.testing.assert_array_equal(l1[1], l2[1], err_msg=f"d={job.dim} {l1[0]}")
