"""Which split launch a serving node goes to, against the library's own rule."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "adaptive-regression-trees-art-_b200" / "csrc"


def test_limits_are_the_library_s():
    from art import autotune

    text = (CSRC / "split_warp.cu").read_text()
    limit = {k: int(re.search(rf"\b{k} = (\d+)", text).group(1)) for k in ("kNarrowAug", "kNarrowDim", "kWideAug", "kWideDim")}
    assert limit["kNarrowDim"] == autotune.WARP_MAX_DIM and limit["kNarrowAug"] == autotune.WARP_MAX_FEATURES + 1
    assert limit["kWideDim"] == autotune.WARP_WIDE_DIM and limit["kWideAug"] == autotune.WARP_WIDE_FEATURES + 1


@pytest.mark.parametrize("rows", [100, 1 << 16, (1 << 16) + 1])
def test_a_launch_never_mixes_forms(rows):
    from art.serving import SurrogateJob, _split_form

    jobs = [SurrogateJob(job_id=d, dim=d, n_initial=10, seed=0) for d in range(1, 65)]

    def warp_form(members):  # the library's rule for a launch of one restart a node
        return max(j.dim for j in members) <= 46 and max(j.n_features for j in members) + 1 <= 48

    groups = {}
    for j in jobs:
        groups.setdefault(_split_form(j, rows), []).append(j)
    for members in groups.values():
        for j in members:
            assert warp_form([j]) == warp_form(members)
        if not warp_form(members):  # the CTA form: one shape a launch
            assert len({(j.dim, j.n_features) for j in members}) == 1
