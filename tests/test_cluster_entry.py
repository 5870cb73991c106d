"""Kernels that reach into another CTA's shared memory: a cluster barrier comes
first.  The CTAs of a cluster are scheduled together, but nothing orders the
start of one before an access by another except a barrier, and no run shows the
order missing, so the sources are read: in every function that maps another
CTA's shared memory, a cluster barrier stands before the first such access."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "adaptive-regression-trees-art-_b200" / "csrc"
BARRIER = re.compile(r"\bcl(uster)?\.sync\(\)|\bcluster_wait\(\)|\bbarrier_wait\(")


def _functions(text):
    """Top-level definitions: they end with a brace in the first column."""

    text = re.sub(r"//[^\n]*", "", text)
    return [body for body in re.split(r"^\};?\s*$", text, flags=re.M) if "map_shared_rank" in body]


@pytest.mark.parametrize("source", ["split.cu", "split_warp.cu", "tree.cu"])
def test_a_cluster_barrier_precedes_the_first_remote_access(source):
    bodies = _functions((CSRC / source).read_text())
    assert bodies
    for body in bodies:
        barrier = BARRIER.search(body)
        assert barrier and barrier.start() < body.index("map_shared_rank"), body.strip()[:400]
