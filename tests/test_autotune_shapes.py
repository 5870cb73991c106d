"""The split tuner times every launch the library would make, and each once."""

import pytest


@pytest.mark.parametrize("R,d,p,tc,warp,cta", [(1, 16, 17, False, 1, 0), (2, 40, 41, False, 1, 0), (1, 50, 51, False, 0, None),
                                               (2, 8, 45, False, 1, 0), (16, 16, 17, False, 1, None),
                                               (16, 40, 41, False, 0, None), (1, 16, 17, True, 0, None)])
def test_each_launch_once(R, d, p, tc, warp, cta):
    from art import autotune

    shapes = autotune.split_candidates(R, 25, d, p, tc)
    timed = autotune._distinct_launches(shapes, R, d, p, tc)
    assert set(timed) <= set(shapes) and len(set(timed)) == len(timed)
    if cta == 0:  # one launch whatever the shape, by the warp form's own where there is one
        assert len(timed) == 1 and timed[0][3] == (1 if any(s[3] for s in shapes) else 0)
    else:
        assert sum(s[3] for s in timed) == warp
        assert [s for s in timed if not s[3]] == [s for s in shapes if not s[3]]
