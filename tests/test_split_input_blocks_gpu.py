"""Warp form of the split search: affine models whose inputs fill whole blocks.

The blocks then hold the inputs alone and the sums with 1 and y are lane sums.
Sizes at and one below a whole block, of every block count, in every gang size,
meet the oracle's search as the other sizes do.
"""

import pytest

from conftest import gpu_available
from oracle import ridge as O
from test_split_gangs_gpu import test_gang_sizes_match_the_oracle as _check

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("d,lead", [(7, 0), (8, 0), (15, 0), (16, 1), (23, 0), (24, 0), (31, 1), (32, 0), (39, 0)])
def test_whole_input_blocks(d, lead):
    _check(O.AFFINE, d, lead)


# one input more, a constant first, none: the general blocks
@pytest.mark.parametrize("kind,d", [(O.AFFINE, 9), (O.AFFINE, 17), (O.AFFINE, 33), (O.POLY1, 8), (O.POLY1, 16)])
def test_other_models_keep_the_general_blocks(kind, d):
    _check(kind, d, 0)
