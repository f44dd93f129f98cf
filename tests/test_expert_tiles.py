"""Which tiles a routed layer sorts its pairs into, at the edges of each range of pairs an expert."""
import pytest

from picolm_b200 import ops
from picolm_b200.parts.feed_forward import tc_tile_rows


@pytest.mark.parametrize("pairs,rows", [(15, 0), (16, 16), (104, 16), (105, 128), (116, 128), (117, 16), (128, 16), (223, 16), (224, 128)])
def test_tiles_by_pairs_an_expert(pairs, rows):
    for experts in (1, 8, ops.TC_EXPERTS):
        assert tc_tile_rows(pairs * experts, experts) == rows


@pytest.mark.parametrize("pairs,rows", [(16, 0), (63, 0), (64, 128), (129, 128)])
def test_more_experts_than_the_kernel_with_weights_on_the_rows_takes(pairs, rows):
    assert tc_tile_rows(pairs * (ops.TC_EXPERTS + 1), ops.TC_EXPERTS + 1) == rows
