"""The FP32 block-row solve on both sides of the width at which its CTAs take 64
columns instead of 32: twice as many columns as all SMs hold at 32 each, two
CTAs per SM."""
import pytest
from test_gpu_trsm32 import test_f32_block_row_solve as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 200, 512])
@pytest.mark.parametrize("ncols", [9471, 9472, 9473, 9503, 9505])
def test_both_sides_of_the_tile_choice(K, ncols):
    check(K, ncols, True, True)
    check(K, ncols, False, True)
