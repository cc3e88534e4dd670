"""The BF16 cost filter at the edges of its tiles.

The 3-D tensor-core convolution computes 4 rows x 32 columns of one disparity per
step and walks the disparities of a place, several steps and places per block.  So:
quarter widths of one tile, one column more and less and less than a tile, quarter
heights that are no multiple of four, one place, and the channel counts fixed at
compile time (12, 6) beside others.  Same emulation and tolerances as
test_bf16_gpu.py: BF16 operands, FP32 sums (TOL_EMU_MAX, TOL_EMU_MEAN there)."""

import pytest

from test_bf16_gpu import _front_check, _random_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(128, 16), (132, 20), (124, 36), (64, 12), (257, 133)])
def test_bf16_front_at_tile_edges(svb, orc, net, W, H):
    _front_check(svb, orc, net, W, H, seed=W + H)


@pytest.mark.parametrize("C,Cm,D,W,H", [(8, 4, 2, 132, 20), (16, 8, 16, 132, 36)])
def test_bf16_front_other_channels(svb, orc, C, Cm, D, W, H):
    _front_check(svb, orc, _random_net(svb, C, Cm, 8, D, seed=C + D), W, H, seed=D)
