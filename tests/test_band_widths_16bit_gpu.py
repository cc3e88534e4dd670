"""Every slot width of the band with 16-bit path costs, and the widest rows of the
static scratch, bit for bit.

P2 = 200 with the 9 x 7 window takes 16-bit path costs (66 + 200 > 255), P2 = 150
8-bit ones.  The bands are the smallest and largest of each width; the arithmetic is
integer and the parabola the reference's, so the tolerance is none: equal bits."""

import numpy as np
import pytest

from test_sgm_gpu import _check
from test_zz_no_alloc import _run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [0, 2, 3, 6, 7, 10, 11, 14, 15, 22, 23, 30, 31, 46, 47, 62, 63, 78,
                               79, 94, 95, 110, 111, 126])
def test_band_widths_with_16_bit_path_costs(svb, orc, R):
    kw = dict(R=R, P1=12.0, P2=200.0, rx=4, ry=3)
    _check(svb, orc, 53, 37, 300 + R, **kw)
    _check(svb, orc, 29, 40, 400 + R, uniq=0.04, paths=4, **kw)


@pytest.mark.parametrize("R", [62, 63, 78, 79, 94, 95, 110, 111, 126])
@pytest.mark.parametrize("P2", [150.0, 200.0])
def test_noalloc_widest_rows(svb, R, P2):
    W, H = 61, 47                         # 256 slots of 16 bits, 8 paths: 11.9 of 16 MB
    pair = svb.synth.make_pair(R, W, H, 1.0, 25.0)
    d0 = pair.disp.ravel() + np.random.default_rng(R).uniform(-3.0, 3.0, W * H)
    ref, out = _run_both(svb, pair, d0, R=R, P1=12.0, P2=P2, rx=4, ry=3)
    assert np.array_equal(ref.view(np.uint64), out.view(np.uint64))
