"""The static scratch's unpadded rows at every width of the band's slots, 8- and
16-bit path costs: bit for bit what the workspace's padded rows give (whose widths
differ for bands of 31 to 46 candidates)."""

import numpy as np
import pytest

from test_zz_no_alloc import _run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [2, 7, 10, 14, 15, 16, 22, 23, 30, 31, 46, 62])
@pytest.mark.parametrize("P2", [150.0, 200.0])
def test_noalloc_at_every_slot_width(svb, R, P2):
    W, H = 97, 61
    pair = svb.synth.make_pair(R, W, H, 1.0, 25.0)
    d0 = pair.disp.ravel() + np.random.default_rng(R).uniform(-3.0, 3.0, W * H)
    ref, out = _run_both(svb, pair, d0, R=R, P1=12.0, P2=P2, rx=4, ry=3)
    assert np.array_equal(ref.view(np.uint64), out.view(np.uint64))
