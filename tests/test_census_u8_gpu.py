"""The 8-bit census of the 9 x 7 window (4 pixels per thread, byte comparisons) at
its edges, bit for bit against the oracle: images narrower than a word and than the
window, widths of every remainder, rows and bases at odd addresses, and the values
on both sides of the bytes' top bit."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (3, 9), (4, 1), (31, 8), (32, 8), (33, 9), (34, 17),
                                 (64, 7), (127, 23)])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_census_u8_matches_oracle(svb, orc, W, H, shift):
    rng = np.random.default_rng(W * 100 + H)
    for values in (np.arange(256), np.array([0, 1, 126, 127, 128, 129, 254, 255])):
        img = rng.choice(values, W * H).astype(np.uint8)
        buf = torch.zeros(W * H + 8, dtype=torch.uint8, device="cuda")
        t = buf[shift:shift + W * H]                     # a view at any address
        t.copy_(torch.as_tensor(img))
        got = svb.refine.census(t, W, H, 4, 3).cpu().numpy().view(np.uint64)
        assert np.array_equal(got, orc.census(img.astype(np.float64), W, H, 4, 3))
