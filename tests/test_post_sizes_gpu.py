"""SLIC and plane snapping where their kernels change course, bit for bit
against the oracle.

Noise, hard edges and a low compactness pull cluster centres away until some pixels
lie in no window and keep their label; windows then grow to hold them.  Sizes below
one window, windows narrower than a warp, clusters larger than the update's buffer,
segments larger than the snap's shared memory (step 30), 1 to 64 trials."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.asarray(a, dtype=np.float64).view(np.uint64)


def _rgb(kind, W, H, rng):
    if kind == "noise":
        return rng.random(3 * W * H)
    if kind == "flat":
        return np.full(3 * W * H, 0.25)
    img = np.zeros((H, W, 3))
    for _ in range(12):                                   # hard-edged bars
        x, y = int(rng.integers(0, W)), int(rng.integers(0, H))
        img[y:y + int(rng.integers(1, H + 1)), x:x + int(rng.integers(1, W // 2 + 2))] = rng.random(3)
    return img.ravel()


@pytest.mark.parametrize("W,H,step,trials", [
    (97, 61, 12, 40), (64, 48, 3, 7), (7, 150, 5, 64), (200, 1, 4, 40), (90, 70, 30, 40),
    (33, 31, 40, 1),
])
@pytest.mark.parametrize("kind", ["noise", "bars", "flat"])
def test_slic_and_snap_match_oracle(svb, orc, kind, W, H, step, trials):
    rng = np.random.default_rng(W * 31 + H + step)
    rgb = _rgb(kind, W, H, rng)
    for comp, iters in ((10.0, 5), (0.5, 3), (40.0, 1)):
        want = orc.slic(rgb, W, H, step, comp, iters)[0]
        assert np.array_equal(svb.post.slic(rgb, W, H, step, comp, iters)[0], want), (comp, iters)
    yy, xx = np.mgrid[0:H, 0:W]
    d = (0.1 * xx + 0.05 * yy + 3.0 + rng.normal(0, 0.6, (H, W))).ravel()
    for valid in (None, rng.random(W * H) < 0.7):
        got = svb.post.plane_snap(d, rgb, W, H, valid=valid, step=step, thr=1.0, min_inl=0.3,
                                  trials=trials)
        ref = orc.plane_snap(d, rgb, W, H, valid=valid, step=step, thr=1.0, min_inl=0.3,
                             trials=trials)
        assert np.array_equal(_bits(got), _bits(ref))
