"""The circular-slot SGM at the edges of its layouts, bit-exact against the
oracle: every slot width's smallest and largest band, both path-cost widths,
4 and 8 paths, the uniqueness test, images narrower than a warp's scanlines or
one pixel long, and band centres that jump past the free slots.  The
arithmetic is integer and the parabola the reference's, so the tolerance is
none: equal bits.
"""

import numpy as np
import pytest

from conftest import bits

pytestmark = pytest.mark.gpu


def _inputs(seed, W, H, dmax, jumps):
    rng = np.random.default_rng(seed)
    left = rng.integers(0, 256, (H, W)).astype(np.uint8)
    right = np.roll(left, -min(3, W - 1), axis=1)
    right[:, ::5] = rng.integers(0, 256, right[:, ::5].shape).astype(np.uint8)
    d = np.full((H, W), dmax / 2.0) + rng.uniform(-1.4, 1.4, (H, W))
    if jumps:                       # steps of every size from 1 px to past the band
        d += np.repeat(rng.integers(0, dmax + 1, (H, W // 4 + 1)), 4, axis=1)[:, :W]
        far = rng.random((H, W)) < 0.1
        d[far] = rng.uniform(0, 3.0 * dmax + 50, int(far.sum()))
    return left.ravel(), right.ravel(), d.ravel()


def _check(svb, orc, W, H, seed, jumps=True, **kw):
    L, R, d = _inputs(seed, W, H, max(2, min(W, 2 * kw["R"] + 6)), jumps)
    out, conf = svb.refine.refine_fullres(L, R, d, W, H, return_conf=True, **kw)
    ref, rconf = orc.refine_fullres(L / 255.0, R / 255.0, d, W, H, return_conf=True, **kw)
    assert np.array_equal(bits(out), bits(ref))
    assert np.array_equal(bits(conf), bits(rconf))


@pytest.mark.parametrize("R", [0, 1, 2, 3, 6, 7, 10, 11, 14, 15, 22, 23, 30, 31, 46, 47, 62, 63,
                               78, 79, 94, 95, 110, 111, 126])
def test_band_widths(svb, orc, R):
    kw = dict(R=R, P1=12.0, P2=150.0, rx=4, ry=3)
    _check(svb, orc, 53, 37, 100 + R, **kw)
    _check(svb, orc, 40, 29, 200 + R, jumps=False, **kw)


@pytest.mark.parametrize("kw", [
    dict(R=10, P1=12.0, P2=186.0, rx=4, ry=3),                     # 16-bit path costs: just past
    dict(R=10, P1=12.0, P2=189.0, rx=4, ry=3),
    dict(R=10, P1=4096.0, P2=4096.0, rx=4, ry=3),
    dict(R=10, P1=0.0, P2=0.0, rx=4, ry=3),
    dict(R=10, P1=100.0, P2=7.0, rx=4, ry=3),                      # P1 above P2
    dict(R=10, P1=3.0, P2=251.0, rx=0, ry=0),                      # one-pixel census
    dict(R=9, P1=2.0, P2=30.0, rx=2, ry=2, paths=4),
    dict(R=10, P1=12.0, P2=150.0, rx=4, ry=3, uniq=0.05),
    dict(R=5, P1=12.0, P2=400.0, rx=4, ry=3, uniq=0.02, paths=4),
    dict(R=20, P1=12.0, P2=150.0, rx=4, ry=3, uniq=0.05),
    dict(R=40, P1=12.0, P2=1000.0, rx=4, ry=3, paths=4)])
def test_penalties_paths_and_uniqueness(svb, orc, kw):
    _check(svb, orc, 61, 41, int(kw["P2"]) + kw["R"], **kw)


@pytest.mark.parametrize("W,H", [(1, 1), (2, 1), (1, 7), (15, 16), (16, 15), (17, 33), (33, 17),
                                 (200, 3), (3, 200)])
@pytest.mark.parametrize("R", [3, 10, 12, 40])
def test_small_and_thin_images(svb, orc, W, H, R):
    _check(svb, orc, W, H, 7 * W + H, R=R, P1=12.0, P2=150.0, rx=4, ry=3)


@pytest.mark.parametrize("W,H", [(97, 61), (61, 97)])
def test_both_views_and_masked_half_widths(svb, orc, W, H):
    """lr_refine of one pair, and the same pair three times in a batch."""
    kw = dict(R=10, P1=12.0, P2=150.0, rx=4, ry=3)
    L, R, d = _inputs(W, W, H, 24, True)
    ref, rst = orc.lr_refine(L / 255.0, R / 255.0, d, W, H, tol=2.0, **kw)
    out, st = svb.refine.lr_refine(L, R, d, W, H, tol=2.0, **kw)
    assert np.array_equal(bits(out), bits(ref)) and np.array_equal(st, rst)
    for out, st in svb.batch.lr_refine_batch([(L, R, d, W, H)] * 3, tol=2.0, **kw):
        assert np.array_equal(bits(out), bits(ref)) and np.array_equal(st, rst)
