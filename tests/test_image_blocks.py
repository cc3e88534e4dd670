"""Huffman blocks of every length around the point from which a block has its own
fast tables (host only, no GPU): bytes equal to zlib's, for dynamic blocks that end
before it, at it and after it, one after the other in a stream."""

import zlib
from importlib import import_module

import numpy as np
import pytest

from test_image_inflate import _content, _png


@pytest.mark.parametrize("kind", ["skewed", "periods", "noise"])
@pytest.mark.parametrize("level", [1, 9])
def test_blocks_around_the_table_threshold(svb, kind, level):
    image = import_module(svb.__name__ + ".image")
    rng = np.random.default_rng(level + len(kind))
    W, H = 256, 256
    rows = _content(kind, W * H, rng).reshape(H, W)
    data = np.concatenate([np.zeros((H, 1), np.uint8), rows], axis=1).tobytes()
    # compressed sizes below and above 512 bytes, in turn
    for sizes in ((40, 300, 600), (500, 520, 540, 560), (700, 1500, 3000, 60), (20000,)):
        z = zlib.compressobj(level)
        body, at, k = b"", 0, 0
        while at < len(data):
            n = sizes[k % len(sizes)]
            body += z.compress(data[at:at + n]) + z.flush(zlib.Z_BLOCK)
            at += n
            k += 1
        raw, _ = image.decode_raw(_png(body + z.flush(), W, H))
        assert np.array_equal(np.asarray(raw).reshape(H, W), rows), sizes


def test_valid_streams_are_never_refused(svb):
    """Damaged streams that zlib reads to their end as the whole image, every row
    unfiltered, decode to the same bytes: nothing valid is rejected.  (The check of
    the stream's sum is the reader's own: it takes none.)"""
    image = import_module(svb.__name__ + ".image")
    rng = np.random.default_rng(11)
    W, H = 90, 64
    rows = np.concatenate([_content(k, W * H // 4, rng) for k in
                           ("skewed", "periods", "noise", "skewed")]).reshape(H, W)
    data = np.concatenate([np.zeros((H, 1), np.uint8), rows], axis=1).tobytes()
    good = zlib.compress(data, 6)
    accepted = 0
    for _ in range(3000):
        z = bytearray(good)
        z[int(rng.integers(2, len(z) - 4))] ^= 1 << int(rng.integers(0, 8))
        d = zlib.decompressobj(-15)
        try:
            want = d.decompress(bytes(z[2:]))
        except zlib.error:
            continue
        px = np.frombuffer(want, np.uint8)
        if not d.eof or px.size != len(data) or px.reshape(H, W + 1)[:, 0].any():
            continue
        accepted += 1
        raw, _ = image.decode_raw(_png(bytes(z), W, H))
        assert np.array_equal(np.asarray(raw).reshape(H, W), px.reshape(H, W + 1)[:, 1:])
    assert accepted >= 20
