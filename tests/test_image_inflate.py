"""The inflater's fast loop at its edges (host only, no GPU).

The loop stops for what its tables do not hold and near the ends of input and
output; the general decoder goes on from there.  So: literal codes of up to 15
bits (longer than the table), copies at distances 1 to 9 and 32768 of lengths 3 to
258, fixed, dynamic and stored blocks, images that end inside a copy's slack, and
damaged streams, all against zlib."""

import zlib
from importlib import import_module

import numpy as np
import pytest


def _png(body, W, H):
    def chunk(tag, b):
        return len(b).to_bytes(4, "big") + tag + b + zlib.crc32(tag + b).to_bytes(4, "big")
    head = W.to_bytes(4, "big") + H.to_bytes(4, "big") + bytes([8, 0, 0, 0, 0])
    return (b"\x89PNG\r\n\x1a\n" + chunk(b"IHDR", head) + chunk(b"IDAT", body) +
            chunk(b"IEND", b""))


def _content(kind, n, rng):
    if kind == "skewed":                # Fibonacci-like frequencies: codes of 15 bits
        p = 0.5 ** np.arange(1, 41)
        return rng.choice(40, n, p=p / p.sum()).astype(np.uint8)
    if kind == "periods":               # copies at short distances
        out = np.empty(0, np.uint8)
        while out.size < n:
            d = int(rng.integers(1, 10))
            out = np.concatenate([out, np.tile(rng.integers(0, 256, d, dtype=np.uint8),
                                               int(rng.integers(1, 300)))])
        return out[:n]
    if kind == "far":                   # copies at the largest distances
        a = rng.integers(0, 256, 32700, dtype=np.uint8)
        return np.resize(a, n)
    return rng.integers(0, 256, n, dtype=np.uint8)


@pytest.mark.parametrize("kind", ["skewed", "periods", "far", "noise"])
@pytest.mark.parametrize("W,H", [(1, 1), (255, 1), (261, 2), (300, 301)])
def test_inflate_matches_zlib(svb, kind, W, H):
    image = import_module(svb.__name__ + ".image")
    rng = np.random.default_rng(W * 1000 + H + len(kind))
    rows = _content(kind, W * H, rng).reshape(H, W)
    data = np.concatenate([np.zeros((H, 1), np.uint8), rows], axis=1).tobytes()
    for level in (0, 1, 6, 9):
        for strategy in (zlib.Z_DEFAULT_STRATEGY, zlib.Z_FIXED, zlib.Z_HUFFMAN_ONLY):
            z = zlib.compressobj(level, zlib.DEFLATED, 15, 8, strategy)
            raw, desc = image.decode_raw(_png(z.compress(data) + z.flush(), W, H))
            assert (desc.width, desc.height) == (W, H)
            assert np.array_equal(np.asarray(raw).reshape(H, W), rows), (level, strategy)


def test_inflate_of_damaged_streams(svb):
    """Whatever zlib still inflates to the whole image decodes alike; whatever stops
    zlib short of it is rejected."""
    image = import_module(svb.__name__ + ".image")
    rng = np.random.default_rng(7)
    W, H = 120, 40
    rows = np.concatenate([_content(k, W * H // 4, rng) for k in
                           ("skewed", "periods", "noise", "skewed")]).reshape(H, W)
    data = np.concatenate([np.zeros((H, 1), np.uint8), rows], axis=1).tobytes()
    good = zlib.compress(data, 6)
    for _ in range(400):
        z = bytearray(good)
        for _ in range(int(rng.integers(1, 4))):
            z[int(rng.integers(2, len(z) - 4))] ^= 1 << int(rng.integers(0, 8))
        try:
            want = zlib.decompressobj(-15).decompress(bytes(z[2:]))
        except zlib.error:
            want = None
        try:
            raw, _ = image.decode_raw(_png(bytes(z), W, H))
        except ValueError:
            raw = None
        if want is None:
            assert raw is None
            continue
        px = np.frombuffer(want[:len(data)], np.uint8)
        if px.size == len(data) and (px.reshape(H, W + 1)[:, 0] == 0).all():
            if raw is not None:          # (zlib stops quietly at the end of its input)
                assert np.array_equal(np.asarray(raw).reshape(H, W), px.reshape(H, W + 1)[:, 1:])
