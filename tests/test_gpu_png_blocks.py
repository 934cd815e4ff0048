"""The PNG encoder's 128-pixel blocks, its strided CRC and its two pack-group sizes: decoded by the
independent reader of pngfile.py (zlib checks every CRC and the Adler-32)."""
import numpy as np
import pytest

import pngfile
from axiomr_gb300 import api

pytestmark = pytest.mark.gpu


def framebuffer(ctx, bgra):
    h, w = bgra.shape[:2]
    fb = api.Framebuffer(ctx, w, h)
    fb.write(np.ascontiguousarray(bgra, np.uint8), np.zeros((h, w), np.float32))
    return fb


def images(rng, w):
    """Rows that end, change or go on at every place a block can see: flat rows, a flat row with one
    other pixel at each of its positions around the block edges, rows equal to the one above, noise
    between flat stretches, runs of every length."""
    flat = np.full((1, w, 4), (9, 80, 200, 255), np.uint8)
    rows = [flat, flat]
    for x in sorted({x for e in range(0, w + 1, 128) for x in range(e - 3, e + 4) if 0 <= x < w}):
        r = flat.copy()
        r[0, x] = (1, 2, 3, 4)
        rows += [r, r, flat]
    for lo in range(0, w, 100):
        r = flat.copy()
        r[0, lo:lo + 70] = rng.integers(0, 256, (min(70, w - lo), 4), dtype=np.uint8)
        rows += [r, r]
    lengths = rng.integers(1, 140, 400)
    r = np.repeat(rng.integers(0, 256, (400, 4), dtype=np.uint8), lengths, axis=0)[:w]
    rows += [r[None], np.roll(r, 1, axis=0)[None]]
    return np.concatenate(rows)


@pytest.mark.parametrize("width", [1, 31, 33, 95, 127, 128, 129, 160, 255, 256, 257, 383, 384, 385, 1000])
@pytest.mark.parametrize("channels", [3, 4])
def test_block_edges(ctx, width, channels):
    img = images(np.random.default_rng(width), width)
    got, ch, _ = pngfile.decode(framebuffer(ctx, img).read_png(channels))
    assert ch == channels and np.array_equal(got, pngfile.expected(img, channels))


# stream lengths of every remainder modulo 4, below and above the CRC's 256 words, and several
# chunks (noise does not compress: 8 or 9 bits a byte)
@pytest.mark.parametrize("height", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 400])
def test_crc_lengths(ctx, height):
    rng = np.random.default_rng(height)
    imgs = [rng.integers(0, 256, (height, w, 4), dtype=np.uint8) for w in (1, 2, 3, 37, 90, 331)]
    for img, data in zip(imgs, api.read_png(ctx, [framebuffer(ctx, i) for i in imgs], 3)):
        assert np.array_equal(pngfile.decode(data)[0], pngfile.expected(img, 3))


# past 12 pack groups of 32 scanlines per SM the groups grow from 8 scanlines to 32
@pytest.mark.parametrize("heights", [[1000] * 59 + [7, 31, 32, 33]])
def test_large_groups(ctx, heights):
    rng = np.random.default_rng(3)
    imgs = []
    for k, h in enumerate(heights):
        img = np.repeat(rng.integers(0, 256, ((h + 4) // 5, 9 + k, 4), dtype=np.uint8), 5, axis=0)[:h]
        imgs.append(img)
    for img, data in zip(imgs, api.read_png(ctx, [framebuffer(ctx, i) for i in imgs], 4)):
        assert np.array_equal(pngfile.decode(data)[0], pngfile.expected(img, 4))
