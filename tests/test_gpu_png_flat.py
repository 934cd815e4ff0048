"""One-colour images: the encoder's zlib stream, byte for byte, against the code sequence its parse
defines (first pixel as literals or, where that is shorter, a match with the scanline above; a run to the end
of the first 32-pixel step; longest matches over whole steps; the remainder)."""
import struct
import zlib

import numpy as np
import pytest

from axiomr_gb300 import api

pytestmark = pytest.mark.gpu


def symbol(s):
    for lo, hi, base, n in ((0, 143, 0x30, 8), (144, 255, 0x190, 9), (256, 279, 0, 7), (280, 287, 0xC0, 8)):
        if lo <= s <= hi:
            return format(base + s - lo, f"0{n}b")


def extra(v, n):
    return format(v, f"0{n}b")[::-1] if n else ""


def length(n):
    sizes = [0] * 8 + [e for e in range(1, 6) for _ in range(4)]
    base, s = 3, 257
    for e in sizes:
        if n < base + (1 << e) and n < 258:
            return symbol(s) + extra(n - base, e)
        base, s = base + (1 << e), s + 1
    return symbol(285)


def distance(d):
    base, c = 1, 0
    while True:
        e = max(0, c // 2 - 1)
        if d < base + (1 << e):
            return format(c, "05b") + extra(d - base, e)
        base, c = base + (1 << e), c + 1


def stream(w, h, ch, rgba):
    bits = ["110"]  # last block, fixed codes
    L = 1 + w * ch
    match = lambda px, d=ch: length(px * ch) + distance(d)  # noqa: E731
    longest = 258 // ch
    for r in range(h):
        bits.append(symbol(0))
        first = "".join(symbol(b) for b in rgba[:ch])
        if r and L <= 32768:
            d = distance(L)
            if 12 + len(d) - 5 < len(first):
                first = length(ch) + d
        bits.append(first)
        s = min(w, 32)
        if s > 1:
            bits.append(match(s - 1))
        whole, rest = (w - s) // 32 * 32, (w - s) % 32
        bits += [match(longest)] * (whole // longest)
        if whole % longest:
            bits.append(match(whole % longest))
        if rest:
            bits.append(match(rest))
    bits.append(symbol(256))
    b = "".join(bits)
    data = bytes(int(b[i:i + 8].ljust(8, "0")[::-1], 2) for i in range(0, len(b), 8))
    raw = (b"\0" + bytes(rgba[:ch]) * w) * h
    return b"\x78\x01" + data + struct.pack(">I", zlib.adler32(raw)), raw


@pytest.mark.parametrize("width", [1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 160, 255, 256, 257, 800, 2731, 5000, 10_923])
@pytest.mark.parametrize("rgba", [(9, 80, 143, 255), (144, 200, 255, 0)])
def test_one_colour(ctx, width, rgba):
    for h in (1, 3):
        fb = api.Framebuffer(ctx, width, h)
        fb.write(np.full((h, width, 4), (rgba[2], rgba[1], rgba[0], rgba[3]), np.uint8), np.zeros((h, width), np.float32))
        for ch in (3, 4):
            png, pos, idat = fb.read_png(ch), 8, b""
            while pos < len(png):
                n, = struct.unpack(">I", png[pos:pos + 4])
                if png[pos + 4:pos + 8] == b"IDAT":
                    idat += png[pos + 8:pos + 8 + n]
                pos += 12 + n
            exp, raw = stream(width, h, ch, rgba)
            assert zlib.decompress(exp) == raw
            assert idat == exp, (h, ch)
        fb.close()
