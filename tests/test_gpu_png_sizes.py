"""A PNG batch's sizes reach the host before its files are written: sizes, files and framebuffers of
encodes enqueued one after another, with fewer files than copy streams and more."""
import numpy as np
import pytest

import pngfile
from axiomr_gb300 import api
from test_gpu_png_blocks import framebuffer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 4, 5, 9])
@pytest.mark.parametrize("channels", [3, 4])
def test_repeated(ctx, count, channels):
    rng = np.random.default_rng(count)
    batch = api.PngBatch(ctx)
    for k in range(6):
        n = max(1, (count * (k + 1)) // 3)  # counts that grow past the first allocation
        imgs = [rng.integers(0, 4 ** (k + 1) % 251 + 2, (40 + 13 * k, 700 + i, 4), dtype=np.uint8) for i in range(n)]
        fbs = [framebuffer(ctx, i) for i in imgs]
        batch.encode(fbs, channels)
        sizes = batch.sizes()
        for fb in fbs:  # the encode has read the planes
            fb.clearColor(0, 0, 0, 0)
        files = batch.read()
        assert [len(f) for f in files] == sizes == batch.sizes()
        for img, f in zip(imgs, files):
            assert np.array_equal(pngfile.decode(f)[0], pngfile.expected(img, channels))
    batch.close()
