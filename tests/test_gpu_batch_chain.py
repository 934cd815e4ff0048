"""The phased form's kernels start while the one before them drains: batches of few units,
launched back to back into the same framebuffers (every kernel overlaps its neighbours), must
leave the frames and the work counts that one launch alone leaves; batches without a drawn face have
no raster kernel before the tile pass."""
import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W
from test_gpu_batch import assert_same, plain_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,scale", [(1, 0.1), (3, 0.25), (24, 0.1)])
@pytest.mark.parametrize("clears", ["both", "depth", "color"])
def test_back_to_back(ctx, count, scale, clears):
    scenes = W.batch_scenes(count=count, seed=11, tex_size=32, resolution_scale=scale)
    draws = api.batch_draws(ctx, scenes)
    for d in draws:
        if clears != "both":
            d.framebuffer.clearColor(3, 5, 7, 9)
            d.framebuffer.clearDepth(float("inf"))
            if clears == "depth":
                d.clear_color = None
            else:
                d.clear_depth = None
    batch = api.Batch(ctx, draws)
    ctx.stats(True)
    ctx.stats()
    batch.launch()
    ctx.sync()
    once = ctx.stats()
    first = [d.framebuffer.read() for d in draws]
    again = 1 if clears == "color" else 20  # with its depth kept, a repeat shades nothing
    for _ in range(again):
        batch.launch()
    ctx.sync()
    many = ctx.stats()
    ctx.stats(False)
    assert many["triangles"] % once["triangles"] == 0 and many["fragments"] % once["fragments"] == 0
    for k, (d, f) in enumerate(zip(draws, first)):
        if clears != "color":
            assert_same(d.framebuffer.read(), f, f"draw {k} after {again} launches")
    if clears == "both":
        for k, (d, e) in enumerate(zip(draws, plain_frames(ctx, scenes, draws))):
            assert_same(d.framebuffer.read(), e, f"draw {k}")
    batch.close()


@pytest.mark.parametrize("vertices", [None, 0])
def test_no_faces(ctx, vertices):
    scenes = W.batch_scenes(count=2, seed=3, tex_size=32, resolution_scale=0.1)
    draws = api.batch_draws(ctx, scenes)
    for d, sc in zip(draws, scenes):
        m = sc.mesh
        d.mesh = api.Mesh(ctx, m.positions[:vertices], m.uvs[:vertices], m.normals[:vertices], m.indices[:0])
    batch = api.Batch(ctx, draws)
    for _ in range(3):
        batch.launch()
    ctx.sync()
    for d in draws:
        bgra, depth = d.framebuffer.read()
        assert (depth == np.float32(d.clear_depth)).all()
        assert (bgra == bgra[0, 0]).all()
    batch.close()
