"""What the library counts and times: tiles with a covered pixel, the key scan's own time, the launches of a
batch, and work that repeats exactly when a batch is launched again."""
import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def covered_tiles(depth):
    """16x16 tiles that hold a covered pixel of a frame cleared to infinity."""
    h, w = depth.shape
    d = np.zeros(((h + 15) // 16 * 16, (w + 15) // 16 * 16), bool)
    d[:h, :w] = np.isfinite(depth)
    return int(d.reshape(d.shape[0] // 16, 16, -1, 16).any(axis=(1, 3)).sum())


# triangles of a pixel or two, many of which cover no pixel centre of their box, in frames of either tile
# pass, from each form
@pytest.mark.parametrize("size,count", [((640, 480), 400), ((1921, 1083), 3000)])
@pytest.mark.parametrize("form", ["draw", "noalloc", api.BATCH_PHASED, api.BATCH_PERSISTENT])
@pytest.mark.parametrize("depth_min", [1.0, 0.09])  # the latter: some cut by the near plane
def test_tiles_with_a_covered_pixel(size, count, form, depth_min):
    if form == "noalloc" and size[0] * size[1] > 1 << 20:
        return  # beyond its limit
    ctx = api.Context(0)
    sc = W.soup_scene(count=count, width=size[0], height=size[1], seed=7, edge_min=0.5, edge_max=4.0, depth_min=depth_min,
                      depth_max=0.5 if depth_min < 0.1 else 50.0)
    sc.shader = W.Shader(W.SHADER_GOURAUD)
    ctx.stats(True)
    ctx.stats()
    if form == "noalloc":
        fb, mesh = api.Framebuffer(ctx, *size), api.Mesh.from_workload(ctx, sc.mesh)
        fb.clearColor(0, 0, 0, 255)
        fb.clearDepth()
        api.TiledPipeline(ctx, api.Camera.from_workload(sc.camera), fb).setShader(api.GouraudShader())
        model = np.ascontiguousarray(sc.model, np.float32)
        api.check(ctx.lib.axr_draw_mesh_noalloc(ctx.handle, mesh.handle, model.ctypes.data), ctx.handle)
        depth = fb.read()[1]
    elif form == "draw":
        ctx.draw_form = api.DRAW_KEYED
        depth = api.render_scene(ctx, sc)[1]
    else:
        ctx.batch_form = form
        draws = api.batch_draws(ctx, [sc])
        api.draw_batch(ctx, draws)
        depth = draws[0].framebuffer.read()[1]
    stats = ctx.stats()
    ctx.close()
    assert stats["shaded"] == np.isfinite(depth).sum() > 0
    assert stats["tiles"] == covered_tiles(depth)


def test_scan_time():
    """A larger frame's key scan (66 MB of keys at 3840x2160: 10 us at 6.8 TB/s, half of them covered and
    written back) is a stage of its own; events alone are a microsecond or two apart."""
    ctx = api.Context(0)
    sc = W.sphere_scene(width=3840, height=2160, lon=64, lat=32, tex_size=64, distance=2.0)
    fb, mesh = api.Framebuffer(ctx, 3840, 2160), api.Mesh.from_workload(ctx, sc.mesh)
    ctx.draw_form = api.DRAW_KEYED
    api.render_scene(ctx, sc, fb, mesh)
    ctx.profile(True)
    ctx.profile()
    for _ in range(10):
        api.render_scene(ctx, sc, fb, mesh)
    p = ctx.profile()
    ctx.close()
    assert p["draws"] == 10
    print(p)
    assert p["scan_ms"] / 10 > 0.006 and p["shade_ms"] > 0.0


KINDS = (W.SHADER_FLAT, W.SHADER_PHONG, W.SHADER_PBR, W.SHADER_BLINN_PHONG, W.SHADER_GOURAUD)


# a phased batch runs all shader kinds in one launch set (two from 128 draws on), the others a set per kind
@pytest.mark.parametrize("form,count,sets", [(api.BATCH_PHASED, 5, 1), (api.BATCH_PHASED, 130, 2), (api.BATCH_PERSISTENT, 5, 5),
                                             (api.BATCH_PERSISTENT, 130, 5), (api.BATCH_BINNED, 5, 5), (api.BATCH_BINNED, 130, 10),
                                             (api.BATCH_PHASED, 0, 0)])
def test_launch_sets(form, count, sets):
    ctx = api.Context(0)
    base = {k: W.sphere_scene(width=64, height=48, lon=16, lat=8, tex_size=16, shader=k) for k in KINDS}
    draws = api.batch_draws(ctx, [base[KINDS[k % 5]] for k in range(count)])
    ctx.batch_form = form
    batch = api.Batch(ctx, draws)
    assert batch.info()["launch_sets"] == sets
    before = ctx.profile()["kernel_launches"]
    batch.launch()
    ctx.sync()
    # kernels per set: vertices, faces, large triangles, tiles; one; vertices, faces, bins. Two sets: their counts merged
    per = {api.BATCH_PHASED: 4, api.BATCH_PERSISTENT: 1, api.BATCH_BINNED: 3}[form]
    merges = 1 if count >= 128 and form != api.BATCH_PERSISTENT else 0
    assert ctx.profile()["kernel_launches"] - before == sets * per + merges
    batch.close()
    ctx.close()


@pytest.mark.parametrize("count,scale", [(1, 0.1), (24, 0.1), (130, 0.05)])
@pytest.mark.parametrize("form", [api.BATCH_PHASED, api.BATCH_PERSISTENT])
def test_work_repeats(count, scale, form):
    ctx = api.Context(0)
    draws = api.batch_draws(ctx, W.batch_scenes(count=count, seed=11, tex_size=32, resolution_scale=scale))
    ctx.batch_form = form
    batch = api.Batch(ctx, draws)
    ctx.stats(True)
    ctx.stats()
    batch.launch()
    once = ctx.stats()
    assert all(once[k] > 0 for k in ("triangles", "fragments", "tiles", "tested", "shaded"))
    for _ in range(20):
        batch.launch()
    assert ctx.stats() == {k: 20 * v for k, v in once.items()}
    batch.close()
    ctx.close()
