"""The face phase's two rasterisers (a thread per box of at most 6 pixels, shared (triangle,
pixel) pairs above) and its limits against the CPU oracle: box sizes around the limits, face
counts around a CTA's share, pair tables that overflow into the large-triangle pass."""
import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W
from helpers import assert_parity

pytestmark = pytest.mark.gpu


def soup(count, edge, width=331, height=213, seed=21):
    return W.soup_scene(count=count, width=width, height=height, seed=seed, edge_min=edge, edge_max=edge + 0.01,
                        depth_min=1.0, depth_max=50.0)


def check(ctx, port, sc, what):
    vp = port.camera(sc.camera)[2]
    assert_parity(api.render_scene(ctx, sc, view_proj=vp), port.draw(sc, vp), what)


# edges from below a pixel to boxes past the 64-pixel limit, wider than an 8-pixel step and
# than a 16-pixel tile
@pytest.mark.parametrize("edge", [0.3, 1.0, 1.8, 3.0, 6.0, 7.0, 8.5, 17.0, 40.0])
def test_box_sizes(ctx, port, edge):
    check(ctx, port, soup(3000, edge), f"edge {edge}")


# one face, around the smallest share of a CTA (16), a warp, a CTA; and past 4 CTAs of 128 on
# each of 152 SMs, where a thread takes a face and each warp shares its own pairs
@pytest.mark.parametrize("count", [1, 15, 16, 17, 31, 33, 127, 128, 129, 77_823, 77_825, 80_001])
def test_face_counts(ctx, port, count):
    check(ctx, port, soup(count, 4.0), f"{count} faces")


# pixel-box limits below, at and above what the pair tables hold for a full CTA (256 pixels a
# box: larger ones overflow into the large-triangle pass)
@pytest.mark.parametrize("limit", [0, 6, 7, 256, 1024, 65536])
@pytest.mark.parametrize("count,edge", [(40, 60.0), (2000, 24.0), (80_000, 14.0), (1_250_000, 9.0)])
def test_pair_tables_overflow(port, limit, count, edge):
    ctx = api.Context(0)
    ctx.set_tuning([limit] * 6)
    sc = soup(count, edge)
    vp = port.camera(sc.camera)[2]
    draws = api.batch_draws(ctx, [sc])
    draws[0].camera = api.Camera.from_matrices(vp, sc.camera.position, sc.camera.viewport)
    expected = port.draw(sc, vp)
    for form in (api.BATCH_PHASED, api.BATCH_PERSISTENT):
        ctx.batch_form = form
        api.draw_batch(ctx, draws)
        got = draws[0].framebuffer.read()
        ctx.sync()
        assert_parity(got, expected, f"limit {limit} form {form}")
    ctx.close()


# spheres that cross one side of the view volume, two at a corner, the near plane, the near
# plane and a side, and triangles that hang over several planes at once: the planes a face
# does not reach are passed over
@pytest.mark.parametrize("target", [(0.0, 0.0, 0.0), (1.1, 0.0, 0.0), (-1.1, 0.2, 0.0), (0.0, 1.0, 0.0), (0.1, -1.0, 0.0),
                                    (0.9, 0.8, 0.0)])
@pytest.mark.parametrize("distance,lon", [(2.2, 48), (1.05, 24), (0.6, 6)])
def test_clip_planes(ctx, port, target, distance, lon):
    sc = W.sphere_scene(width=241, height=163, lon=lon, lat=max(4, lon // 2), shader=W.SHADER_PHONG)
    sc.camera = W.Camera((0.0, 0.0, float(distance)), target, 60.0, float(np.float32(241 / 163)), (0, 0, 241, 163))
    check(ctx, port, sc, f"target {target} distance {distance}")


# frames on both sides of the limit (30 tiles per SM: 4,560 on 152 SMs) between the one-kernel tile
# pass and the scan and shade kernels, with ragged right and top edges, clipped and not
@pytest.mark.parametrize("size", [(1, 1), (15, 17), (1216, 960), (1215, 961), (1301, 977)])
@pytest.mark.parametrize("shader", [W.SHADER_FLAT, W.SHADER_PBR])
@pytest.mark.parametrize("distance", [3.0, 1.3])
def test_tile_passes(ctx, port, size, shader, distance):
    sc = W.sphere_scene(width=size[0], height=size[1], lon=48, lat=24, tex_size=64, shader=shader, distance=distance)
    check(ctx, port, sc, f"{size} shader {shader} distance {distance}")


# more clipped triangles than their records hold (65,536, or 16,384 of the no-allocation draw): the
# winners past them re-run the clipper
@pytest.mark.parametrize("entry,count", [("axr_draw_mesh", 50_000), ("axr_draw_mesh_noalloc", 21_000)])
def test_clipped_records_overflow(ctx, port, entry, count):
    sc = W.soup_scene(count=count, width=96, height=64, seed=33, edge_min=60.0, edge_max=200.0, depth_min=0.12, depth_max=50.0)
    sc.shader = W.Shader(W.SHADER_GOURAUD)
    vp = port.camera(sc.camera)[2]
    fb, mesh = api.Framebuffer(ctx, sc.width, sc.height), api.Mesh.from_workload(ctx, sc.mesh)
    fb.clearColor(0, 0, 0, 255)
    fb.clearDepth()
    api.TiledPipeline(ctx, api.Camera.from_matrices(vp, sc.camera.position, sc.camera.viewport), fb).setShader(api.GouraudShader())
    api.check(getattr(ctx.lib, entry)(ctx.handle, mesh.handle, np.ascontiguousarray(sc.model, np.float32).ctypes.data), ctx.handle)
    got = fb.read()
    ctx.sync()
    assert_parity(got, port.draw(sc, vp), entry)
