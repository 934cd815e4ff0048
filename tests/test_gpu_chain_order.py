"""Kernels that start while the one before them drains: calls enqueued without a wait between them
(mesh update, clears, draw, PNG encode, batch) must leave what the same calls leave one at a time, also from
a captured graph."""
import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def poses(sc, k):
    """k poses of the scene's mesh, each scaled about its origin."""
    m = sc.mesh
    return [(m.positions * np.float32(1.0 - 0.15 * i), m.uvs, m.normals, m.indices, m.tangents, m.bitangents) for i in range(k)]


@pytest.mark.parametrize("width,height", [(64, 48), (333, 201), (1920, 1080)])
def test_frames(ctx, width, height):
    sc = W.sphere_scene(width, height, tex_size=32)
    mesh = api.Mesh.from_workload(ctx, sc.mesh)
    fbs = [api.Framebuffer(ctx, width, height) for _ in range(6)]
    pipe = api.TiledPipeline(ctx)
    pipe.setCamera(api.Camera.from_workload(sc.camera))
    pipe.setShader(api.Shader(sc.shader.kind, tuple(sc.shader.light_direction), tuple(sc.shader.light_color)))

    def frames(wait):
        for fb, pose in zip(fbs, poses(sc, len(fbs))):
            mesh.update(*pose)
            wait()
            fb.clearColor(1, 2, 3, 255)
            wait()
            fb.clearDepth(1.0)
            wait()
            pipe.setFramebuffer(fb)
            pipe.drawMesh(sc.model, mesh)
            wait()
        png = api.PngBatch(ctx)
        png.encode(fbs, 4)
        wait()
        files = png.read()
        return [fb.read() for fb in fbs], [bytes(f) for f in files]

    exp, exp_png = frames(ctx.sync)
    for _ in range(4):
        got, got_png = frames(lambda: None)
        for (gb, gd), (eb, ed) in zip(got, exp):
            assert np.array_equal(gb, eb) and np.array_equal(gd.view(np.uint32), ed.view(np.uint32))
        assert got_png == exp_png


def test_captured(ctx):
    own = api.Context(0)
    sc = W.sphere_scene(333, 201, tex_size=32)
    mesh = api.Mesh.from_workload(own, sc.mesh)
    fb = api.Framebuffer(own, 333, 201)
    scenes = W.batch_scenes(count=6, seed=2, tex_size=32, resolution_scale=0.1)
    draws = api.batch_draws(own, scenes)
    batch = api.Batch(own, draws)
    pipe = api.TiledPipeline(own)
    pipe.setCamera(api.Camera.from_workload(sc.camera))
    pipe.setShader(api.Shader(sc.shader.kind, tuple(sc.shader.light_direction), tuple(sc.shader.light_color)))
    pipe.setFramebuffer(fb)
    own.reserve(mesh.num_faces)

    def work():
        batch.launch()
        fb.clearColor(9, 8, 7, 255)
        fb.clearDepth(1.0)
        pipe.drawMesh(sc.model, mesh)
        batch.launch()

    work()
    own.sync()
    exp = [f.read() for f in [fb] + [d.framebuffer for d in draws]]
    g = api.Graph(own).begin()
    work()
    g.end()
    for _ in range(5):
        g.launch()
    own.sync()
    for f, (eb, ed) in zip([fb] + [d.framebuffer for d in draws], exp):
        gb, gd = f.read()
        assert np.array_equal(gb, eb) and np.array_equal(gd.view(np.uint32), ed.view(np.uint32))
    g.close()
