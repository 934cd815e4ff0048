"""Draws and mesh updates recorded into a graph: what a replay draws is decided by the vertices it finds
on the device, which may cross the view volume although none did when it was recorded, and an update that a
graph may repeat at any time says nothing about the vertices of a later draw. And draws outside a graph, of a
mesh whose bounds come from the device."""
import dataclasses

import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W
from test_gpu_mesh_import import pin

pytestmark = pytest.mark.gpu

# in view; across the left, right and top planes; across the near plane (but for the coarsest mesh); in view again
SHIFTS = [(0.0, 0.0, 0.0), (-1.4, 0.0, 0.0), (1.3, 0.9, 0.0), (0.0, 0.0, 1.901), (0.0, 0.0, -0.5)]


class Frame:
    """A context of its own with one mesh and one frame of the sphere scene."""

    def __init__(self, lon, size=(241, 163), shader=W.SHADER_BLINN_PHONG, entry="axr_draw_mesh"):
        self.ctx = api.Context(0)
        self.sc = W.sphere_scene(width=size[0], height=size[1], lon=lon, lat=lon // 2, tex_size=32, shader=shader)
        self.mesh = api.Mesh.from_workload(self.ctx, self.sc.mesh)
        self.fb = api.Framebuffer(self.ctx, *size)
        self.pipe = api.TiledPipeline(self.ctx, api.Camera.from_workload(self.sc.camera), self.fb)
        sh = self.sc.shader
        self.pipe.setShader(api.Shader(sh.kind, tuple(sh.light_direction), tuple(sh.light_color)))
        self.model = np.ascontiguousarray(self.sc.model, np.float32)
        self.entry = getattr(self.ctx.lib, entry)
        self.ctx.reserve(self.mesh.num_faces)

    def draw(self):
        b, g, r, a = self.sc.clear_bgra
        self.fb.clearColor(r, g, b, a)
        self.fb.clearDepth()
        api.check(self.entry(self.ctx.handle, self.mesh.handle, self.model.ctypes.data), self.ctx.handle)

    def pose(self, shift):
        m = self.sc.mesh
        return [m.positions + np.float32(shift), m.uvs, m.normals, m.indices, m.tangents, m.bitangents]

    def expected(self, ctx, shift):
        """The same frame of a mesh created with these positions, drawn at once."""
        sc = dataclasses.replace(self.sc, mesh=dataclasses.replace(self.sc.mesh, positions=self.pose(shift)[0]))
        return api.render_scene(ctx, sc)

    def check(self, ctx, shift, what):
        self.ctx.sync()
        (gb, gd), (eb, ed) = self.fb.read(), self.expected(ctx, shift)
        assert np.isfinite(ed).any()
        assert np.array_equal(gd.view(np.uint32), ed.view(np.uint32)) and np.array_equal(gb, eb), (what, shift)


@pytest.mark.parametrize("lon", [32, 128])  # 561 and 8,385 vertices: bounds on the host and on the device
@pytest.mark.parametrize("size", [(241, 163), (1301, 977)])  # either tile pass
@pytest.mark.parametrize("shader", [W.SHADER_BLINN_PHONG, W.SHADER_PBR])
def test_recorded_draw(ctx, lon, size, shader):
    f = Frame(lon, size, shader)
    f.draw()
    f.ctx.sync()
    g = api.Graph(f.ctx).begin()
    f.draw()
    g.end()
    for shift in SHIFTS:
        f.mesh.update(*f.pose(shift))
        g.launch()
        f.check(ctx, shift, "replayed")
    g.close()


@pytest.mark.parametrize("lon", [32, 128])
@pytest.mark.parametrize("pinned", [True, False])  # one kernel reads the arrays, or copies do
def test_recorded_update(ctx, lon, pinned):
    """An update recorded with the draw behind it, then a graph with the update alone and draws outside it."""
    f = Frame(lon)
    keep = [pin(a) if a is not None else (None, None) for a in f.pose(SHIFTS[0])]
    pose = [k[0] for k in keep]
    if not pinned:  # (a pageable copy cannot be recorded; one array a word off an aligned address can)
        keep[2] = pin(pose[2], 4)
        pose[2] = keep[2][0]
    f.mesh.update(*pose)  # allocates what later updates need
    f.draw()
    f.ctx.sync()
    both, alone = api.Graph(f.ctx), api.Graph(f.ctx)
    both.begin()
    f.mesh.update(*pose)
    f.draw()
    both.end()
    alone.begin()
    f.mesh.update(*pose)
    alone.end()
    cls = api.density_class(api.Draw(f.mesh, f.fb, api.Camera.from_workload(f.sc.camera), api.FlatShader()))
    for shift in SHIFTS:
        pose[0][...] = f.pose(shift)[0]
        both.launch()
        f.check(ctx, shift, "update and draw replayed")
    for shift in SHIFTS:
        pose[0][...] = f.pose(shift)[0]
        alone.launch()
        f.draw()
        f.check(ctx, shift, "update replayed, then drawn")
    # planning goes by the bounds known last, and a batch draws the mesh as it is
    draw = api.Draw(f.mesh, f.fb, api.Camera.from_workload(f.sc.camera), api.Shader(f.sc.shader.kind, tuple(
        f.sc.shader.light_direction), tuple(f.sc.shader.light_color)), f.sc.model, (0, 0, 0, 255), float("inf"))
    assert api.density_class(draw) == cls
    api.draw_batch(f.ctx, [draw])
    f.check(ctx, SHIFTS[-1], "batch")
    both.close()
    alone.close()


@pytest.mark.parametrize("lon", [130, 256])
def test_update_across_planes(ctx, lon):
    """Updates outside a graph of a mesh whose bounds come from the device (above 8,192 vertices), drawn while
    they are under way and after they are known: the clip pass runs where a face needs it."""
    f = Frame(lon)
    assert f.mesh.num_vertices > 8192
    for shift in SHIFTS + SHIFTS[::-1]:
        f.mesh.update(*f.pose(shift))
        f.draw()  # the bounds may still be under way
        f.check(ctx, shift, "drawn at once")
        f.draw()  # now they are known
        f.check(ctx, shift, "drawn later")


@pytest.mark.parametrize("shader", [W.SHADER_FLAT, W.SHADER_PBR])
def test_recorded_noalloc_draw(ctx, shader):
    """The draw without allocations, a chain of kernels behind a memset and before an ordinary one, recorded."""
    f = Frame(64, shader=shader, entry="axr_draw_mesh_noalloc")
    f.draw()  # looks the device array up
    f.ctx.sync()
    g = api.Graph(f.ctx).begin()
    f.draw()
    f.draw()
    g.end()
    for shift in SHIFTS:
        f.mesh.update(*f.pose(shift))
        g.launch()
        g.launch()
        f.check(ctx, shift, "replayed")
    g.close()
