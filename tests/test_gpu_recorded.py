"""Draws recorded into a graph: what a replay draws is decided by the vertices it finds on the device,
which may cross the view volume although none did when it was recorded; and draws outside a graph, of a mesh whose
bounds come from the device."""
import dataclasses

import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W

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
