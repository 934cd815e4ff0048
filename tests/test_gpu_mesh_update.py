"""Mesh updates: the widened arrays, read back exactly, and the bounds computed with them, at vertex
counts around the kernels' blocks and the host / device limit of the bounds, for meshes created from
arrays (all arrays staged at once) and ingested ones (one at a time)."""
import ctypes as C

import numpy as np
import pytest

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def arrays(rng, n, scale):
    f = lambda k: rng.uniform(-scale, scale, (n, k)).astype(np.float32)  # noqa: E731
    return f(3), f(2), f(3), f(3), f(3)


def vertices(ctx, mesh):
    out = np.zeros((mesh.num_vertices, 14), np.float32)
    api.check(ctx.lib.axr_mesh_read(ctx.handle, mesh.handle, out.ctypes.data, None), ctx.handle)
    return out


@pytest.mark.parametrize("frames", [True, False])
@pytest.mark.parametrize("n", [1, 3, 255, 256, 257, 8192, 8193, 131_071, 131_073, 300_001])
def test_update(ctx, n, frames):
    rng = np.random.default_rng(n)
    idx = rng.integers(0, n, (max(1, n // 3), 3)).astype(np.uint32)
    p, uv, nrm, t, b = arrays(rng, n, 1.0)
    mesh = api.Mesh(ctx, p, uv, nrm, idx, tangents=t if frames else None, bitangents=b if frames else None)
    cam = api.Camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 60.0, 1.0, (0, 0, 64, 64))
    draw = api.Draw(mesh, api.Framebuffer(ctx, 64, 64), cam, api.FlatShader())
    for scale in (0.4, 0.9, 0.001):
        p, uv, nrm, t, b = arrays(rng, n, scale)
        mesh.update(p, uv, nrm, idx, t if frames else None, b if frames else None)
        z = np.zeros_like(p)
        exp = np.concatenate([p, uv, nrm, t if frames else z, b if frames else z], axis=1)
        assert np.array_equal(vertices(ctx, mesh).view(np.uint32), exp.view(np.uint32))
        # the bounds a new mesh of these arrays gets on the host give the same density class
        fresh = api.Mesh(ctx, p, uv, nrm, idx)
        assert api.density_class(draw) == api.density_class(api.Draw(fresh, draw.framebuffer, cam, api.FlatShader()))
    ctx.sync()
