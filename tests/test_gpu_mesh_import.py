"""Mesh uploads read by the GPU straight from pinned host memory: the arrays, read back exactly, at
vertex and face counts around the kernel's blocks and 16-byte words, for buffers that change between
updates, that are not aligned or only partly pinned (copied as before), and under capture."""
import numpy as np
import pytest
import torch

from axiomr_gb300 import api
from test_gpu_mesh_update import vertices

pytestmark = pytest.mark.gpu


def pin(a, offset=0):
    """A pinned copy of `a`, its first byte `offset` bytes past the allocation's."""
    a = np.ascontiguousarray(a)
    t = torch.empty(a.nbytes + 64, dtype=torch.uint8, pin_memory=True)
    v = t.numpy()[offset:offset + a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    return v, t


def arrays(rng, n, faces, frames):
    f = lambda k: rng.uniform(-1, 1, (n, k)).astype(np.float32)  # noqa: E731
    return [f(3), f(2), f(3), rng.integers(0, n, (faces, 3)).astype(np.uint32), f(3) if frames else None,
            f(3) if frames else None]


def check(ctx, mesh, a):
    p, uv, nrm, idx, t, b = a
    z = np.zeros_like(p)
    exp = np.concatenate([p, uv, nrm, z if t is None else t, z if b is None else b], axis=1)
    assert np.array_equal(vertices(ctx, mesh).view(np.uint32), exp.view(np.uint32))
    got = np.zeros((len(idx), 3), np.uint32)
    api.check(ctx.lib.axr_mesh_read(ctx.handle, mesh.handle, None, got.ctypes.data), ctx.handle)
    assert np.array_equal(got, idx)


@pytest.mark.parametrize("frames", [True, False])
@pytest.mark.parametrize("n,faces", [(1, 1), (3, 2), (255, 3), (256, 4), (257, 5), (8192, 1001), (8193, 16_383),
                                     (131_071, 50_001), (131_073, 43_690), (300_001, 100_003)])
def test_pinned(ctx, n, faces, frames):
    rng = np.random.default_rng(n)
    first = arrays(rng, n, faces, frames)
    mesh = api.Mesh(ctx, *first[:4], tangents=first[4], bitangents=first[5])
    keep, pose = zip(*((None, None) if a is None else pin(a)[::-1] for a in arrays(rng, n, faces, frames)))
    cam = api.Camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 60.0, 1.0, (0, 0, 64, 64))
    draw = api.Draw(mesh, api.Framebuffer(ctx, 64, 64), cam, api.FlatShader())
    for scale in (1.0, 0.5, 0.001):  # the same buffers, other contents
        for buf in pose:
            if buf is not None and buf.dtype == np.float32:
                buf *= np.float32(scale)
        pose[3][...] = rng.integers(0, n, (faces, 3))
        mesh.update(*pose)
        check(ctx, mesh, pose)
        fresh = api.Mesh(ctx, *[np.array(a) for a in pose[:4]])
        assert api.density_class(draw) == api.density_class(api.Draw(fresh, draw.framebuffer, cam, api.FlatShader()))
    made = api.Mesh(ctx, *pose[:4], tangents=pose[4], bitangents=pose[5])  # and at creation
    check(ctx, made, pose)


@pytest.mark.parametrize("which", range(6))
@pytest.mark.parametrize("offset", [None, 4, 8, 16])
def test_mixed(ctx, which, offset):
    """One array in ordinary memory (None) or `offset` bytes past an aligned address."""
    rng = np.random.default_rng(which)
    a = arrays(rng, 1000, 777, True)
    mesh = api.Mesh(ctx, *[np.zeros_like(x) for x in a[:4]], tangents=np.zeros_like(a[4]), bitangents=np.zeros_like(a[5]))
    keep = [pin(x, (offset or 0) if k == which else 0) for k, x in enumerate(a)]
    pose = [x if k == which and offset is None else keep[k][0] for k, x in enumerate(a)]
    mesh.update(*pose)
    check(ctx, mesh, a)


def test_captured():
    own = api.Context(0)
    rng = np.random.default_rng(9)
    a = arrays(rng, 500, 300, True)
    mesh = api.Mesh(own, *a[:4], tangents=a[4], bitangents=a[5])
    keep, pose = zip(*(pin(x)[::-1] for x in a))
    g = api.Graph(own).begin()
    mesh.update(*pose)
    g.end()
    for _ in range(3):
        for buf, x in zip(pose, arrays(rng, 500, 300, True)):
            buf[...] = x
        g.launch()
        own.sync()
        check(own, mesh, pose)
    g.close()
