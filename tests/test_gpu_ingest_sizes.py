"""OBJ ingest at corner counts around its scans' blocks, with the bounds' effect, faults reported as
before, and meshes that outlive the context they were ingested on."""
import ctypes as C

import numpy as np
import pytest

import objfile
from axiomr_gb300 import api
from helpers import same_bits
from test_gpu_ingest import ingest, read

pytestmark = pytest.mark.gpu


def fan_model(n_poly, size, seed):
    """n_poly polygons of 2 to `size` corners over a shared pool."""
    rng = np.random.default_rng(seed)
    n = max(3, n_poly // 2)
    sizes = rng.integers(2, size + 1, n_poly).astype(np.uint32) if size > 3 else np.full(n_poly, 3, np.uint32)
    corners = np.stack([rng.integers(0, n, int(sizes.sum())), rng.integers(-1, n, int(sizes.sum())),
                        rng.integers(-1, n, int(sizes.sum()))], axis=1).astype(np.int32)
    nrm = rng.normal(size=(n, 3)).astype(np.float32)
    return {"positions": rng.uniform(-1, 1, (n, 3)).astype(np.float32), "uvs": rng.uniform(0, 1, (n, 2)).astype(np.float32),
            "normals": nrm / np.linalg.norm(nrm, axis=1, keepdims=True), "corners": corners, "polygon_sizes": sizes,
            "num_faces": int(np.maximum(sizes.astype(np.int64) - 2, 0).sum())}


@pytest.mark.parametrize("n_poly,size", [(1, 3), (341, 3), (342, 3), (1023, 5), (1024, 5), (1025, 6), (2049, 3), (40_000, 7)])
def test_sizes_match_port(ctx, port, n_poly, size):
    parsed = fan_model(n_poly, size, n_poly)
    h = ingest(ctx, parsed)
    verts, faces = read(ctx, h)
    ctx.lib.axr_mesh_destroy(ctx.handle, h)
    pv, pf = port.obj_ingest(parsed)
    assert same_bits(verts, pv) and np.array_equal(faces, pf)


@pytest.mark.parametrize("where,value", [(0, -1), (7, 10_000), (1500, -5), (2999, 500)])
def test_bad_corner_is_named(ctx, where, value):
    parsed = fan_model(1000, 3, 5)
    parsed["corners"][where, 0] = value
    with pytest.raises(api.AxrError, match=f"corner {where} names position {value} of 500"):
        ingest(ctx, parsed)
    good = fan_model(1000, 3, 5)  # and the context goes on
    h = ingest(ctx, good)
    ctx.lib.axr_mesh_destroy(ctx.handle, h)


def test_mesh_outlives_its_context(ctx, port):
    parsed = objfile.parse_obj(objfile.sphere_obj(64, 32))
    other = api.Context(0)
    h = ingest(other, parsed)
    other.close()
    for _ in range(3):  # the pool's memory is not handed out again while the mesh lives
        ctx.lib.axr_mesh_destroy(ctx.handle, ingest(ctx, parsed))
    verts, faces = read(ctx, h)
    pv, pf = port.obj_ingest(parsed)
    assert same_bits(verts, pv) and np.array_equal(faces, pf)
    ctx.lib.axr_mesh_destroy(None, h)
