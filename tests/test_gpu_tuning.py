"""The batched form's pixel-box limits: a limit that was set is the one used, whatever the batch's size; and
boxes that the pair tables of the face phase do not hold go to the large-triangle pass. The triangles sent there
are counted from the clip stage's records by the face phase's rules. And the autotuner times its limits in the
batch that they are for."""
import numpy as np
import pytest
import torch

from axiomr_gb300 import api
from axiomr_gb300 import workloads as W
from helpers import assert_parity

pytestmark = pytest.mark.gpu

THREAD_PIXELS, CLIPPED_PIXELS, WARP_PAIRS = 6, 8, 8192  # boxes of a thread, of a clipped triangle; a warp's table


def expected_large(records, width, height, limit, faces_per_cta, faces):
    """Triangles for the large-triangle pass: boxes past the limit, and in each warp those from the first that its
    table does not hold."""
    tag = records[:, 0].view(np.uint32)
    lo = np.maximum(np.floor(records[:, 10:12]), 0).astype(np.int64)
    hi = np.minimum(np.ceil(records[:, 12:14]), [width, height]).astype(np.int64)
    px = np.where((hi > lo).all(axis=1), (hi - lo).prod(axis=1), 0)
    cut = (tag & 8) != 0
    large = int((cut & (px > min(limit, CLIPPED_PIXELS))).sum())
    shared = np.zeros(faces, np.int64)  # by draw-order position: pixels of a box that a group's threads share
    at, px = tag[~cut] >> 4, px[~cut]
    most = max(limit, THREAD_PIXELS)
    large += int((px > most).sum())
    mine = (px > THREAD_PIXELS) & (px <= most)
    shared[at[mine]] = px[mine]
    for first in range(0, faces, faces_per_cta):
        for warp in range(first, min(first + faces_per_cta, faces), 32):
            boxes = shared[warp:min(warp + 32, first + faces_per_cta, faces)]
            past = np.cumsum(boxes) > WARP_PAIRS
            large += int((past & (boxes > 0)).sum())
    return large


def faces_per_cta(form, faces):
    if form == api.BATCH_PERSISTENT:
        return 256
    sms, n = torch.cuda.get_device_properties(0).multi_processor_count, 128
    while n > 16 and faces < 4 * sms * n:
        n //= 2
    return n


def check(port, sc, limit, form):
    """The scene as a batch of one under `limit`: the oracle's frame and the expected large triangles."""
    ctx = api.Context(0)
    ctx.set_tuning([limit] * 6)
    assert ctx.tuning() == [limit] * 6
    vp = port.camera(sc.camera)[2]
    draws = api.batch_draws(ctx, [sc])
    draws[0].camera = api.Camera.from_matrices(vp, sc.camera.position, sc.camera.viewport)
    ctx.batch_form = form
    ctx.stats(True)
    ctx.stats()
    api.draw_batch(ctx, draws)
    assert_parity(draws[0].framebuffer.read(), port.draw(sc, vp), f"limit {limit} form {form}")
    stats = ctx.stats()
    mesh = draws[0].mesh
    records = api.TiledPipeline(ctx).debugTriangles(mesh, sc.model, vp, sc.width, sc.height)
    ctx.close()
    faces = mesh.num_faces
    assert stats["triangles"] == len(records)
    expected = expected_large(records, sc.width, sc.height, limit, faces_per_cta(form, faces), faces)
    assert stats["large"] == min(expected, max(65536, faces))  # the list's entries: those past it are rasterised at once
    return stats


def soup(count, edge, edge_max=None, width=331, height=213, seed=21):
    return W.soup_scene(count=count, width=width, height=height, seed=seed, edge_min=edge, edge_max=edge_max or edge + 0.01,
                        depth_min=1.0, depth_max=50.0)


# boxes of at most 35 x 32 pixels, six faces of them: within a warp's table, whatever the limit
@pytest.mark.parametrize("form", [api.BATCH_PHASED, api.BATCH_PERSISTENT])
@pytest.mark.parametrize("limit", [0, 64, 256, 2048, 65536])
def test_limit_is_used(port, form, limit):
    s = check(port, soup(6, 30.0), limit, form)
    few = check(port, soup(6, 30.0), 0, form)["large"]
    assert (s["large"] < few) == (limit >= 2048)


# a warp's 32 (or, of few faces, 16) boxes together past 8,192 pixels, single boxes past the whole table, boxes
# of all sizes mixed; the cut falls anywhere among them
@pytest.mark.parametrize("form", [api.BATCH_PHASED, api.BATCH_PERSISTENT])
@pytest.mark.parametrize("limit", [256, 1024, 4096, 65536])
@pytest.mark.parametrize("count,edge,edge_max", [(40, 60.0, None), (300, 24.0, 60.0), (2000, 2.0, 100.0), (64, 90.0, 200.0),
                                                 (80_000, 20.0, 40.0)])
def test_pair_tables_overflow(port, form, limit, count, edge, edge_max):
    s = check(port, soup(count, edge, edge_max), limit, form)
    assert 0 < s["large"] <= s["triangles"]


def test_autotune_times_the_whole_batch():
    """Each launch of the search for the limits draws the whole batch. With one repeat every setting is launched twice:
    the binned form's 21 a class, all classes together once the batch; three forms; the limits, five per class
    of the batch and the table as it was."""
    ctx = api.Context(0)
    draws = api.batch_draws(ctx, W.batch_scenes(count=24, seed=5, tex_size=32, resolution_scale=0.25))
    classes = len({api.density_class(d) for d in draws})
    assert classes >= 3
    ctx.batch_form = api.BATCH_PHASED
    batch = api.Batch(ctx, draws)
    ctx.stats(True)
    ctx.stats()
    batch.launch()
    whole = ctx.stats()["triangles"]
    api.autotune(ctx, draws, repeats=1)
    launches = ctx.stats()["triangles"] / whole
    # (the search ends with the forms where the binned one, which has no such limits, is the fastest)
    assert launches == 2 * (21 + 3 + (0 if ctx.batch_form == api.BATCH_BINNED else 1 + 5 * classes))
    batch.close()
    ctx.close()
