"""The calls a user of the renderer makes, as cases that a timing harness can run.

A case is a plain dict; `listed()` gives the fixed ones, `draw(rng)` one more of the same
ranges. `prepare(case, seed)` makes what a program has in hand before the call (meshes,
textures, framebuffers, a planned batch, a running server), `run(state)` is one pass through
the public entry points, `work(case)` what the pass cannot do without, and `exact(case, seed)`
the depth planes from a float64 rasteriser (colour is bytes and has no such value).

Kinds of case:
  frame    one frame as a frame loop draws it: clearColor, clearDepth, setCamera /
           setFramebuffer / setShader, drawMesh; with "graph" the recorded frame replayed
           from a CUDA graph (the context's scratch reserved beforehand)
  animate  the same frame after the mesh's vertices were replaced from pinned host memory
  batch    a planned batch (Batch.launch), one framebuffer per draw
  oneshot  draw_batch on a host draw table: planned and uploaded on every call
  farm     a planned batch whose frames are encoded to PNG files in device memory
  png      one finished frame to a PNG file in pinned host memory
  ingest   an OBJ model's pools and corners to a device mesh, drawn once, released
  serve    requests through the serving loop, colour planes back in pinned host memory
Launch forms and tuning tables are the library's defaults.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from axiomr_gb300 import _lib, api
from axiomr_gb300 import workloads as W

SHADERS = {"flat": W.SHADER_FLAT, "phong": W.SHADER_PHONG, "pbr": W.SHADER_PBR, "blinn": W.SHADER_BLINN_PHONG,
           "gouraud": W.SHADER_GOURAUD}
# FP32 operations per shaded pixel, counted in the shaders' formulas
SHADE_OPS = {"flat": 40, "phong": 220, "pbr": 300, "blinn": 129, "gouraud": 30}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest frame: an icon-sized preview, where launches and latency are everything
        frame("icon", "sphere", "flat", 96, 96, size=16, tex=16, far=1.0),
        # the plain small configuration (4k triangles, 512x512), replayed from a CUDA graph
        frame("sphere", "sphere", "blinn", 512, 512, size=64, tex=256, far=1.0, graph=True),
        # a close-up of a textured model in a window of no particular size: five maps, large
        # triangles, the frame's borders cut through the model, no 16-byte row pitch
        frame("closeup_pbr", "sphere", "pbr", 1365, 767, size=128, tex=1024, distance=1.6, far=1.0),
        # the plain large-mesh configuration: 2M triangles at 1920x1080
        frame("terrain", "terrain", "blinn", 1920, 1080, size=1024, tex=2048, far=1.0),
        # the small-triangle / overdraw stress configuration: 200k triangles at 3840x2160
        frame("soup", "soup", "gouraud", 3840, 2160, size=200_000, tex=0, far=1.0),
        # a deforming mesh: vertices uploaded, then drawn, every frame
        dict(name="animated", kind="animate", scene="terrain", shader="phong", width=1280, height=720, size=256,
             tex=512, distance=2.5, far=1.0, graph=False),
        # a sheet of views rendered together (the mixed batch's meshes and resolutions)
        dict(name="batch", kind="batch", count=30, shader="blinn", tex=1024, scale=1.0, odd=False),
        # a host draw list rendered with one call: every shader, resolutions of any width
        dict(name="oneshot", kind="oneshot", count=20, shader="all", tex=256, scale=0.25, odd=True),
        # the mixed batch of 512 draws delivered as PNG files
        dict(name="farm", kind="farm", count=512, shader="blinn", tex=1024, scale=1.0, odd=False, channels=3),
        # a screenshot of one frame
        dict(name="screenshot", kind="png", width=1920, height=1080, channels=4),
        # opening a model of 65k triangles and drawing its first frame
        dict(name="open_model", kind="ingest", lon=256, shader="pbr", width=800, height=600, tex=256),
        # a burst of requests at the serving loop
        dict(name="serve", kind="serve", requests=32, assets=6, size=20_000, width=640, height=360, batch=16),
    ]


def frame(name, scene, shader, width, height, size, tex, distance=3.0, far=None, graph=False):
    """A frame case; far: the clearDepth value (None: +inf)."""
    return dict(name=name, kind="frame", scene=scene, shader=shader, width=width, height=height, size=size, tex=tex,
                distance=distance, far=far, graph=graph)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["batch"] * 2 + ["oneshot", "farm", "png", "animate", "ingest", "serve"])
    if kind in ("frame", "animate"):
        scene = "terrain" if kind == "animate" else rng.choice(["sphere", "sphere", "terrain", "soup"])
        width = _log(rng, 64, 3840 if scene == "soup" else 1920)
        height = max(48, int(width * rng.uniform(0.5, 1.0)))
        c = frame("", scene, "gouraud" if scene == "soup" else rng.choice(["flat", "phong", "pbr", "blinn"]),
                  width, min(height, 2160),
                  size={"sphere": 2 * _log(rng, 4, 256), "terrain": _log(rng, 16, 256 if kind == "animate" else 1024),
                        "soup": _log(rng, 500, 200_000)}[scene],
                  tex=_log(rng, 16, 1024), distance=round(rng.uniform(2.2, 3.5) if scene == "terrain" else rng.uniform(1.5, 6.0), 3),
                  far=rng.choice([None, 1.0]), graph=kind == "frame" and rng.random() < 0.4)
        c.update(kind=kind)
        del c["name"]
        return c
    if kind in ("batch", "oneshot"):
        return dict(kind=kind, count=_log(rng, 2, 32), shader=rng.choice(["blinn", "phong", "flat", "pbr", "all"]),
                    tex=_log(rng, 32, 1024), scale=round(math.exp(rng.uniform(math.log(0.125), 0.0)), 4),
                    odd=rng.random() < 0.5)
    if kind == "farm":
        return dict(kind=kind, count=_log(rng, 16, 512), shader=rng.choice(["blinn", "blinn", "phong"]),
                    tex=_log(rng, 64, 1024), scale=round(rng.uniform(0.25, 0.9), 4), odd=rng.random() < 0.3,
                    channels=rng.choice([3, 4]))
    if kind == "png":
        width = _log(rng, 64, 3840)
        return dict(kind=kind, width=width, height=max(48, int(width * rng.uniform(0.4, 1.0))), channels=rng.choice([3, 4]))
    if kind == "ingest":
        return dict(kind=kind, lon=2 * _log(rng, 8, 128), shader=rng.choice(["phong", "pbr", "blinn"]),
                    width=_log(rng, 200, 1920), height=_log(rng, 200, 1080), tex=_log(rng, 32, 512))
    return dict(kind="serve", requests=_log(rng, 4, 64), assets=rng.randint(1, 8), size=_log(rng, 500, 40_000),
                width=_log(rng, 128, 1280), height=_log(rng, 128, 720), batch=rng.choice([4, 16, 64]))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=300)
def _sphere_parts(lon, lat):
    return W.uv_sphere(lon, lat)


def _material(shader, tex, seed):
    mat = W.Material(specular_exponent=1.0)
    if shader not in ("flat", "gouraud"):
        mat.diffuse = W.noise_texture(tex, seed=seed)
    if shader in ("phong", "pbr"):
        mat.bump = W.noise_texture(tex, seed=seed + 1)
    if shader == "pbr":
        mat.metallic, mat.roughness, mat.ao = (W.noise_texture(tex, seed=seed + k) for k in (2, 3, 4))
    return mat


def _mesh(parts, mat):
    pos, uv, nrm, tan, bit, idx = parts
    return W.Mesh(pos, uv, nrm, tan, bit, idx, np.asarray([[0, idx.shape[0], 0]], np.uint32), [mat])


def _light(shader):
    return (5.6, 5.6, 5.6) if shader == "pbr" else (0.6, 0.6, 0.6)


def _scene(c, seed):
    """The W.Scene of a frame or animate case: the seed moves the camera and makes the textures
    (and the terrain and the soup)."""
    u = W.uniform(seed, 4, stream=9)
    w, h = c["width"], c["height"]
    shader = W.Shader(SHADERS[c["shader"]], (-0.3, -0.8, -0.52), _light(c["shader"]))
    if c["scene"] == "soup":
        sc = W.soup_scene(c["size"], w, h, seed=seed % 1_000_003 + 4)
        sc.shader = shader
        return sc
    mat = _material(c["shader"], c["tex"], 1000 + 16 * (seed % 1_000_003))
    if c["scene"] == "sphere":
        parts = _sphere_parts(c["size"], max(4, c["size"] // 2))
        cam = W.orbit_camera(c["distance"], 40.0 * (u[0] - 0.5), 360.0 * u[1], w, h)
    else:
        parts = W.heightfield(c["size"], seed=seed % 1_000_003 + 2)
        cam = W.orbit_camera(c["distance"], 30.0 + 8.0 * (u[0] - 0.5), 30.0 * (u[1] - 0.5), w, h)
    return W.Scene(c["scene"], _mesh(parts, mat), cam, shader, w, h)


def _plan(c):
    """The draws of a batch case: W.batch_plan's meshes and resolutions, scaled (odd: of any
    width), the same for every seed; the seed turns the cameras."""
    kinds = [k for k in SHADERS if k != "gouraud"] if c["shader"] == "all" else [c["shader"]]
    out = []
    for k, d in enumerate(W.batch_plan(c["count"], seed=5)):
        w, h = max(16, int(d.width * c["scale"])), max(16, int(d.height * c["scale"]))
        if c["odd"]:
            w, h = w + (7 * k) % 13, h + (5 * k) % 11
        out.append((d, w, h, kinds[k % len(kinds)]))
    return out


def _batch_scenes(c, seed):
    texs, scenes, meshes = {}, [], {}
    u = W.uniform(seed, 3 * c["count"], stream=11).reshape(-1, 3)
    for k, (d, w, h, kind) in enumerate(_plan(c)):
        if (d.texture, kind) not in texs:
            texs[d.texture, kind] = _material(kind, c["tex"], 5000 + 97 * (seed % 1_000_003) + 8 * d.texture)
        if (d.lon, d.texture, kind) not in meshes:
            meshes[d.lon, d.texture, kind] = _mesh(_sphere_parts(d.lon, d.lat), texs[d.texture, kind])
        p = np.linalg.norm(d.camera.position)
        cam = W.orbit_camera(float(p), -60.0 + 120.0 * u[k, 0], 360.0 * u[k, 1], w, h)
        scenes.append(W.Scene(f"draw{k}", meshes[d.lon, d.texture, kind], cam,
                              W.Shader(SHADERS[kind], (-0.3, -0.8, -0.52), _light(kind)), w, h))
    return scenes


def _obj(c, seed):
    """An OBJ sphere of quads as a host parser hands it over: v / vt / vn pools and face-line
    corners. The seed scales the model's axes."""
    lon, lat = c["lon"], c["lon"] // 2
    u = 0.8 + 0.2 * W.uniform(seed, 3, stream=13)
    i, j = np.meshgrid(np.arange(lat + 1), np.arange(lon + 1), indexing="ij")
    th, ph = np.pi * i / lat, 2 * np.pi * j / lon
    unit = np.stack([np.sin(th) * np.cos(ph), np.cos(th), -np.sin(th) * np.sin(ph)], -1).reshape(-1, 3)
    nrm = unit / u
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    uv = np.stack([j / lon, 1.0 - i / lat], -1).reshape(-1, 2)
    a = (np.arange(lat)[:, None] * (lon + 1) + np.arange(lon)[None, :]).reshape(-1)
    quad = np.stack([a, a + lon + 1, a + lon + 2, a + 1], 1).reshape(-1)
    corners = np.repeat(quad[:, None], 3, axis=1)
    return {"positions": np.ascontiguousarray(unit * u, np.float32), "uvs": np.ascontiguousarray(uv, np.float32),
            "normals": np.ascontiguousarray(nrm, np.float32), "corners": np.ascontiguousarray(corners, np.int32),
            "sizes": np.full(lon * lat, 4, np.uint32), "faces": 2 * lon * lat}


# ------------------------------------------------------------------ states
@functools.lru_cache(maxsize=1)
def _context():
    """The program's context: one for all its meshes, framebuffers and batches."""
    return api.Context(0)


class _Plane:
    """A device array for torch: a tensor made from it keeps the owner of the memory alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _planes(fb):
    """A framebuffer's colour and depth planes as tensors on its own memory."""
    c, d = C.c_void_p(), C.c_void_p()
    api.check(_lib.load().axr_framebuffer_device_pointers(fb.handle, C.byref(c), C.byref(d)))
    return {"bgra": torch.as_tensor(_Plane(fb, c.value, (fb.height, fb.width, 4), "|u1"), device="cuda"),
            "depth": torch.as_tensor(_Plane(fb, d.value, (fb.height, fb.width), "<f4"), device="cuda")}


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
    return t, t.numpy()


class State:
    """What the program keeps; `go` is one pass."""

    def __init__(self, go, **kept):
        self.go, self.kept = go, kept


def _frame_pass(pipe, fb, cam, shader, mesh, model, far):
    fb.clearColor(0, 0, 0, 255)
    fb.clearDepth(far)
    pipe.setCamera(cam)
    pipe.setFramebuffer(fb)
    pipe.setShader(shader)
    pipe.drawMesh(model, mesh)


def _api_shader(sh):
    return api.Shader(sh.kind, tuple(sh.light_direction), tuple(sh.light_color))


def _prepare_frame(c, seed):
    ctx = api.Context(0) if c["graph"] else _context()  # a recorded frame has scratch of its own
    sc = _scene(c, seed)
    mesh = api.Mesh.from_workload(ctx, sc.mesh)
    fb = api.Framebuffer(ctx, sc.width, sc.height)
    far = math.inf if c["far"] is None else c["far"]
    args = (api.TiledPipeline(ctx), fb, api.Camera.from_workload(sc.camera), _api_shader(sc.shader), mesh, sc.model, far)
    out = _planes(fb)
    if c["graph"]:
        ctx.reserve(mesh.num_faces)
        _frame_pass(*args)
        ctx.sync()
        graph = api.Graph(ctx).begin()
        _frame_pass(*args)
        graph.end()

        def go():
            graph.launch()
            return out
    elif c["kind"] == "animate":
        m = sc.mesh
        keep, pose = zip(*(_pinned(a) for a in (m.positions, m.uvs, m.normals, m.indices, m.tangents, m.bitangents)))

        def go(keep=keep):
            mesh.update(*pose)
            _frame_pass(*args)
            return out
    else:
        def go():
            _frame_pass(*args)
            return out
    return State(go, args=args, ctx=ctx)


def _prepare_batch(c, seed):
    ctx = _context()
    scenes = _batch_scenes(c, seed)
    draws = api.batch_draws(ctx, scenes)
    for k, d in enumerate(draws):
        d.clear_depth = 1.0
        if c["kind"] == "oneshot" and k % 4 == 3:
            d.clear_color = None  # drawn over the plane's earlier content
    if c["kind"] == "oneshot":
        table = api.draw_table(draws)
        out = [_planes(d.framebuffer) for d in draws]

        def go():
            api.draw_batch(ctx, table)
            return out
        return State(go, draws=draws)
    batch = api.Batch(ctx, draws)
    if c["kind"] == "batch":
        out = [_planes(d.framebuffer) for d in draws]

        def go():
            batch.launch()
            return out
        return State(go, draws=draws)
    # farm: every file in one device buffer, at the offsets its worst-case sizes give
    n, ch = len(draws), c["channels"]
    bounds = [api.png_bound(d.framebuffer.width, d.framebuffer.height, ch) for d in draws]
    at = np.concatenate([[0], np.cumsum([(b + 255) // 256 * 256 for b in bounds])])
    files = torch.zeros(int(at[-1]), dtype=torch.uint8, device="cuda")
    sizes = torch.zeros(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    fbs = (C.c_void_p * n)(*[d.framebuffer.handle for d in draws])
    outs = (C.c_void_p * n)(*[files.data_ptr() + int(a) for a in at[:-1]])
    caps = (C.c_uint64 * n)(*bounds)

    def go():
        batch.launch()
        api.check(ctx.lib.axr_framebuffers_encode_png(ctx.handle, n, fbs, ch, outs, caps, C.c_void_p(sizes.data_ptr())),
                  ctx.handle)
        return {"files": files, "sizes": sizes}
    return State(go, draws=draws, batch=batch)


def _prepare_png(c, seed):
    """A finished frame: a textured sphere before a plain background."""
    s = _prepare_frame(frame("", "sphere", "blinn", c["width"], c["height"], size=64, tex=512), seed)
    s.go()
    s.kept["ctx"].sync()
    fb = s.kept["args"][1]
    png = api.PngBatch(s.kept["ctx"])
    handles = (C.c_void_p * 1)(fb.handle)
    file, view = _pinned(np.zeros(api.png_bound(fb.width, fb.height, c["channels"]), np.uint8))
    ptrs, caps = (C.c_void_p * 1)(view.ctypes.data), (C.c_uint64 * 1)(view.nbytes)

    def go():
        png.encode(handles, c["channels"])
        size = png.sizes()
        png.read_into(ptrs, caps)
        return {"file": file, "size": size}
    return State(go, frame=s)


def _prepare_ingest(c, seed):
    ctx, o = _context(), _obj(c, seed)
    tex = {}
    mat = _material(c["shader"], c["tex"], 1000 + 16 * (seed % 1_000_003))
    maps = {f: api.Texture(ctx, getattr(mat, f)) for f in ("diffuse", "bump", "metallic", "roughness", "ao")
            if getattr(mat, f) is not None}
    mats = (_lib.MaterialDesc * 1)(api.Material(**maps).desc())
    groups = (_lib.GroupDesc * 1)(_lib.GroupDesc(0, o["faces"], 0))
    desc = _lib.ObjDesc(len(o["positions"]), o["positions"].ctypes.data, len(o["uvs"]), o["uvs"].ctypes.data,
                        len(o["normals"]), o["normals"].ctypes.data, len(o["corners"]), o["corners"].ctypes.data,
                        len(o["sizes"]), o["sizes"].ctypes.data, 1, C.cast(groups, C.c_void_p), 1,
                        C.cast(mats, C.c_void_p))
    fb = api.Framebuffer(ctx, c["width"], c["height"])
    cam, shader, pipe = api.Camera.from_workload(_obj_camera(c, seed)), api.Shader(
        SHADERS[c["shader"]], (-0.3, -0.8, -0.52), _light(c["shader"])), api.TiledPipeline(ctx)
    model = np.eye(4, dtype=np.float32).reshape(16)
    out = _planes(fb)

    def go():
        h = C.c_void_p()
        api.check(ctx.lib.axr_mesh_create_from_obj(ctx.handle, C.byref(desc), C.byref(h)), ctx.handle)
        fb.clearColor(0, 0, 0, 255)
        fb.clearDepth(1.0)
        pipe.setCamera(cam)
        pipe.setFramebuffer(fb)
        pipe.setShader(shader)
        api.check(ctx.lib.axr_draw_mesh(ctx.handle, h, model.ctypes.data), ctx.handle)
        ctx.lib.axr_mesh_destroy(ctx.handle, h)
        return out
    return State(go, obj=o, maps=maps, mats=mats, groups=groups, tex=tex)


def _obj_camera(c, seed):
    u = W.uniform(seed, 2, stream=15)
    return W.orbit_camera(2.2, 40.0 * (u[0] - 0.5), 360.0 * u[1], c["width"], c["height"])


def _prepare_serve(c, seed):
    """A server with registered assets (soups drawn with Gouraud, and a textured sphere every
    third request) and the burst of requests, their colour planes one after another in one
    pinned buffer."""
    w, h, n = c["width"], c["height"], c["requests"]
    srv = api.Server(0, max_batch=c["batch"])
    soups = [W.soup_scene(c["size"], w, h, seed=(seed + k) % 1_000_003 + 4, depth_min=1.0) for k in range(c["assets"])]
    sphere = W.sphere_scene(w, h, tex_seed=seed % 1_000_003 + 1)
    ids = [(srv.add_mesh(s.mesh), s) for s in soups]
    sid = srv.add_mesh(sphere.mesh)
    u = W.uniform(seed, 2 * n, stream=17).reshape(n, 2)
    reqs = []
    for k in range(n):
        if k % 3 == 2:
            cam = W.orbit_camera(2.5, 60.0 * (u[k, 0] - 0.5), 360.0 * u[k, 1], w, h)
            reqs.append((sid, api.Camera.from_workload(cam), _api_shader(sphere.shader)))
        else:
            i, s = ids[int(u[k, 0] * len(ids))]
            reqs.append((i, api.Camera.from_workload(s.camera), _api_shader(s.shader)))
    frames, view = _pinned(np.zeros((n, h, w, 4), np.uint8))

    def go():
        tickets = [srv.submit(i, cam, sh, w, h, out_bgra=view[k]) for k, (i, cam, sh) in enumerate(reqs)]
        for t in tickets:
            r = srv.wait(t)
            if r["status"] != 0:
                raise RuntimeError(f"request failed with status {r['status']}")
        return frames
    return State(go, srv=srv, frames=frames)


PREPARE = {"frame": _prepare_frame, "animate": _prepare_frame, "batch": _prepare_batch, "oneshot": _prepare_batch,
           "farm": _prepare_batch, "png": _prepare_png, "ingest": _prepare_ingest, "serve": _prepare_serve}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def run(state):
    return state.go()


# ------------------------------------------------------------------ the least work of a pass
def _mesh_size(scene, size):
    """(vertices, faces) of a scene's mesh."""
    if scene == "sphere":
        lat = max(4, size // 2)
        return (lat + 1) * (size + 1), 2 * size * (lat - 1)
    return (size * size, 2 * (size - 1) ** 2) if scene == "terrain" else (3 * size, size)


def _covered(scene, width, height, size, distance=3.0):
    """Roughly the pixels a scene covers (60 degrees field of view)."""
    if scene == "soup":
        return min(width * height, size * 2.6)  # mean area of its triangles
    if scene == "terrain":
        return 0.45 * width * height
    if distance <= 1.001:
        return width * height
    r = height / 2 / math.tan(math.radians(30.0)) / math.sqrt(distance * distance - 1.0)
    return min(width * height, math.pi * r * r)


def _frame_work(scene, shader, width, height, size, tex, distance=3.0):
    """Mesh and texels read once, both planes written once; the shader on each covered pixel
    and the transform of each vertex."""
    v, f = _mesh_size(scene, size)
    px = _covered(scene, width, height, size, distance)
    maps = {"flat": 0, "gouraud": 0, "blinn": 1, "phong": 2, "pbr": 5}[shader]
    per_vertex = 60 if shader in ("phong", "pbr") else 24 if shader == "flat" else 20 if shader == "gouraud" else 32
    return (v * per_vertex + f * 12 + width * height * 8 + maps * 4 * min(tex * tex, px),
            v * 60 + f * 40 + px * (SHADE_OPS[shader] + 30))


def work(case):
    c, k = case, case["kind"]
    if k in ("frame", "animate"):
        b, f = _frame_work(c["scene"], c["shader"], c["width"], c["height"], c["size"], c["tex"], c["distance"])
        if k == "animate":  # the pose is read on the host and written on the device besides
            v, nf = _mesh_size(c["scene"], c["size"])
            b += 56 * v + 12 * nf
    elif k in ("batch", "oneshot", "farm"):
        b = f = 0.0
        for d, w, h, kind in _plan(c):
            db, df = _frame_work("sphere", kind, w, h, d.lon, c["tex"], float(np.linalg.norm(d.camera.position)))
            b, f = b + db, f + df
            if k == "farm":  # the colour plane read, a file of about 15% of its pixels' bytes written
                b += w * h * 4 + 0.15 * c["channels"] * w * h
    elif k == "png":
        b, f = c["width"] * c["height"] * (4 + 0.25 * c["channels"]), c["width"] * c["height"] * 10
    elif k == "ingest":
        lon, lat = c["lon"], c["lon"] // 2
        v, nf = (lon + 1) * (lat + 1), 2 * lon * lat
        b = v * 32 + 4 * lon * lat * 12 + v * 56 + nf * 12  # pools and corners in, mesh out
        db, f = _frame_work("sphere", c["shader"], c["width"], c["height"], lon, c["tex"], 2.2)
        b += db
    else:
        b = f = 0.0
        for i in range(c["requests"]):
            scene, size = ("sphere", 64) if i % 3 == 2 else ("soup", c["size"])
            db, df = _frame_work(scene, "blinn" if scene == "sphere" else "gouraud", c["width"], c["height"], size, 256)
            b, f = b + db + c["width"] * c["height"] * 4, f + df  # and the colour plane to the host
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ depth planes in 64 bits
def _view_proj64(cam):
    """Right-handed view and OpenGL projection (near 0.1, far 100) of a look-at camera, row-major."""
    p, t = np.asarray(cam.position, np.float64), np.asarray(cam.target, np.float64)
    f = (t - p) / np.linalg.norm(t - p)
    s = np.cross(f, [0.0, 1.0, 0.0])
    s /= np.linalg.norm(s)
    u = np.cross(s, f)
    view = np.eye(4)
    view[0, :3], view[1, :3], view[2, :3] = s, u, -f
    view[:3, 3] = -view[:3, :3] @ p
    g = 1.0 / math.tan(math.radians(cam.fov_degrees) / 2)
    n, far = 0.1, 100.0
    proj = np.zeros((4, 4))
    proj[0, 0], proj[1, 1], proj[2, 2], proj[2, 3], proj[3, 2] = g / cam.aspect, g, -(far + n) / (far - n), -2 * far * n / (far - n), -1.0
    return proj @ view


def _depth64(positions, indices, cam, width, height, far):
    """NDC depth of the nearest front-facing triangle at each pixel centre, `far` where there is
    none; None when a vertex lies behind the near plane (such triangles would need clipping)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pos = torch.as_tensor(np.asarray(positions, np.float64), device=dev)
    m = torch.as_tensor(_view_proj64(cam), device=dev)
    clip = torch.cat([pos, torch.ones_like(pos[:, :1])], 1) @ m.T
    if bool((clip[:, 2] < -clip[:, 3]).any()):
        return None
    ndc = clip[:, :3] / clip[:, 3:]
    xy = (ndc[:, :2] + 1) * 0.5 * torch.tensor([width, height], dtype=torch.float64, device=dev)
    idx = torch.as_tensor(np.asarray(indices, np.int64), device=dev)
    p, z = xy[idx], ndc[:, 2][idx]  # (F, 3, 2), (F, 3)
    area = (p[:, 1, 0] - p[:, 0, 0]) * (p[:, 2, 1] - p[:, 0, 1]) - (p[:, 2, 0] - p[:, 0, 0]) * (p[:, 1, 1] - p[:, 0, 1])
    size = torch.tensor([width, height], dtype=torch.float64, device=dev)
    lo = torch.minimum(torch.clamp(torch.floor(p.amin(1)), min=0.0), size).long()
    hi = torch.minimum(torch.clamp(torch.ceil(p.amax(1)), min=0.0), size).long()
    box = (hi - lo).clamp(min=0)
    n = torch.where(area > 0, box[:, 0] * box[:, 1], torch.zeros_like(box[:, 0]))
    depth = torch.full((width * height,), far, dtype=torch.float64, device=dev)
    keep = torch.nonzero(n).flatten()
    ends = torch.cumsum(n[keep], 0)
    first = 0
    while first < len(keep):  # about 16M (triangle, pixel) pairs at a time
        done = int(ends[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(ends, done + (1 << 24))))
        t = keep[first:last]
        tri = torch.repeat_interleave(t, n[t])
        k = torch.arange(len(tri), device=dev) - torch.repeat_interleave(ends[first:last] - n[t] - done, n[t])
        px, py = lo[tri, 0] + k % box[tri, 0], lo[tri, 1] + k // box[tri, 0]
        cx, cy = px.double() + 0.5, py.double() + 0.5
        q = p[tri]
        e = [(q[:, (i + 1) % 3, 0] - cx) * (q[:, (i + 2) % 3, 1] - cy) - (q[:, (i + 2) % 3, 0] - cx) * (q[:, (i + 1) % 3, 1] - cy)
             for i in range(3)]
        inside = (e[0] >= 0) & (e[1] >= 0) & (e[2] >= 0)
        zz = (z[tri, 0] * e[0] + z[tri, 1] * e[1] + z[tri, 2] * e[2]) / area[tri]
        inside &= zz <= 1.0
        depth.scatter_reduce_(0, (py * width + px)[inside], zz[inside], "amin")
        first = last
    return depth.reshape(height, width)


def exact(case, seed):
    c = case
    if c["kind"] in ("frame", "animate"):
        sc = _scene(c, seed)
        z = _depth64(sc.mesh.positions, sc.mesh.indices, sc.camera, sc.width, sc.height,
                     math.inf if c["far"] is None else c["far"])
        return None if z is None else {"bgra": None, "depth": z}
    if c["kind"] in ("batch", "oneshot"):
        out = [_depth64(s.mesh.positions, s.mesh.indices, s.camera, s.width, s.height, 1.0) for s in _batch_scenes(c, seed)]
        return [None if z is None else {"bgra": None, "depth": z} for z in out]
    if c["kind"] == "ingest":
        o = _obj(c, seed)
        q = o["corners"][:, 0].reshape(-1, 4)
        tri = np.stack([q[:, [0, 1, 2]], q[:, [0, 2, 3]]], 1).reshape(-1, 3)
        z = _depth64(o["positions"], tri, _obj_camera(c, seed), c["width"], c["height"], 1.0)
        return None if z is None else {"bgra": None, "depth": z}
    return None  # files and colour planes: bytes
