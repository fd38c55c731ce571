"""Workloads of the raster pipeline through its public entry points, for timing.

A case is a dict of plain values. `path` names the entry point a program calls:

  frame    Renderer.render + framebuffer_async into a CUDA tensor (a render loop whose images
           stay on the device)
  sync     Renderer.render + framebuffer into host memory, then stats (one image at a time)
  stream   two resident meshes and two page-locked images used in turn: update_async, render,
           framebuffer_async, then wait_output (animated geometry from one host thread)
  noalloc  rast_render_noalloc on the caller's device buffers and stream
  batch    BatchRenderer.render of many scenes into device memory
  replay   the same batch captured once (BatchRenderer.capture) and replayed
  serve    RenderServer: requests submitted together, then waited for one by one

and `scene` what is drawn: `cube` and `demo` (the crate's demo objects), `soup` (independent
triangles, projected edge min_px..max_px, a tenth of them across the near plane) and `terrain`
(an indexed heightfield of small triangles); the batch paths draw `count` soups of mixed size,
resolution and sample count. Outputs are ARGB images (32-bit integers) and counters: they are
whole numbers, for which there is no 64-bit value to be near to.
"""
import ctypes

import numpy as np
import torch

from rusterizer_gb300 import _lib, mesh, renderer, scenes
from rusterizer_gb300 import math as rm
from rusterizer_gb300.batch import BatchRenderer
from rusterizer_gb300.server import RenderServer

ALL_WARPS = 0xFFFFFFFF  # Renderer.set_heavy_tile_entries: every bin one warp per tile


def listed():
    return [
        # the crate's demo cube, one displayed image after another
        {"name": "cube_sync_800x600", "path": "sync", "scene": "cube", "width": 800, "height": 600, "msaa": 4,
         "fs": 0, "tex": 64},
        # a thumbnail for a host that owns all device memory: the smallest call
        {"name": "sphere_noalloc_256x192", "path": "noalloc", "scene": "sphere", "width": 256, "height": 192,
         "msaa": 4, "fs": 0, "tex": 64},
        # the crate's demo scene: several draws with different shaders in one frame
        {"name": "demo_frame_1280x720", "path": "frame", "scene": "demo", "width": 1280, "height": 720, "msaa": 4,
         "fs": 0, "tex": 256},
        # mixed triangle sizes with clipping, full HD: an ordinary scene
        {"name": "soup100k_frame_1080p", "path": "frame", "scene": "soup", "tris": 100_000, "min_px": 1.0,
         "max_px": 64.0, "width": 1920, "height": 1080, "msaa": 4, "fs": 0, "tex": 1024},
        # large overlapping triangles: fill-bound, deep overdraw
        {"name": "overdraw3k_frame_1440p", "path": "frame", "scene": "soup", "tris": 3_000, "min_px": 32.0,
         "max_px": 512.0, "width": 2560, "height": 1440, "msaa": 4, "fs": 0, "tex": 512},
        # dense mesh of sub-pixel triangles, 4K: the largest single frame
        {"name": "terrain2m_frame_4k", "path": "frame", "scene": "terrain", "grid": 1000, "width": 3840,
         "height": 2160, "msaa": 4, "fs": 0, "tex": 2048},
        # one sample per pixel, vertex colours, sizes that no tile divides
        {"name": "terrain180k_msaa1_1366x769", "path": "frame", "scene": "terrain", "grid": 301, "width": 1366,
         "height": 769, "msaa": 1, "fs": 1, "tex": 64},
        # a small scene's depth view read back at once, odd sizes
        {"name": "soup2k_depth_sync_517x389", "path": "sync", "scene": "soup", "tris": 2_001, "min_px": 1.0,
         "max_px": 64.0, "width": 517, "height": 389, "msaa": 4, "fs": 2, "tex": 64},
        # animated geometry: the mesh from the host and the image to the host, every frame
        {"name": "terrain500k_stream_1080p", "path": "stream", "scene": "terrain", "grid": 500, "width": 1920,
         "height": 1080, "msaa": 4, "fs": 0, "tex": 1024},
        # independent scenes rendered together, library defaults
        {"name": "batch20", "path": "batch", "count": 20, "min_tris": 100, "max_tris": 200_000, "split": 0,
         "tile": 0},
        # the same kind of batch captured, with the settings that tuning picks for such mixes
        {"name": "replay20_warp", "path": "replay", "count": 20, "min_tris": 100, "max_tris": 200_000,
         "split": ALL_WARPS, "tile": 32},
        # a burst of requests to the render server
        {"name": "serve40", "path": "serve", "count": 20, "min_tris": 100, "max_tris": 200_000, "split": 0,
         "tile": 0, "requests": 40},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    path = rng.choice(["frame", "frame", "frame", "frame", "sync", "sync", "noalloc", "stream", "batch", "replay",
                       "serve"])
    if path in ("batch", "replay", "serve"):
        lo = _log_uniform(rng, 50, 1000)
        c = {"path": path, "count": rng.randint(3, 20), "min_tris": lo, "max_tris": lo * _log_uniform(rng, 4, 150),
             "split": rng.choice([0, ALL_WARPS]), "tile": rng.choice([0, 16, 32])}
        if path == "serve":
            c["requests"] = rng.randint(c["count"], 40)
        return c
    w = _log_uniform(rng, 200, 2560)
    c = {"path": path, "width": w, "height": max(100, int(w * rng.uniform(0.4, 1.0))), "msaa": rng.choice([4, 4, 1]),
         "fs": rng.choice([0, 0, 1, 2]), "tex": rng.choice([32, 64, 100, 256, 512, 1024])}
    kinds = {"noalloc": ["sphere", "soup", "terrain"], "stream": ["terrain"]}
    c["scene"] = rng.choice(kinds.get(path, ["cube", "demo", "soup", "soup", "soup", "terrain", "terrain"]))
    if c["scene"] == "soup":
        # few large triangles, or many small ones: total covered area stays bounded
        c["tris"] = _log_uniform(rng, 500, 20_000 if path == "noalloc" else 150_000)
        c["min_px"] = 1.0 if c["tris"] > 4_000 else float(_log_uniform(rng, 1, 32))
        c["max_px"] = c["min_px"] * _log_uniform(rng, 8, 64 if c["tris"] > 4_000 else 16)
    elif c["scene"] == "terrain":
        # up to a grid cell per pixel column
        c["grid"] = _log_uniform(rng, 20, 100 if path == "noalloc" else min(700, w))
    return c


# ---- scenes

def _view(case):
    w, h = case["width"], case["height"]
    return rm.camera_view(), rm.project(0.1, 100.0, np.float32(h / w), np.float32(np.deg2rad(60.0)))


def _placed(rng, x, z):
    a = rng.uniform(-np.pi, np.pi, 2).astype(np.float32)
    return rm.mat4_mul(rm.translate(x, 0.0, z), rm.rotate(a[0], a[1], 0.0))


def _scene(case, rng):
    kind, w, h, fs = case["scene"], case["width"], case["height"], case["fs"]
    if kind == "terrain":
        n = case["grid"]
        m = scenes.heightfield(n=n, rng=rng)
        d = np.array([0.0, -1.0, 1.0]) / np.sqrt(2.0)
        view = rm.camera_view(pos=-scenes.HEIGHTFIELD_CAMERA_DISTANCE * rng.uniform(0.9, 1.0) * d, up=(0.0, 1.0, 0.0),
                              direction=d)
        proj = rm.project(0.1, 100.0, np.float32(h / w), np.float32(np.deg2rad(60.0)))
        m["idx"] = scenes._orient_indexed(m["pos"], m["idx"], view)
        draws = [dict(m, world=rm.identity(), fs=fs)]
    elif kind == "soup":
        m = scenes.soup(case["tris"], w, h, rng, min_px=case["min_px"], max_px=case["max_px"])
        view, proj = rm.identity(), rm.project(0.1, 100.0, np.float32(h / w), np.float32(np.deg2rad(60.0)))
        draws = [dict(m, world=rm.identity(), fs=fs)]
    else:
        view, proj = _view(case)
        cube, ball = mesh.cube(1.0), mesh.sphere(0.5)
        if kind == "cube":
            draws = [dict(cube, world=_placed(rng, 0.0, -2.0), fs=fs)]
        elif kind == "sphere":
            draws = [dict(ball, world=_placed(rng, 0.0, -1.0), fs=fs)]
        else:  # demo: cubes and spheres, textured, coloured and by depth
            draws = [dict(cube, world=_placed(rng, -0.9, -2.0), fs=fs), dict(ball, world=_placed(rng, 0.7, -2.2), fs=1),
                     dict(ball, world=_placed(rng, 0.1, -1.2), fs=fs), dict(cube, world=_placed(rng, 1.4, -3.5), fs=2)]
    n = case["tex"]
    tex = scenes.checkerboard(n, max(1, n // 16)) if kind in ("terrain", "cube") else scenes.noise_texture(n, rng)
    return {"width": w, "height": h, "msaa": case["msaa"], "view": view, "proj": proj, "textures": [tex],
            "draws": draws}


def _mix(case, rng):
    """Soups of mixed triangle count, resolution and sample count, 512 x 512 textures."""
    out = []
    for k in range(case["count"]):
        # triangle counts spread evenly over the logarithm of the range
        t = (k + rng.random()) / case["count"]
        n = int(round(case["min_tris"] * (case["max_tris"] / case["min_tris"]) ** t))
        w, h = scenes.RESOLUTIONS[k % 4]
        out.append(scenes.soup_scene(n, w, h, (1, 4)[(k // 4) % 2], rng, 512))
    # shuffled, the same way for every seed: the images keep their sizes and places
    return [out[i] for i in np.random.default_rng(len(out)).permutation(len(out))]


# ---- the paths

class _Frame:
    """A Renderer with its scene resident."""

    def __init__(self, case, rng):
        sc = _scene(case, rng)
        self.sc = sc
        self.r = renderer.Renderer(sc["width"], sc["height"], sc["msaa"])
        self.r.uniforms().bind_texture(0, renderer.Texture(sc["textures"][0]))
        blk = self.r.uniforms().write_block()
        blk.view, blk.projection = sc["view"], sc["proj"]
        self.meshes = [renderer.Mesh.from_dict(d) for d in sc["draws"]]
        for m in self.meshes:
            self.r.upload(m)

    def queue(self):
        blk = self.r.uniforms().write_block()
        for d, m in zip(self.sc["draws"], self.meshes):
            blk.world = d["world"]
            self.r.render(m, renderer.VS_MVP, d["fs"])


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    path = case["path"]
    if path in ("batch", "replay", "serve"):
        return _prepare_many(case, rng)
    if path == "noalloc":
        return _prepare_noalloc(case, rng)
    s = _Frame(case, rng)
    s.path = path
    w, h = case["width"], case["height"]
    if path == "frame":
        s.out = torch.zeros((h, w), dtype=torch.int32, device="cuda")
        s.queue()
        s.r.framebuffer()  # sizes the context's buffers, as framebuffer_async asks for
    elif path == "sync":
        s.pinned = torch.empty((h, w), dtype=torch.int32, pin_memory=True)
        s.out = s.pinned.numpy().view(np.uint32)
    else:
        s.images = [torch.empty((h, w), dtype=torch.int32, pin_memory=True) for _ in range(2)]
        m = s.meshes[0]
        s.meshes.append(renderer.Mesh(m.pos, m.uv, m.idx, m.rgba))
        s.r.upload(s.meshes[1])
        s.host = []
        for k in range(2):  # the two frames of an animation: the terrain, and the terrain raised
            pos = m.pos.copy()
            pos[:, 1] *= 1.0 + 0.25 * k
            s.host.append([torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).pin_memory()
                           for a in (pos, m.uv, m.idx, m.rgba)])
        s.r.render(m, renderer.VS_MVP, case["fs"])
        s.r.framebuffer()
        s.fs = case["fs"]
    return s


class _NoAlloc:
    pass


def _prepare_noalloc(case, rng):
    sc = _scene(case, rng)
    d, s = sc["draws"][0], _NoAlloc()
    s.path, s.case = "noalloc", case
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()  # noqa: E731
    s.pos, s.uv, s.rgba, s.idx, s.tex = (dev(a) for a in (d["pos"], d["uv"], d["rgba"], d["idx"], sc["textures"][0]))
    s.nverts, s.ntris = len(d["pos"]), len(d["idx"])
    s.mats = [(ctypes.c_float * 16)(*np.asarray(m, np.float32).reshape(16).tolist())
              for m in (d["world"], sc["view"], sc["proj"])]
    s.out = torch.zeros((case["height"], case["width"]), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


class _Many:
    """Resident scenes; their images lie one after another in one device buffer."""

    def __init__(self, case, rng):
        mix = _mix(case, rng)
        self.path = case["path"]
        self.br = BatchRenderer()
        self.br.r.set_heavy_tile_entries(case["split"])
        for sc in mix:
            self.br.add_scene(sc, tile=case["tile"])
        order = list(range(len(mix)))
        if self.path == "serve":
            order = [int(i) for i in rng.permutation(np.arange(case["requests"]) % len(mix))]
        self.order = order
        px = [mix[i]["width"] * mix[i]["height"] for i in order]
        self.out = torch.zeros(sum(px), dtype=torch.int32, device="cuda")
        at = np.concatenate([[0], np.cumsum(px)])[:-1]
        self.ptrs = [self.out.data_ptr() + 4 * int(o) for o in at]
        self.graph = self.br.capture(self.ptrs) if self.path == "replay" else None
        self.server = RenderServer(self.br) if self.path == "serve" else None

    def close(self):
        if self.server:
            self.server.close()
            self.server = None
        if self.br:
            self.br.close()
            self.br = None

    def __del__(self):
        self.close()


def _prepare_many(case, rng):
    s = _Many(case, rng)
    torch.cuda.synchronize()
    return s


def run(s):
    if s.path == "frame":
        s.queue()
        s.r.framebuffer_async(s.out)
        return s.out
    if s.path == "sync":
        s.queue()
        s.r.framebuffer(s.out)
        return {"image": s.pinned, "stats": s.r.stats()}
    if s.path == "stream":
        for m, host, img in zip(s.meshes, s.host, s.images):
            s.r.update_async(m, host[0], host[1], host[2], host[3])
            s.r.render(m, renderer.VS_MVP, s.fs)
            s.r.framebuffer_async(img)
        s.r.wait_output()
        return s.images
    if s.path == "noalloc":
        c = s.case
        st = _lib.load().rast_render_noalloc(
            c["width"], c["height"], c["msaa"], 0, float(np.finfo(np.float32).max), s.pos.data_ptr(), s.uv.data_ptr(),
            s.rgba.data_ptr(), s.nverts, s.idx.data_ptr(), s.ntris, s.mats[0], s.mats[1], s.mats[2], s.tex.data_ptr(),
            c["tex"], c["tex"], c["fs"], s.out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st not in (_lib.OK, _lib.TEXTURE_OOB):
            raise _lib.RastError(st, "render_noalloc")
        return s.out
    if s.path == "batch":
        return {"images": s.out, "status": s.br.render(s.ptrs)}
    if s.path == "replay":
        return {"images": s.out, "status": BatchRenderer.replay(s.graph)}
    ids = [s.server.submit(i, p) for i, p in zip(s.order, s.ptrs)]
    return {"images": s.out, "status": np.array([s.server.wait(i)[0] for i in ids], np.int32)}


# ---- the least that a pass has to move and compute

def _counts(case):
    """(vertices, triangles, pixels, samples, texels) of one pass."""
    if case["path"] in ("batch", "replay", "serve"):
        n = case["count"]
        ratio = case["max_tris"] / case["min_tris"]
        # the mean of a log-uniform triangle count, and of the resolutions in turn
        tris = int(n * case["min_tris"] * (ratio - 1) / np.log(ratio)) if ratio > 1 else n * case["min_tris"]
        px = sum(w * h for w, h in (scenes.RESOLUTIONS[k % 4] for k in range(n)))
        smp = sum((scenes.RESOLUTIONS[k % 4][0] * scenes.RESOLUTIONS[k % 4][1]) * (1, 4)[(k // 4) % 2]
                  for k in range(n))
        f = case["requests"] / n if case["path"] == "serve" else 1.0
        return tuple(int(f * v) for v in (3 * tris, tris, px, smp, n * 512 * 512))
    px = case["width"] * case["height"]
    tex = case["tex"] ** 2 if case["fs"] == 0 else 0
    kind = case["scene"]
    if kind == "terrain":
        v, t = (case["grid"] + 1) ** 2, 2 * case["grid"] ** 2
    elif kind == "soup":
        v, t = 3 * case["tris"], case["tris"]
    else:
        v, t = {"cube": (24, 12), "sphere": (153, 256), "demo": (354, 536)}[kind]
    k = 2 if case["path"] == "stream" else 1
    return k * v, k * t, k * px, k * px * case["msaa"], k * tex


def work(case):
    v, t, px, smp, tex = _counts(case)
    attr = 8 if case.get("fs", 0) == 0 else 16 if case["fs"] == 1 else 0  # uv, colour, or neither
    nbytes = (12 + attr) * v + 12 * t + 4 * tex + 4 * px
    # vertex transform, divide and viewport; triangle setup and box; one resolve add per sample
    flops = 45 * v + 60 * t + 3 * smp
    return {"bytes": int(nbytes), "flops": int(flops)}
