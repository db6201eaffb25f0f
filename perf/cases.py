"""The work a headless Vulkan application has this ICD do, as measurable cases.

A pass is what such an application does for one answer: it submits its
recorded frame (one frame for a request, several back to back for a frame
loop), waits for the fence, copies the attachments out and reads them on the
host. Scenes come from the repository's seeded generators, and everything goes
through the package's Context / Scene / Renderer / Server and the harness's C
entry points. The outputs are the attachments' bytes.

The kinds of work and what each stands for in real use:

  program     small scenes of one shader program: latency and launches count
              (thumbnails, user-interface layers, conformance-style draws);
              with large targets, heavy overdraw by a few hundred
              interpolated triangles under stencil, depth and blending
  cube        the frame loop of the draw_cube sample: 36 vertices, 500 x 500,
              BGRA8 and D16
  request     one offscreen request of the serving workload: a textured
              icosphere into a square RGBA8 + D32 target
  heightfield a textured terrain grid with a mip chain and a trilinear
              sampler, RGBA8 + D32
  blend       many screen-space quads blended in order, no depth
  batch       one render pass of many indexed, partly instanced draws, 70%
              opaque and 30% blended, RGBA8 + D32
  serve       the continuous-batching loop: clients' requests over the
              device's queues
"""
import math

import numpy as np

import cpvulkan_gb300 as c

# variant bits of the program scenes: depth format (0x8 D16, 0x10 D32, 0x18
# D32S8), 0x20 blending, 0x100 stencil, 0x200 BGRA8, 0x400 strips, 0x1000
# 16-bit indices (one draw, whatever the seed), 0x10000 points and lines
D16, D32, D32S8, BLEND, STENCIL, BGRA, INDEX16 = 0x8, 0x10, 0x18, 0x20, 0x100, 0x200, 0x1000
LINES = 0x10000 | 0x400
WIDE_LINES = LINES | 0x20000
RGBA8, RGBA16F = 0, 97  # 0: the program scenes' default (RGBA8, or BGRA8 by variant)


def listed():
    return [
        # the smallest call: a thumbnail of two dozen triangles, colour and depth read
        {"name": "program_64x48", "kind": "program", "program": c.PROGRAM_CUBE, "variant": D16 | INDEX16, "width": 64, "height": 48,
         "triangles": 24, "format": RGBA8, "frames": 1, "depth": True},
        # the sample's frame loop: 32 frames in flight, the last one read
        {"name": "cube_500_loop", "kind": "cube", "frames": 32, "depth": False},
        # the smallest and the largest request of the serving range
        {"name": "request_256_1k", "kind": "request", "side": 256, "triangles": 1000, "frames": 1, "depth": False},
        {"name": "request_2048_500k", "kind": "request", "side": 2048, "triangles": 500000, "frames": 1, "depth": False},
        # overdraw by large interpolated triangles into a half-float target with stencil, depth and blending
        {"name": "overdraw_hdr_720p", "kind": "program", "program": c.PROGRAM_CUBE, "variant": D32S8 | STENCIL | BLEND | INDEX16, "width": 1280,
         "height": 720, "triangles": 300, "format": RGBA16F, "frames": 1, "depth": True},
        # the terrain benchmark's frame
        {"name": "heightfield_1080p", "kind": "heightfield", "grid": 1024, "width": 1920, "height": 1080, "frames": 4, "depth": False},
        # a terrain of an ordinary size on an odd grid and a ragged target
        {"name": "heightfield_301_wxga", "kind": "heightfield", "grid": 301, "width": 1366, "height": 767, "frames": 4, "depth": True},
        # the blend benchmark's frame: one flat colour per quad
        {"name": "blend_200k_1080p", "kind": "blend", "quads": 200000, "width": 1920, "height": 1080, "smooth": 0, "frames": 1, "depth": False},
        # the same with a colour per corner, interpolated: an ordinary number of quads
        {"name": "blend_smooth_6k_720p", "kind": "blend", "quads": 6000, "width": 1280, "height": 720, "smooth": 1, "frames": 1, "depth": False},
        # a small pass of several dozen draws
        {"name": "batch_64_360p", "kind": "batch", "draws": 64, "triangles": 4000, "width": 640, "height": 360, "frames": 1, "depth": True},
        # a large pass: an eighth of the 4096-draw benchmark's draws, its mesh sizes and target
        {"name": "batch_512_1440p", "kind": "batch", "draws": 512, "triangles": 200000, "width": 2560, "height": 1440, "frames": 1, "depth": False},
        # the serving loop above its capacity: sixteen clients on sixteen queues
        {"name": "serve_16_clients", "kind": "serve", "clients": 16, "triangles": 100000, "side": 1024, "window_us": 5000, "gap_us": 100},
    ]


def _log_uniform(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(("program", "program", "cube", "request", "request", "heightfield", "blend", "batch", "batch", "serve"))
    if kind == "program":
        variant = rng.choice((D16, D32, D32S8 | STENCIL, D32 | BGRA)) | rng.choice((0, BLEND)) | INDEX16
        program = rng.choice((c.PROGRAM_CUBE, c.PROGRAM_TEXLIT, c.PROGRAM_NOPERSP, c.PROGRAM_FLATQUAD, c.PROGRAM_DISCARD))
        if rng.random() < 0.25:
            program, variant = c.PROGRAM_CUBE, variant | rng.choice((LINES, WIDE_LINES))
        return {"kind": kind, "program": program, "variant": variant, "width": _log_uniform(rng, 64, 1280), "height": _log_uniform(rng, 48, 720),
                "triangles": _log_uniform(rng, 12, 600), "format": RGBA16F if program == c.PROGRAM_CUBE and rng.random() < 0.5 else RGBA8,
                "frames": rng.randint(1, 4), "depth": True}
    if kind == "cube":
        return {"kind": kind, "frames": rng.randint(1, 64), "depth": rng.random() < 0.5}
    if kind == "request":
        return {"kind": kind, "side": _log_uniform(rng, 256, 2048), "triangles": _log_uniform(rng, 1000, 500000), "frames": 1, "depth": False}
    if kind == "heightfield":
        return {"kind": kind, "grid": _log_uniform(rng, 64, 1024), "width": _log_uniform(rng, 480, 1920), "height": _log_uniform(rng, 270, 1080),
                "frames": rng.randint(1, 4), "depth": rng.random() < 0.5}
    if kind == "blend":
        smooth = rng.randint(0, 1)
        return {"kind": kind, "quads": _log_uniform(rng, 500, 10000 if smooth else 200000), "width": _log_uniform(rng, 480, 1920),
                "height": _log_uniform(rng, 270, 1080), "smooth": smooth, "frames": 1, "depth": False}
    if kind == "batch":
        return {"kind": kind, "draws": _log_uniform(rng, 16, 400), "triangles": _log_uniform(rng, 2000, 100000), "width": _log_uniform(rng, 480, 2560),
                "height": _log_uniform(rng, 270, 1440), "frames": rng.randint(1, 2), "depth": rng.random() < 0.5}
    return {"kind": kind, "clients": rng.randint(4, 20), "triangles": _log_uniform(rng, 2000, 100000), "side": rng.choice((256, 512, 1024)),
            "window_us": rng.randint(1000, 5000), "gap_us": rng.randint(100, 200)}


_ctx = None


def _context():
    """The process's one Vulkan instance and device, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = c.Context()
    return _ctx


def _scene(case, seed):
    k = case["kind"]
    if k == "program":
        return c.Scene(c.PROGRAM, seed, [case["program"], case["variant"], case["width"], case["height"], case["triangles"], 0, case["format"]])
    if k == "cube":
        return c.Scene(c.CUBE, 1, [1 + seed % 359])
    if k == "request":
        return c.Scene(c.SERVE, seed, [case["side"], case["triangles"], seed % 64])
    if k == "heightfield":
        return c.Scene(c.HEIGHTFIELD, seed, [case["grid"], case["width"], case["height"]])
    if k == "blend":
        return c.Scene(c.BLEND, seed, [case["quads"], case["width"], case["height"], case["smooth"]])
    return c.Scene(c.BATCH, seed, [case["draws"], case["triangles"], case["width"], case["height"]])


def _host_image(scene, texel):
    return np.zeros((scene.height, scene.width, texel), np.uint8)


class _Frame:
    """A renderer (its Vulkan objects and recorded frame), and the host
    buffers its program reads the attachments into."""

    def __init__(self, case, seed):
        self.frames = case["frames"]
        self.renderer = None
        self.scene = _scene(case, seed)
        self.renderer = c.Renderer(_context(), self.scene)
        self.out = {"colour": _host_image(self.scene, c.colour_texel_bytes(self.scene.color_format))}
        if case["depth"] and self.scene.depth_format:
            self.out["depth"] = _host_image(self.scene, c.depth_texel_bytes(self.scene.depth_format))

    def run(self):
        self.renderer.render(self.frames)
        _read(self.renderer, self.out["colour"], self.out.get("depth"))
        return self.out

    def __del__(self):
        if self.renderer is not None:
            self.renderer.close()


class _Serving:
    """A server with its resident clients, and a host buffer per client that
    holds an image of the largest side (the clients' sides follow the seed)."""

    def __init__(self, case, seed):
        self.server = None
        self.server = c.Server(_context(), clients=case["clients"], slots=16, mean_interarrival_ms=case["gap_us"] / 1e3,
                               duration_s=case["window_us"] / 1e6, seed=seed % 1000003, min_tris=1000, max_tris=case["triangles"], max_side=case["side"])
        self.out = [np.zeros(case["side"] * case["side"] * 4, np.uint8) for _ in range(case["clients"])]

    def run(self):
        self.server.run()
        for i, image in enumerate(self.out):
            _read(self.server.client(i), image, None)
        return self.out

    def __del__(self):
        if self.server is not None:
            self.server.close()


def _read(renderer, colour, depth):
    r = c.harness().cpvh_readback(renderer.ptr, colour.ctypes.data, depth.ctypes.data if depth is not None else None)
    if r != c.VK_SUCCESS:
        raise RuntimeError("readback failed (%d)" % r)


def prepare(case, seed):
    return _Serving(case, seed) if case["kind"] == "serve" else _Frame(case, seed)


def run(state):
    return state.run()


def work(case):
    """Bytes of one pass: the frame's vertices, indices and texture read once
    and its attachments written once, per frame. Operations: the vertex
    transforms (28 a vertex), the triangles' edges (30 a triangle) and, for
    the blended quads, 8 a fragment."""
    k = case["kind"]
    if k == "program":
        colour = 8 if case["format"] == RGBA16F else 4
        depth = {D16: 2, D32: 4, D32S8: 8}[case["variant"] & 0x18]
        vertices = 3 * case["triangles"]
        inputs, pixels, texel, triangles = 34 * vertices, case["width"] * case["height"], colour + depth, case["triangles"]
    elif k == "cube":
        vertices, triangles, pixels, texel = 36, 12, 500 * 500, 6
        inputs = 32 * vertices
    elif k == "request":
        triangles = case["triangles"]
        vertices, pixels, texel = triangles // 2, case["side"] ** 2, 8
        inputs = 32 * vertices + 12 * triangles + 4 * 512 * 512 * 4 // 3
    elif k == "heightfield":
        vertices, triangles = case["grid"] ** 2, 2 * (case["grid"] - 1) ** 2
        pixels, texel = case["width"] * case["height"], 8
        inputs = 32 * vertices + 12 * triangles + 4 * 1024 * 1024 * 4 // 3
    elif k == "blend":
        vertices, triangles = 4 * case["quads"], 2 * case["quads"]
        pixels, texel = case["width"] * case["height"], 4
        inputs = 24 * vertices + 4 * 3 * triangles
    elif k == "batch":
        # mesh triangles log-uniform from 12, a quarter of the draws with 32.5 instances on average
        mesh = case["draws"] * (case["triangles"] - 12) / math.log(case["triangles"] / 12)
        triangles, vertices = 8.875 * mesh, 8.875 * mesh / 2
        inputs, pixels, texel = 24 * mesh, case["width"] * case["height"], 8
    else:
        requests = case["clients"] * case["window_us"] / case["gap_us"]
        mean = (case["triangles"] - 1000) / math.log(case["triangles"] / 1000)
        triangles, vertices = requests * mean, requests * mean / 2
        sides = [min(s, case["side"]) for s in (256, 512, 1024, 2048)]
        inputs, pixels, texel = 28 * triangles, requests * sum(s * s for s in sides) / 4, 8
    frames = case.get("frames", 1)
    flops = frames * (28 * vertices + 30 * triangles)
    if k == "blend":
        flops += frames * 8 * 3672 * case["quads"]  # a quad covers 3672 pixels on average
    return {"bytes": frames * (inputs + pixels * texel), "flops": flops}


def exact(case, seed):
    """The outputs are encoded attachment bytes: every value is a whole number."""
    return None
