"""Timed cases of the ray-trace path: what programs built on it call, over the sizes they call it with.

A case is a dict with an "op" and that op's sizes:

    trace    Scene.trace: closest hit of device rays (camera batches, random
             batches; fp64-refined or raw fp32 t/u/v; any of the three trees)
    host     Scene.trace_host: the same through host arrays, copies included
    render   Scene.render of one image (and its export to RGBA8 where "export")
    batch    Batch.launch_graph: one pass over many scenes of mixed sizes
    upload   Context.upload_scene of a new scene, its tree read back (what the
             reference's createBvh gives), its first 256 x 256 frame and its
             release: the time from triangles on the host to the first image
    denoise  denoise_image of a noisy image

Scenes come from the package's own generators (displaced icospheres, Cornell
boxes with a triangle soup, a grid of flattened icospheres), seeded by the
case's seed; rays and images are made on the GPU.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "vulkan-compute-ray-tracing_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rtgb  # noqa: E402

TMIN, TMAX = 1e-4, 1e4
_EXACT_PAIRS = 6e10  # ray-triangle pairs that the all-pairs reference takes a few seconds for


# ------------------------------------------------------------------- cases
def listed():
    return [
        # A picking or line-of-sight query: a handful of rays, latency only.
        dict(name="trace_probe_1000", op="trace", mesh="ico", level=5, rays="random", n=1000, builder=0, fp32=False),
        # An ordinary secondary-ray batch on the tightest tree, hits kept as the fp32 formula gives them.
        dict(name="trace_random_300k_ploc_fp32", op="trace", mesh="ico", level=6, rays="random", n=300007, builder=2,
             fp32=True),
        # The closest-hit benchmark's two batches: 2048 x 2048 camera rays and as many random ones, 1.31M triangles.
        dict(name="trace_camera_4m", op="trace", mesh="ico", level=8, rays="camera", width=2048, height=2048, builder=0,
             fp32=False),
        dict(name="trace_random_4m", op="trace", mesh="ico", level=8, rays="random", n=4194304, builder=0, fp32=False),
        # A host application that keeps its rays and hits in its own memory.
        dict(name="trace_host_1m", op="host", mesh="ico", level=5, rays="random", n=1048583, builder=0),
        # The small render of the reference's scale: Cornell box, 12K triangles, 256 x 256, 1 sample, 8 bounces.
        dict(name="render_256", op="render", mesh="cornell", soup=12000, spheres=0, width=256, height=256, spp=1,
             bounces=8, export=False),
        # A preview image of odd size with spheres in the scene, several samples in one call.
        dict(name="render_500x375_spheres", op="render", mesh="cornell", soup=100003, spheres=16, width=500,
             height=375, spp=4, bounces=8, export=False),
        # One displayed frame of a progressive viewer on a large scene: a sample per pixel, then RGBA8.
        dict(name="frame_1080p_2m", op="render", mesh="grid", gx=5, gz=5, level=6, width=1920, height=1080, spp=1,
             bounces=8, export=True),
        # Batched rendering and serving: many scenes of 1K to 300K triangles and mixed sizes in one graph launch.
        dict(name="batch_16", op="batch", jobs=16, soup_lo=1000, soup_hi=300000, side_lo=128, side_hi=512, spp=2,
             bounces=8),
        # A new scene: a small one as a server admits per request, and the benchmark's mesh.
        dict(name="upload_12k", op="upload", mesh="cornell", soup=12000, spheres=4, builder=0),
        dict(name="upload_1m3", op="upload", mesh="ico", level=8, builder=0),
        # The reference's denoise filter at its shipped strength over a full-HD image.
        dict(name="denoise_1080p", op="denoise", width=1920, height=1080, sigma=2.0, ksigma=2.0, threshold=0.05),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["trace", "trace", "host", "render", "render", "batch", "upload", "denoise"])
    if op == "trace":
        c = dict(op=op, mesh="ico", level=rng.randint(4, 8), rays=rng.choice(["random", "camera"]),
                 builder=rng.choice([0, 0, 1, 2]), fp32=rng.random() < 0.3)
        if c["rays"] == "camera":
            c.update(width=_logint(rng, 16, 2048), height=_logint(rng, 16, 2048))
        else:
            c.update(n=_logint(rng, 100, 4194304))
        return c
    if op == "host":
        return dict(op=op, mesh="ico", level=rng.randint(4, 7), rays="random", n=_logint(rng, 1000, 4000000),
                    builder=rng.choice([0, 2]))
    if op == "render":
        if rng.random() < 0.3:
            return dict(op=op, mesh="grid", gx=rng.randint(2, 5), gz=rng.randint(2, 5), level=rng.randint(4, 6),
                        width=rng.randint(320, 1920), height=rng.randint(200, 1080), spp=1,
                        bounces=rng.randint(2, 8), export=True)
        return dict(op=op, mesh="cornell", soup=_logint(rng, 1000, 300000), spheres=rng.randint(0, 16),
                    width=_logint(rng, 48, 1024), height=_logint(rng, 48, 1024), spp=rng.randint(1, 4),
                    bounces=rng.randint(2, 8), export=rng.random() < 0.5)
    if op == "batch":
        return dict(op=op, jobs=rng.randint(2, 16), soup_lo=1000, soup_hi=_logint(rng, 5000, 300000), side_lo=64,
                    side_hi=rng.choice([128, 256, 512]), spp=rng.randint(1, 2), bounces=8)
    if op == "upload":
        if rng.random() < 0.5:
            return dict(op=op, mesh="cornell", soup=_logint(rng, 200, 500000), spheres=rng.randint(0, 16),
                        builder=rng.choice([0, 0, 1, 2]))
        return dict(op=op, mesh="ico", level=rng.randint(3, 8), builder=rng.choice([0, 0, 1, 2]))
    # Only radii whose tap rows do not meet their end within a rounding.
    return dict(op=op, width=_logint(rng, 33, 1920), height=_logint(rng, 33, 1080), sigma=rng.choice([1.0, 1.5, 2.0]),
                ksigma=2.0, threshold=round(rng.uniform(0.03, 0.2), 3))


# ------------------------------------------------------------------ inputs
_CTX = None


def _context():
    """The program's context, kept for its lifetime as a user's is."""
    global _CTX
    if _CTX is None:
        torch.cuda.set_device(0)
        _CTX = rtgb.Context(0)
    return _CTX


def _triangles(case):
    """Triangles of the case's mesh, by its generator and sizes."""
    if case["mesh"] == "ico":
        return 20 * 4 ** case["level"]
    if case["mesh"] == "cornell":
        return 12 + case["soup"]
    return case["gx"] * case["gz"] * 20 * 4 ** case["level"] + 12


def _mesh(case, seed):
    """(triangles, materials, spheres) on the host."""
    if case["mesh"] == "ico":
        return rtgb.gen_icosphere(seed, case["level"]), rtgb.gen_cornell(1, 0)[1], None
    if case["mesh"] == "cornell":
        return rtgb.gen_cornell(seed, case["soup"], case["spheres"])
    t, m = rtgb.gen_grid(seed, case["gx"], case["gz"], case["level"], 0.35, 0.05, (1 << 31) - 1, 3.0)
    return t, m, None


def _camera(case, seed, width, height):
    jitter = np.random.RandomState(seed % (1 << 31)).uniform(-0.3, 0.3, 2)
    if case["mesh"] == "ico":
        eye, at = [jitter[0], jitter[1], -3.0], [0, 0, 0]
    elif case["mesh"] == "cornell":
        eye, at = [jitter[0], jitter[1], -14.0], [0, 0, 0]
    else:
        eye, at = [jitter[0], 2.0 + jitter[1], -40.0], [0, -6, 0]
    return rtgb.camera_look_at(eye, at, [0, 1, 0], 40.0, width, height)


def _rays(case, seed):
    """The case's ray batch (n, 8) on the GPU: origin, tmin, direction, tmax."""
    if case["rays"] == "camera":
        w, h = case["width"], case["height"]
        cam = torch.from_numpy(_camera(case, seed, w, h).as_array()).cuda()
        x = (torch.arange(w, device="cuda", dtype=torch.float32) / w).repeat(h)
        y = (torch.arange(h, device="cuda", dtype=torch.float32) / h).repeat_interleave(w)
        d = cam[3:6] + x[:, None] * cam[6:9] + y[:, None] * cam[9:12] - cam[0:3]
        o = cam[0:3].expand(w * h, 3)
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        o = torch.rand((n, 3), generator=g, device="cuda") * 3.0 - 1.5
        d = torch.randn((n, 3), generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    r = torch.empty((len(d), 8), device="cuda")
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = o, TMIN, d, TMAX
    return r


def _ray_count(case):
    return case["width"] * case["height"] if case["rays"] == "camera" else case["n"]


def _noisy_image(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["height"], case["width"]
    y = torch.linspace(0, 6, h, device="cuda")[:, None, None]
    x = torch.linspace(0, 9, w, device="cuda")[None, :, None]
    c = torch.arange(4, device="cuda", dtype=torch.float32)
    img = 0.5 + 0.4 * torch.sin(x + c) * torch.cos(y - c) + 0.08 * torch.randn((h, w, 4), generator=g, device="cuda")
    img = img.clamp_(0.0, 4.0)
    img[:, :, 3] = 1.0
    return img.contiguous()


class _State:
    """One case's inputs and handles; its scenes and batch are given back with it."""

    def __init__(self, case):
        self.case = case
        self.ctx = _context()
        self.scenes = []
        self.batch = None

    def upload(self, mesh, builder=0):
        self.ctx.set_tuning("bvh.builder", builder)
        try:
            sc = self.ctx.upload_scene(mesh[0], mesh[1], spheres=mesh[2])
        finally:
            self.ctx.set_tuning("bvh.builder", 0)
        self.scenes.append(sc)
        return sc

    def __del__(self):
        if self.batch is not None:
            self.batch.destroy()
        for sc in self.scenes:
            sc.release()


def prepare(case, seed):
    s = _State(case)
    op = case["op"]
    if op in ("trace", "host"):
        s.scene = s.upload(_mesh(case, seed), case["builder"])
        s.rays = _rays(case, seed + 1)
        s.n = len(s.rays)
        if op == "host":
            s.rays = s.rays.cpu().pin_memory().numpy()
            s.hits = torch.empty((s.n, 4), dtype=torch.float32, pin_memory=True).numpy()
        else:
            s.hits = torch.empty((s.n, 4), dtype=torch.float32, device="cuda")
            s.out = {"tri": s.hits.view(torch.int32)[:, 0], "tuv": s.hits[:, 1:]}
    elif op == "render":
        s.scene = s.upload(_mesh(case, seed))
        s.scene.set_camera(_camera(case, seed + 1, case["width"], case["height"]))
        s.image = torch.zeros((case["height"], case["width"], 4), device="cuda")
        s.bytes = torch.zeros((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
    elif op == "batch":
        jobs, n = [], case["jobs"]
        s.images = []
        for i in range(n):
            f = i / max(n - 1, 1)
            job = dict(mesh="cornell", soup=round(case["soup_lo"] * (case["soup_hi"] / case["soup_lo"]) ** f),
                       spheres=i % 5)
            # Sides cycle over the powers of two from side_lo to side_hi, so that small and large scenes meet both.
            side = case["side_lo"] << (i % (1 + round(math.log2(case["side_hi"] / case["side_lo"]))))
            sc = s.upload(_mesh(job, seed + 100 * i))
            image = torch.zeros((side, side, 4), device="cuda")
            s.images.append(image)
            jobs.append(rtgb.make_job(sc, _camera(job, seed + i, side, side), image, side, side, case["spp"],
                                      case["bounces"]))
        s.batch = s.ctx.batch(jobs)
    elif op == "upload":
        s.mesh = _mesh(case, seed)
        s.camera = _camera(case, seed + 1, 256, 256)
        s.image = torch.zeros((256, 256, 4), device="cuda")
        s.nodes = torch.zeros((2 * len(s.mesh[0]) - 1, rtgb.NODE_WORDS), dtype=torch.int32, pin_memory=True).numpy()
    else:
        s.noisy = _noisy_image(case, seed)
        s.image = torch.empty_like(s.noisy)
    return s


# ------------------------------------------------------------------ passes
def run(s):
    c = s.case
    op = c["op"]
    if op == "trace":
        s.scene.trace(s.rays, s.n, s.hits, rtgb.HIT_FP32 if c["fp32"] else 0)
        return s.out
    if op == "host":
        s.scene.trace_host(s.rays, s.hits)
        return {"tri": s.hits.view(np.int32)[:, 0], "tuv": s.hits[:, 1:]}
    if op == "render":
        s.scene.render(s.image, c["width"], c["height"], c["spp"], c["bounces"])
        if not c["export"]:
            return s.image
        rtgb.export_image(s.ctx, s.image, c["width"], c["height"], s.bytes)
        return {"image": s.image, "rgba8": s.bytes}
    if op == "batch":
        s.batch.launch_graph()
        return s.images
    if op == "upload":
        sc = s.upload(s.mesh, c["builder"])
        sc.set_camera(s.camera)
        sc.render(s.image, 256, 256, 1, 8)
        s.ctx.check(rtgb.LIB.rtDownloadBvh(s.ctx.handle, sc.id, s.nodes.ctypes.data, len(s.nodes)), "rtDownloadBvh")
        s.scenes.remove(sc)
        sc.release()
        return {"nodes": s.nodes, "image": s.image}
    rtgb.denoise_image(s.ctx, s.noisy, c["width"], c["height"], s.image, c["sigma"], c["ksigma"], c["threshold"])
    return s.image


def _cast_work(rays, tris):
    """Least work of `rays` closest-hit queries in a tree of `tris` triangles:
    a descent of its depth (a box test a level) and one triangle test a ray;
    every triangle once at most."""
    depth = math.log2(max(tris, 2)) + 1
    return (min(48.0 * tris, 48.0 * rays * depth), rays * (12.0 * depth + 47.0))


def work(case):
    op = case["op"]
    if op in ("trace", "host"):
        n = _ray_count(case)
        b, f = _cast_work(n, _triangles(case))
        return {"bytes": b + 48.0 * n, "flops": f}
    if op == "render":
        pixels = case["width"] * case["height"]
        b, f = _cast_work(pixels * case["spp"] * (1 + case["bounces"] / 2), _triangles(case))
        return {"bytes": b + (16.0 + 4.0 * case["export"]) * pixels, "flops": f}
    if op == "batch":
        b = f = 0.0
        n = case["jobs"]
        for i in range(n):
            tris = case["soup_lo"] * (case["soup_hi"] / case["soup_lo"]) ** (i / max(n - 1, 1))
            side = case["side_lo"] << (i % (1 + round(math.log2(case["side_hi"] / case["side_lo"]))))
            x, y = _cast_work(side * side * case["spp"] * (1 + case["bounces"] / 2), tris)
            b, f = b + x + 16.0 * side * side, f + y
        return {"bytes": b, "flops": f}
    if op == "upload":
        # Triangles in, the tree out; a comparison and a box union a level and triangle.
        tris = _triangles(case)
        return {"bytes": (48.0 + 96.0) * tris, "flops": 13.0 * tris * math.log2(max(tris, 2))}
    pixels = case["width"] * case["height"]
    radius = round(case["ksigma"] * case["sigma"])
    return {"bytes": 32.0 * pixels, "flops": pixels * math.pi * radius * radius * 60.0}


# --------------------------------------------------------- 64-bit reference
def _exact_hits(tris, rays):
    """t, u, v of every ray's closest triangle by testing all pairs in fp64
    (0 where nothing is hit): with a = v0 - v1, b = v2 - v0, n = b x a,
    t = n.(v0 - o) / n.d and, with q = (v0 - o) x d, u = q.b / n.d, v = q.a / n.d."""
    T = torch.from_numpy(tris).cuda().double()
    R = rays.double()
    v0, v1, v2 = T[:, 0:3], T[:, 4:7], T[:, 8:11]
    a, b = v0 - v1, v2 - v0
    n = torch.linalg.cross(b, a)
    # q.b = (v0 x d).b - (o x d).b = d.(b x v0) - (o x d).b, and q.a alike.
    bv, av, nv = torch.linalg.cross(b, v0), torch.linalg.cross(a, v0), (n * v0).sum(1)
    one = torch.ones(1, device="cuda", dtype=torch.float64)
    out = torch.zeros((len(R), 3), device="cuda", dtype=torch.float64)
    step = max(1, int(1.2e8 / len(T)))
    for i in range(0, len(R), step):
        o, d = R[i:i + step, 0:3], R[i:i + step, 4:7]
        od = torch.linalg.cross(o, d)
        idet = 1.0 / (d @ n.T)
        t = (nv - o @ n.T) * idet
        u = torch.cat([d, -od], 1) @ torch.cat([bv, b], 1).T * idet
        v = torch.cat([d, -od], 1) @ torch.cat([av, a], 1).T * idet
        miss = (t <= TMIN) | (t >= TMAX) | (u < 0) | (u > 1) | (v < 0) | (u + v > 1) | ~torch.isfinite(t)
        t = torch.where(miss, math.inf * one, t)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        at = torch.stack([best, u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]], 1)
        out[i:i + step] = torch.where(hit[:, None], at, 0.0 * one)
    return out


def _exact_denoise(img, case):
    """The filter of denoise_image in fp64: columns x, rows -pt, -pt + 1, ... <= pt
    with pt = sqrt(radius^2 - x^2), a linear tap between two texel rows."""
    c = img.double()
    sigma, thr = case["sigma"], case["threshold"]
    radius = round(case["ksigma"] * sigma)
    z = torch.zeros_like(c[:, :, :1])
    acc = torch.zeros_like(c)
    for x in range(-radius, radius + 1):
        pt = math.sqrt(radius * radius - x * x)
        column = torch.roll(c, -x, 1)
        for k in range(int(math.floor(2 * pt + 1e-9)) + 1):
            y = k - pt
            j = math.floor(y)
            w = (1 - (y - j)) * torch.roll(column, -j, 0) + (y - j) * torch.roll(column, -j - 1, 0)
            blur = math.exp(-(x * x + y * y) / (2 * sigma * sigma)) / (2 * math.pi * sigma * sigma)
            dc2 = (w - c).square().sum(2, keepdim=True)
            delta = torch.exp(-dc2 / (2 * thr * thr)) / (math.sqrt(2 * math.pi) * thr) * blur
            z += delta
            acc += delta * w
    return acc / z


def exact(case, seed):
    """What run() returns in fp64, where that is a number of its own (a path
    traced image is one draw of a random walk, a hit's triangle an index)."""
    if case["op"] in ("trace", "host"):
        if float(_ray_count(case)) * _triangles(case) > _EXACT_PAIRS:
            return None
        return {"tri": None, "tuv": _exact_hits(_mesh(case, seed)[0], _rays(case, seed + 1))}
    if case["op"] == "denoise":
        return _exact_denoise(_noisy_image(case, seed), case)
    return None
