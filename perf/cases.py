"""Performance cases of the path-tracing library: the calls a renderer makes, from a thumbnail to
a full frame, with their inputs, one pass of each, and its algorithmic work.

A case is a dict with a "kind":

  render    one frame of a seeded scene (box room, sphere field, displaced mesh, quads, material
            zoo), into a host image or a device buffer, plain or with adaptive sampling
  backward  gradients of a frame's materials for a given dL/d(image)
  batch     many uneven scenes rendered together
  tonemap   a linear HDR frame through the LDR colour chain, device to device
  ldr       a frame rendered and tone mapped into host RGBA bytes
  aov       depth, normal and albedo passes of a frame
  rays      closest hits of a host ray set against a terrain mesh

Every render traces `spp` stratified samples per pixel; `seed` keys its random numbers, moves the
camera of the frame cases and draws the scene where a scene is cheap to draw.
"""
import functools
import math

import numpy as np
import torch

import luminara_b200 as L
from luminara_b200 import abi
from luminara_b200 import workloads as W

CURVES = {"aces": abi.TONEMAP_ACES, "reinhard": abi.TONEMAP_REINHARD, "filmic": abi.TONEMAP_FILMIC,
          "none": abi.TONEMAP_NONE}
FILTERS = {"box": abi.FILTER_BOX, "triangle": abi.FILTER_TRIANGLE, "gaussian": abi.FILTER_GAUSSIAN,
           "mitchell": abi.FILTER_MITCHELL}

# Flops of one path in the scene's usual depth (box, primitive and plane tests of its segments and
# shadow rays, counted on the device and charged per test as bench.py does).
PATH_FLOPS = {"room": 1200, "spheres": 760, "mesh": 1000, "quads": 1300, "zoo": 900, "uneven": 900}


def render_case(name, scene, w, h, spp, depth, **more):
    return {"name": name, "kind": "render", "scene": scene, "w": w, "h": h, "spp": spp, "depth": depth, "level": 8,
            "filter": "box", "exposure": 1.0, "adaptive": False, "host": True, **more}


def listed():
    return [
        # a material preview or thumbnail: the smallest call, launches and the readback count
        render_case("room_preview", "room", 128, 128, 16, 8),
        # the box room at its own size: light sampling on every bounce, a quarter million pixels
        render_case("room_256", "room", 256, 256, 64, 8),
        # the headline frame: a sphere field under a sky at full HD, left on the device
        render_case("spheres_1080", "spheres", 1920, 1080, 256, 16, host=False),
        # the largest scene: 1.3 M triangles with GGX patches, disk lights and fog at full HD
        render_case("mesh_1080", "mesh", 1920, 1080, 128, 8, host=False),
        # an optimisation step's two halves: the forward image and the gradients of 1,004 materials
        render_case("quads_forward", "quads", 512, 512, 64, 6),
        {"name": "quads_backward", "kind": "backward", "w": 512, "h": 512, "spp": 64, "depth": 6, "filter": "box"},
        # a render farm's queue: scenes of uneven size, resolution and samples in one call
        {"name": "batch_12", "kind": "batch", "n": 12, "max_res": 1024, "max_spp": 64, "max_prims": 50000},
        # the headline frame with adaptive sampling (the reference's default threshold)
        render_case("spheres_adaptive", "spheres", 1920, 1080, 256, 16, adaptive=True, host=False),
        # a still for print: an 8K frame through the common colour chain
        {"name": "tonemap_8k", "kind": "tonemap", "w": 7680, "h": 4320, "curve": "aces", "gamma": 0.0,
         "exposure": 1.0, "auto": False, "graded": False},
        # a graded full HD frame: auto-exposure and the optional colour steps
        {"name": "grade_1080", "kind": "tonemap", "w": 1920, "h": 1080, "curve": "filmic", "gamma": 2.2,
         "exposure": 1.0, "auto": True, "graded": True},
        # denoiser and compositing inputs of a frame
        {"name": "aov_1080", "kind": "aov", "w": 1920, "h": 1080, "grid": 11},
        # picking, baking, visibility queries: a million rays from host memory and their hits
        {"name": "rays_1m", "kind": "rays", "n": 1000003, "side": 200},
    ]


def draw(rng):
    def between(lo, hi):   # a whole number, even over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def frame(max_px):     # odd widths and heights of common shapes
        px = between(64 * 48, max_px)
        aspect = rng.choice([1.0, 4 / 3, 16 / 9, 9 / 16, 2.39])
        w = max(9, int(math.sqrt(px * aspect)) + rng.randrange(3))
        return w, max(7, int(w / aspect))

    kind = rng.choice(["render", "render", "render", "render", "backward", "batch", "tonemap", "tonemap", "ldr",
                       "aov", "rays"])
    if kind in ("render", "ldr"):
        scene = rng.choice(["room", "spheres", "mesh", "quads", "zoo"])
        w, h = frame(1920 * 1080)
        budget = 64e6 if scene in ("mesh", "zoo") else 200e6
        spp = min(between(4, 256), max(4, int(budget / (w * h))))
        c = {"kind": kind, "scene": scene, "w": w, "h": h, "spp": spp, "depth": rng.choice([2, 5, 6, 8, 16, 50]),
             "level": rng.choice([3, 5, 6, 7]), "filter": rng.choice(["box", "box", "triangle", "gaussian", "mitchell"]),
             "exposure": rng.choice([1.0, 1.0, 2.0, 0.7])}
        if kind == "render":
            c["adaptive"] = rng.random() < 0.2
            c["host"] = rng.random() < 0.5
        return c
    if kind == "backward":
        w, h = frame(512 * 512)
        return {"kind": kind, "w": w, "h": h, "spp": between(4, 64), "depth": rng.choice([2, 4, 6, 8]),
                "filter": rng.choice(["box", "box", "gaussian"])}
    if kind == "batch":
        return {"kind": kind, "n": between(2, 16), "max_res": rng.choice([256, 512, 1024]),
                "max_spp": rng.choice([16, 64]), "max_prims": between(100, 50000)}
    if kind == "tonemap":
        w, h = frame(7680 * 4320)
        graded = rng.random() < 0.35
        return {"kind": kind, "w": w, "h": h, "curve": rng.choice(sorted(CURVES)), "gamma": rng.choice([0.0, 0.0, 2.2]),
                "exposure": rng.choice([1.0, 1.0, 0.5, 1.7]), "auto": rng.random() < 0.35, "graded": graded}
    if kind == "aov":
        w, h = frame(2560 * 1440)
        return {"kind": kind, "w": w, "h": h, "grid": rng.choice([3, 8, 11, 20])}
    return {"kind": "rays", "n": between(1000, 2000000), "side": between(4, 400)}


# ------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=1)
def mesh_world(level):
    """The displaced mesh of one level: the geometry is the same for every seed."""
    return W.dense_mesh(level=level)[0]


def scene_of(case, seed):
    scene, size = case["scene"], {"width": case["w"], "height": case["h"]}
    if scene == "room":
        world = W.box_room(**size)[0]
        world.camera.look_from = (278.0 + seed % 41 - 20.0, 278.0, -800.0)
    elif scene == "spheres":
        world = W.random_spheres(scene_seed=seed, **size)[0]
    elif scene == "mesh":
        world = mesh_world(case["level"])
        a = 0.1 * (seed % 63)
        world.camera.look_from = (4.2 * math.sin(a), 0.6, 4.2 * math.cos(a))
        world.camera.aspect_ratio = case["w"] / case["h"]
    elif scene == "quads":
        world = W.diff_quads(scene_seed=seed, **size)[0]
    else:
        world = W.material_zoo(**size)[0]
        world.camera.look_from = (0.1 * (seed % 21) - 1.0, 4.5, 9.5)
    background = {"spheres": abi.BG_SKY}.get(scene, abi.BG_SOLID)
    colour = {"mesh": (0.05, 0.05, 0.08), "zoo": (0.05, 0.05, 0.08)}.get(scene, (0.0, 0.0, 0.0))
    cfg = L.RenderConfig(samples_per_pixel=case["spp"], max_depth=case["depth"], seed=seed, background=background,
                         bg_color=colour, pixel_filter=FILTERS[case["filter"]], exposure=case.get("exposure", 1.0),
                         adaptive=case.get("adaptive", False), **size)
    return world, cfg


def batch_shapes(case):
    """(primitives, resolution, spp) of a batch's scenes: the same for every seed."""
    rng = np.random.default_rng(case["n"])
    res = [r for r in (128, 256, 512, 1024) if r <= case["max_res"]]
    spp = [s for s in (16, 64) if s <= case["max_spp"]]
    return [(int(round(math.exp(rng.uniform(math.log(10), math.log(case["max_prims"]))))), int(rng.choice(res)),
             int(rng.choice(spp))) for _ in range(case["n"])]


def terrain(side, seed):
    """A height field of side x side cells over [-4, 4]^2 as vertices (f32 values) and triangles."""
    rng = np.random.default_rng(seed)
    g = np.linspace(-4.0, 4.0, side + 1)
    x, z = np.meshgrid(g, g, indexing="ij")
    y = sum(rng.uniform(0.05, 0.3) * np.sin(rng.uniform(0.5, 4.0) * x + rng.uniform(0.5, 4.0) * z + rng.uniform(0, 6.3))
            for _ in range(6))
    v = np.stack([x, y, z], -1).reshape(-1, 3).astype(np.float32).astype(np.float64)
    i = (np.arange(side)[:, None] * (side + 1) + np.arange(side)[None, :]).reshape(-1)
    f = np.concatenate([np.stack([i, i + 1, i + side + 1], -1), np.stack([i + 1, i + side + 2, i + side + 1], -1)])
    return v, f.astype(np.uint32)


def ray_set(n, seed):
    """Rays from above the terrain, aimed at points on and around it (some miss)."""
    rng = np.random.default_rng(seed + 1)
    o = rng.uniform((-5.0, 2.0, -5.0), (5.0, 5.0, 5.0), (n, 3)).astype(np.float32)
    d = (rng.uniform((-5.0, -0.5, -5.0), (5.0, 0.5, 5.0), (n, 3)) - o).astype(np.float32)
    return o, d


def hdr_frame(w, h, seed):
    """A linear radiance frame: smooth regions over five decades with per-pixel sampling noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    coarse = torch.randn((1, 3, max(2, h // 32), max(2, w // 32)), generator=g, device="cuda") * 1.5 - 1.0
    smooth = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=False)[0]
    noise = torch.randn((h, w, 3), generator=g, device="cuda") * 0.1
    return torch.exp(smooth.permute(1, 2, 0) + noise).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("render", "ldr"):
        world, cfg = scene_of(case, seed)
        st = {"kind": kind, "scene": L.GpuScene(world), "cfg": cfg}
        if kind == "ldr":
            st["tm"] = L.ToneMapConfig()
        elif not case["host"]:
            st["out"] = torch.empty(cfg.out_shape(), device="cuda")
        return st
    if kind == "backward":
        world, cfg = scene_of({**case, "scene": "quads"}, seed)
        rng = np.random.default_rng(seed)
        dl = rng.normal(0.0, 1e-3, cfg.out_shape()).astype(np.float32)
        return {"kind": kind, "scene": L.GpuScene(world), "cfg": cfg, "dl": dl, "lm": world.light_material_indices()}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        items = [W.uneven_scene(rng, n, r, r, s, seed=seed + k) for k, (n, r, s) in enumerate(batch_shapes(case))]
        scenes, cfgs = [L.GpuScene(w) for w, _ in items], [c for _, c in items]
        outs = [torch.empty(c.out_shape(), device="cuda") for c in cfgs]
        return {"kind": kind, "batch": L.Batch(scenes, cfgs, config={"mode": abi.BATCH_STREAMS}), "outs": outs}
    if kind == "tonemap":
        tm = L.ToneMapConfig(tone_map=CURVES[case["curve"]], gamma=case["gamma"], exposure=case["exposure"],
                             auto_exposure=case["auto"])
        if case["graded"]:
            tm.saturation, tm.white_balance, tm.vignette, tm.contrast = 1.2, 0.4, 0.3, 1.1
            tm.grade_shadows, tm.grade_highlights = (0.95, 1.0, 1.1), (1.05, 1.0, 0.95)
        return {"kind": kind, "hdr": hdr_frame(case["w"], case["h"], seed), "tm": tm, "w": case["w"], "h": case["h"],
                "scratch": torch.empty(abi.TONEMAP_SCRATCH_BYTES, dtype=torch.uint8, device="cuda"),
                "rgba": torch.empty((case["h"], case["w"], 4), dtype=torch.uint8, device="cuda")}
    if kind == "aov":
        world, cfg = W.random_spheres(case["w"], case["h"], scene_seed=seed, seed=seed, grid=case["grid"])
        return {"kind": kind, "scene": L.GpuScene(world), "cfg": cfg}
    world = L.World()
    v, f = terrain(case["side"], seed)
    m = L.Lambertian((0.5, 0.5, 0.5))
    world.add_mesh(L.Mesh(positions=v, indices=f, tri_material=np.full(len(f), world.material_index(m), np.int32)))
    o, d = ray_set(case["n"], seed)
    return {"kind": kind, "scene": L.GpuScene(world), "rays": L.make_rays(o, d)}


# -------------------------------------------------------------------------------------- passes
def run(st):
    kind = st["kind"]
    if kind == "render":
        if "out" not in st:
            return st["scene"].render(st["cfg"])[0]
        st["scene"].render_device(st["cfg"], st["out"].data_ptr())
        return st["out"]
    if kind == "ldr":
        return st["scene"].render_ldr(st["cfg"], st["tm"])[0]
    if kind == "backward":
        return list(st["scene"].backward(st["cfg"], st["dl"], st["lm"])[:3])
    if kind == "batch":
        st["batch"].render_device([o.data_ptr() for o in st["outs"]])
        return st["outs"]
    if kind == "tonemap":
        L.tonemap_device(st["hdr"].data_ptr(), st["w"], st["h"], st["tm"], st["scratch"].data_ptr(),
                         st["rgba"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return st["rgba"]
    if kind == "aov":
        return list(st["scene"].render_aov(st["cfg"]))
    h = st["scene"].intersect(st["rays"])
    return {k: h[k] for k in ("t", "u", "v", "normal", "prim_id", "front_face", "material")}


# ---------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "batch":
        shapes = batch_shapes(case)
        return {"bytes": sum(12 * r * r + 112 * n for n, r, _ in shapes),
                "flops": sum(r * r * s for _, r, s in shapes) * PATH_FLOPS["uneven"]}
    if kind == "rays":
        # 48 bytes in and 40 out per ray; a walk of a balanced tree and one leaf
        return {"bytes": 88 * case["n"], "flops": case["n"] * (36 * math.log2(2 * case["side"] ** 2) + 52)}
    px = case["w"] * case["h"]
    if kind == "tonemap":
        return {"bytes": 16 * px, "flops": px * (300 if case["graded"] else 30)}
    if kind == "aov":
        return {"bytes": 10 * px, "flops": px * (36 * 10 + 28 * 2)}
    strata = math.ceil(math.sqrt(case["spp"])) ** 2
    flops = px * strata * PATH_FLOPS["quads" if kind == "backward" else case["scene"]]
    if kind == "backward":
        return {"bytes": 12 * px, "flops": 2 * flops}
    if case.get("adaptive"):
        flops *= 0.4   # samples kept at the default threshold on these scenes
    scene = {"mesh": 20 * 4 ** case["level"] * 110}.get(case["scene"], 0)   # nodes and records read once
    return {"bytes": (4 if kind == "ldr" else 12) * px + scene, "flops": flops}


# ---------------------------------------------------------------------------- values in 64 bits
def exact(case, seed):
    """What run returns, in 64 bits, without the library.  A frame's pixels are sums over paths
    whose discrete choices (roulette, lobes, visibility) turn on single roundings: the box room,
    small and diffuse, is traced here path by path; the other frames and gradients have no value
    of their own in 64 bits and would take minutes."""
    kind = case["kind"]
    if kind == "render" and case["scene"] == "room" and not case["adaptive"]:
        paths = case["w"] * case["h"] * math.ceil(math.sqrt(case["spp"])) ** 2
        return room_exact(case, seed) if paths <= 20e6 else None
    if kind == "aov":
        depth = sphere_depth_exact(case, seed)
        return [depth, None, None]
    if kind == "rays":
        if case["n"] * 2 * case["side"] ** 2 > 1e11:
            return None
        t, n = terrain_exact(case, seed)
        return {"t": t, "u": None, "v": None, "normal": n, "prim_id": None, "front_face": None, "material": None}
    return None


def draws(seed, pixel, stratum, bounce, call):
    """Philox4x32-10 (Salmon et al., SC'11) keyed by the seed, at counter (pixel, stratum, bounce,
    call): four uniforms in [0, 1) of 24 bits each."""
    m32 = 0xFFFFFFFF

    def mulhilo(m, x):     # 32 x 32 -> 64 bits in signed 64-bit arithmetic, by halves
        lo, hi = m * (x & 0xFFFF), m * (x >> 16)
        s = lo + ((hi & 0xFFFF) << 16)
        return (hi >> 16) + (s >> 32), s & m32

    c = [pixel, stratum, torch.full_like(pixel, bounce), torch.full_like(pixel, call)]
    k0, k1 = seed & m32, (seed >> 32) & m32
    for _ in range(10):
        h0, l0 = mulhilo(0xD2511F53, c[0])
        h1, l1 = mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return [(x >> 8).double() / 16777216.0 for x in c]


def vec(*xs):
    return torch.tensor(xs, dtype=torch.float64, device="cuda")


def unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def camera_frame(look_from, look_at, vfov, aspect, focus):
    """Origin, lower-left corner, horizontal, vertical and the lens axes of a camera."""
    o = vec(*look_from)
    w = unit(o - vec(*look_at))
    u = unit(torch.linalg.cross(vec(0.0, 1.0, 0.0), w))
    v = torch.linalg.cross(w, u)
    vh = 2.0 * math.tan(math.radians(vfov) / 2.0)
    hor, ver = u * (vh * aspect * focus), v * (vh * focus)
    return o, o - hor / 2 - ver / 2 - w * focus, hor, ver, u, v


def sphere_depth_exact(case, seed):
    """Depth of the sphere field along each pixel's centre ray (stratum 0's lens draw)."""
    rng = np.random.default_rng(seed)
    centres, radii = [(0, -1000, 0), (0, 1, 0), (-4, 1, 0), (4, 1, 0)], [1000.0, 1.0, 1.0, 1.0]
    for a in range(-case["grid"], case["grid"]):
        for b in range(-case["grid"], case["grid"]):
            choose = rng.random()
            centres.append((a + 0.9 * rng.random(), 0.2, b + 0.9 * rng.random()))
            radii.append(0.2)
            if choose < 0.8:
                rng.random(3), rng.random(3)
            elif choose < 0.95:
                rng.random(3), rng.random()
    w, h = case["w"], case["h"]
    o, llc, hor, ver, u, v = camera_frame((13, 2, 3), (0, 0, 0), 20.0, w / h, 10.0)
    pixel = torch.arange(w * h, device="cuda")
    _, _, lr, la = draws(seed, pixel, torch.zeros_like(pixel), 0, 0)
    x, y = (pixel % w).double() + 0.5, (h - 1 - pixel // w).double() + 0.5
    r = lr.sqrt() * 0.05
    off = u * (r * torch.cos(2 * math.pi * la))[:, None] + v * (r * torch.sin(2 * math.pi * la))[:, None]
    d = llc + hor * (x / (w - 1))[:, None] + ver * (y / (h - 1))[:, None] - o - off
    org = o + off
    a = (d * d).sum(-1)
    best = torch.full_like(a, math.inf)
    for c, rad in zip(centres, radii):
        oc = org - vec(*c)
        b = (oc * d).sum(-1)
        disc = b * b - a * ((oc * oc).sum(-1) - rad * rad)
        root = disc.clamp(min=0).sqrt()
        for t in ((-b - root) / a, (-b + root) / a):
            best = torch.where((disc >= 0) & (t >= 0.001) & (t < best), t, best)
    return torch.where(best.isfinite(), best, torch.zeros_like(best)).reshape(h, w)


def terrain_exact(case, seed):
    """Nearest hit distance and facing normal of every ray (Moller-Trumbore in f64 against every
    triangle whose block's bounding box the ray crosses)."""
    v, f = terrain(case["side"], seed)
    tri = torch.from_numpy(v).cuda()[torch.from_numpy(f.astype(np.int64)).cuda()]
    o, d = (torch.from_numpy(x).cuda().double() for x in ray_set(case["n"], seed))
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    normal = unit(torch.linalg.cross(e1, e2))
    best = torch.full((len(o),), math.inf, dtype=torch.float64, device="cuda")
    n = torch.zeros((len(o), 3), dtype=torch.float64, device="cuda")
    block = 128
    for k in range(0, len(tri), block):
        pts = tri[k:k + block].reshape(-1, 3)
        lo, hi = pts.min(0).values - 1e-6, pts.max(0).values + 1e-6
        ta, tb = (lo - o) / d, (hi - o) / d
        near, far = torch.minimum(ta, tb).max(-1).values, torch.maximum(ta, tb).min(-1).values
        idx = ((near <= far) & (far > 0) & (near < best)).nonzero()[:, 0]
        if not len(idx):
            continue
        for part in idx.split(1 << 18):
            oo, dd = o[part][:, None], d[part][:, None]
            a1, a2, p0 = e1[k:k + block][None], e2[k:k + block][None], tri[k:k + block, 0][None]
            hh = torch.linalg.cross(dd.expand(-1, a2.shape[1], -1), a2.expand(len(part), -1, -1))
            inv = 1.0 / (a1 * hh).sum(-1)
            s = oo - p0
            uu = (s * hh).sum(-1) * inv
            q = torch.linalg.cross(s, a1.expand(len(part), -1, -1))
            vv = (dd * q).sum(-1) * inv
            t = (a2 * q).sum(-1) * inv
            t = torch.where((uu >= 0) & (vv >= 0) & (uu + vv <= 1) & (t >= 0.001), t, math.inf)
            tm, at = t.min(-1)
            nearer = tm < best[part]
            best[part[nearer]] = tm[nearer]
            n[part[nearer]] = normal[k + at[nearer]]
    n = torch.where(((n * d).sum(-1) < 0)[:, None], n, -n)
    return best, torch.where(best.isfinite()[:, None], n, torch.zeros_like(n))


def room_quads():
    """Corner, edges, colour and emission of the box room's rectangles."""
    white, red, green = (0.73, 0.73, 0.73), (0.65, 0.05, 0.05), (0.12, 0.45, 0.15)
    quads = [((0, 0, 555), (555, 0, 0), (0, 555, 0), white, 0.0), ((213, 554, 227), (130, 0, 0), (0, 0, 105), (1, 1, 1), 15.0),
             ((0, 0, 0), (555, 0, 0), (0, 0, 555), white, 0.0), ((0, 555, 0), (555, 0, 0), (0, 0, 555), white, 0.0),
             ((0, 0, 0), (0, 555, 0), (0, 0, 555), red, 0.0), ((555, 0, 0), (0, 555, 0), (0, 0, 555), green, 0.0)]
    for (sx, sy, sz), degrees, shift in (((165, 330, 165), 15.0, (265, 0, 295)), ((165, 165, 165), -18.0, (130, 0, 65))):
        c, s = math.cos(math.radians(degrees)), math.sin(math.radians(degrees))

        def turn(p):
            return (c * p[0] + s * p[2], p[1], -s * p[0] + c * p[2])

        ex, ey, ez = (sx, 0, 0), (0, sy, 0), (0, 0, sz)
        for q, a, b in (((0, 0, 0), ex, ey), ((0, 0, sz), ex, ey), ((0, 0, 0), ex, ez), ((0, sy, 0), ex, ez),
                        ((0, 0, 0), ey, ez), ((sx, 0, 0), ey, ez)):
            quads.append((tuple(x + y for x, y in zip(turn(q), shift)), turn(a), turn(b), white, 0.0))
    return quads


def room_exact(case, seed):
    """The box room's frame, path by path in f64 on the same random numbers: diffuse bounces, one
    light sample per bounce, roulette on the survivors, luminance clamped at 100."""
    w, h, depth = case["w"], case["h"], case["depth"]
    root = math.ceil(math.sqrt(case["spp"]))
    quads = [(vec(*q), vec(*a), vec(*b)) for q, a, b, _, _ in room_quads()]
    normals = [torch.linalg.cross(a, b) for _, a, b in quads]
    ws = [n / (n * n).sum() for n in normals]
    colour = torch.stack([vec(*c) for _, _, _, c, _ in room_quads()])
    glow = torch.stack([vec(e, e, e) for *_, e in room_quads()])
    light_n, light_area = vec(0.0, -1.0, 0.0), 130.0 * 105.0
    look_from = (278.0 + seed % 41 - 20.0, 278.0, -800.0)
    o, llc, hor, ver, _, _ = camera_frame(look_from, (278, 278, 0), 40.0, w / h, 1.0)

    def hits(org, d, far):
        best, which = far.clone(), torch.full((len(org),), -1, dtype=torch.int64, device="cuda")
        for k, ((q, a, b), n) in enumerate(zip(quads, ws)):
            den = d @ n
            t = ((q * n).sum() - org @ n) / den
            rel = org + d * t[:, None] - q
            al, be = torch.linalg.cross(rel, b.expand_as(rel)) @ n, torch.linalg.cross(a.expand_as(rel), rel) @ n
            ok = (t >= 0.001) & (t <= best) & (al >= 0) & (al <= 1) & (be >= 0) & (be <= 1)
            best, which = torch.where(ok, t, best), torch.where(ok, k, which)
        return best, which

    total = torch.zeros((w * h, 3), dtype=torch.float64, device="cuda")
    weight = torch.zeros((w * h, 1), dtype=torch.float64, device="cuda")
    per = max(1, (1 << 21) // (w * h))
    for s0 in range(0, root * root, per):
        st = torch.arange(s0, min(root * root, s0 + per), device="cuda").repeat_interleave(w * h)
        pixel = torch.arange(w * h, device="cuda").repeat(len(st) // (w * h))
        cx, cy, _, _ = draws(seed, pixel, st, 0, 0)
        jx, jy = ((st % root) + cx) / root, ((st // root) + cy) / root
        d = (llc + hor * (((pixel % w) + jx) / (w - 1))[:, None] +
             ver * (((h - 1 - pixel // w) + jy) / (h - 1))[:, None] - o)
        org, path = o.expand_as(d), torch.arange(len(d), device="cuda")
        beta, radiance = torch.ones_like(d), torch.zeros_like(d)
        lit = torch.ones(len(d), dtype=torch.bool, device="cuda")   # emission counts at the next hit
        for bounce in range(depth):
            if not len(path):
                break
            t, k = hits(org, d, torch.full((len(org),), math.inf, dtype=torch.float64, device="cuda"))
            on = k >= 0
            path, org, d, t, k, beta, lit = (x[on] for x in (path, org, d, t, k, beta, lit))
            radiance.index_add_(0, path, beta * glow[k] * lit[:, None])
            p = org + d * t[:, None]
            n = unit(torch.stack(normals))[k]
            n = torch.where(((n * d).sum(-1) < 0)[:, None], n, -n)
            px, sx = pixel[path], st[path]
            a, b, _, _ = draws(seed, px, sx, bounce, 2)
            r0, ly, lu, lv = draws(seed, px, sx, bounce, 3)
            z = 1 - 2 * a
            r = (1 - z * z).clamp(min=0).sqrt()
            out = n + torch.stack([r * torch.cos(2 * math.pi * b), r * torch.sin(2 * math.pi * b), z], -1)
            albedo = colour[k]
            survive = albedo.max(-1).values.clamp(0.05, 1.0)
            keep = (glow[k][:, 0] == 0) & ~((depth - bounce < 47) & (r0 > survive))
            path, p, n, out, albedo, beta, survive, lu, lv = (
                x[keep] for x in (path, p, n, out, albedo, beta, survive, lu, lv))
            to = vec(213, 554, 227) + vec(130, 0, 0) * lu[:, None] + vec(0, 0, 105) * lv[:, None] - p
            d2 = (to * to).sum(-1)
            ld = to / d2.sqrt()[:, None]
            ct, cl = (n * ld).sum(-1), (ld @ light_n).abs()
            _, block = hits(p, ld, d2.sqrt() - 0.001)
            seen = (ct > 0) & (cl > 0.001) & (block < 0)
            gain = torch.where(seen, ct * cl * light_area / (math.pi * d2), torch.zeros_like(ct))
            radiance.index_add_(0, path, beta * albedo * 15.0 * gain[:, None])
            beta = beta * albedo / (survive[:, None] if depth - bounce < 47 else 1.0)
            org, d, lit = p, out, torch.zeros(len(path), dtype=torch.bool, device="cuda")
        lum = radiance @ vec(0.2126, 0.7152, 0.0722)
        radiance = radiance * (100.0 / lum.clamp(min=100.0))[:, None]
        x, y = jx - 0.5, jy - 0.5
        f = filter_weight(case["filter"], x, y)[:, None]
        total.index_add_(0, pixel, radiance * f)
        weight.index_add_(0, pixel, f)
    weight = torch.where(weight > 0, weight, torch.ones_like(weight))
    return (total / weight * case["exposure"]).reshape(h, w, 3)


def filter_weight(name, x, y):
    def mitchell(v):
        v = v.abs()
        near = ((12 - 9 / 3 - 6 / 3) * v ** 3 + (-18 + 12 / 3 + 6 / 3) * v ** 2 + 6 - 2 / 3) / 6
        far = ((-1 / 3 - 6 / 3) * v ** 3 + (6 / 3 + 30 / 3) * v ** 2 + (-12 / 3 - 48 / 3) * v + 8 / 3 + 24 / 3) / 6
        return torch.where(v < 1, near, torch.where(v < 2, far, torch.zeros_like(v)))

    if name == "triangle":
        return (1 - 2 * x.abs()).clamp(min=0) * (1 - 2 * y.abs()).clamp(min=0)
    if name == "gaussian":
        return torch.exp(-(x * x + y * y) / (2 * 0.35 ** 2))
    if name == "mitchell":
        return mitchell(2 * x) * mitchell(2 * y)
    return torch.ones_like(x)
