"""Performance cases of the path tracer, through its public entry points.

Each case is one call (or one submit / run / fetch round) as a program that
uses pcr_b200.capi makes it: a context and its resident scenes are kept, the
inputs (render seeds, rays, images, triangles) are new ones per seed.

Kinds
  plain     Context.render: one render, images returned in host arrays
  noalloc   Context.render_noalloc: one render into caller device buffers
  batch     submit all, run_until_idle, fetch each into the caller's buffers
  rays      Context.trace_closest / trace_bvh / trace_shadow on host rays
  bvh       Context.build_bvh: SAH tree of a triangle soup
  post      Context.tonemap: 8-bit image of a linear image (and denoise)

Images have no value in 64 bits apart from the renderer's own: a path is a
chain of decisions on float32 comparisons (which surface is hit first, which
of two coplanar quads wins a tie, whether a shadow point lies 1e-3 in front
of a light), which the renderer makes with the reference's float32
operations; another precision traces other paths.  exact() therefore gives
values for ray queries against scenes without a mesh, whose distances do
have one.
"""
import functools
import math
import os

import numpy as np
import torch

from pcr_b200 import capi, workloads

# scenes of the repository by name; ico* are the seeded mesh scenes of its
# batched-mesh workload (about 70k triangles)
PLANE_SCENES = ["cornell", "cornell-spec", "cornell-glass", "cornell-spheres", "closed-cornell-spec",
                "cornell-large-light", "bright-cornell-glass", "closed-cornell-glass", "cornell-frank"]
MESH_SCENES = ["cornell-bunny", "ico59-diffuse", "ico59-glass"]


def listed():
    return [
        # the smallest call: a thumbnail, where launches and host work are all there is
        {"name": "thumbnail", "kind": "plain", "scene": "cornell", "width": 64, "height": 64, "depth": 2, "samples": 1,
         "shadow": 1, "spectral": False},
        # the reference's default-quality spectral render of the Cornell box
        {"name": "cornell-256", "kind": "plain", "scene": "cornell", "width": 256, "height": 256, "depth": 4,
         "samples": 16, "shadow": 4, "spectral": True},
        # an RGB preview at an odd size with every sampling option on
        {"name": "preview-rgb", "kind": "plain", "scene": "cornell-spheres", "width": 719, "height": 405, "depth": 3,
         "samples": 4, "shadow": 2, "spectral": False, "mis": True, "russian": True, "stratified": True, "aces": True},
        # dispersive glass, deep paths: hero wavelengths fork
        {"name": "glass-deep", "kind": "plain", "scene": "closed-cornell-glass", "width": 500, "height": 500,
         "depth": 8, "samples": 8, "shadow": 2, "spectral": True},
        # a triangle mesh through the plain method
        {"name": "bunny", "kind": "plain", "scene": "cornell-bunny", "width": 320, "height": 320, "depth": 4,
         "samples": 8, "shadow": 4, "spectral": True},
        # adaptive anti-aliasing rounds and the denoiser
        {"name": "adaptive", "kind": "plain", "scene": "cornell-large-light", "width": 300, "height": 300, "depth": 3,
         "samples": 2, "shadow": 2, "spectral": True, "aa": 12, "adaptive": True, "denoise": True},
        # a host that may not allocate while it renders: device buffers in, device buffers out
        {"name": "noalloc", "kind": "noalloc", "scene": "cornell-spec", "width": 256, "height": 256, "depth": 4,
         "samples": 8, "shadow": 4, "spectral": True},
        # the throughput workload: uneven requests over all scene variants in one wavefront
        {"name": "batch-uneven", "kind": "batch", "requests": 24, "scenes": "variants", "res_lo": 128, "res_hi": 1024,
         "depth_hi": 8, "spp_hi": 64, "shadow_hi": 8, "layout": 2026},
        # mesh renders batched, glass and Lambertian
        {"name": "batch-mesh", "kind": "batch", "requests": 6, "scenes": "mesh", "res_lo": 384, "res_hi": 640,
         "depth_hi": 8, "spp_hi": 32, "shadow_hi": 4, "layout": 11},
        # closest-hit queries on caller rays
        {"name": "rays-closest", "kind": "rays", "what": "closest", "scene": "cornell-spheres", "rays": 400_001},
        # the device BVH build of a mid-size mesh
        {"name": "bvh-build", "kind": "bvh", "triangles": 200_000},
        # tone map and denoise of a finished HDR frame
        {"name": "denoise-720p", "kind": "post", "width": 1280, "height": 720, "denoise": True, "aces": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "plain", "noalloc", "batch", "batch", "rays", "bvh", "post"])
    if kind in ("plain", "noalloc"):
        mesh = kind == "plain" and rng.random() < 0.3
        side = (16, 256) if kind == "noalloc" else (24, 400) if mesh else (24, 1024)
        w, h = _log_int(rng, *side), _log_int(rng, *side)
        c = {"kind": kind, "scene": rng.choice(MESH_SCENES if mesh else PLANE_SCENES), "width": w, "height": h,
             "depth": rng.randint(1, 8), "samples": _log_int(rng, 1, 32), "shadow": rng.randint(1, 8),
             "spectral": rng.random() < 0.7, "mis": rng.random() < 0.3, "russian": rng.random() < 0.3,
             "stratified": rng.random() < 0.3, "aces": rng.random() < 0.3, "denoise": rng.random() < 0.2}
        if kind == "plain" and rng.random() < 0.3:
            c["aa"] = rng.randint(2, 4)
        if rng.random() < 0.2:
            c["hero"] = rng.randint(1, 3)
        if rng.random() < 0.2:
            c["terminate"] = True
        # at most the largest listed render's work
        while w * h * c["samples"] * c.get("aa", 1) > (2_000_000 if mesh else 20_000_000):
            c["samples"] = max(1, c["samples"] // 2)
            if c["samples"] == 1:
                c.pop("aa", None)
                break
        return c
    if kind == "batch":
        mesh = rng.random() < 0.3
        return {"kind": "batch", "requests": rng.randint(2, 5 if mesh else 20), "scenes": "mesh" if mesh else "variants",
                "res_lo": 64, "res_hi": _log_int(rng, 128, 512 if mesh else 1024), "depth_hi": rng.randint(3, 8),
                "spp_hi": _log_int(rng, 2, 8 if mesh else 48), "shadow_hi": rng.randint(1, 4 if mesh else 8),
                "layout": rng.randrange(1 << 30)}
    if kind == "rays":
        return {"kind": "rays", "what": rng.choice(["closest", "bvh", "shadow"]),
                "scene": rng.choice(["cornell", "cornell-spheres", "cornell-bunny", "ico59-diffuse"]),
                "rays": _log_int(rng, 100, 1_000_000)}
    if kind == "bvh":
        return {"kind": "bvh", "triangles": _log_int(rng, 10, 250_000)}
    return {"kind": "post", "width": _log_int(rng, 30, 1920), "height": _log_int(rng, 30, 1080),
            "denoise": rng.random() < 0.5, "aces": rng.random() < 0.5}


# ------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=None)
def _context(queue_capacity):
    if queue_capacity:
        # a tuned throughput context (what the autotuner picks, at a queue size that leaves room beside it)
        return capi.Context(queue_capacity=queue_capacity, block_size=256, chunk_paths=1 << 14, regen_every=2)
    return capi.Context()


@functools.lru_cache(maxsize=None)
def _scene(queue_capacity, name):
    if name.startswith("ico59"):
        path = workloads.mesh_scene(59, 1, glass=name.endswith("glass"))
        data = workloads.DEFAULT_DATA
    else:
        path, data = workloads.scene_path(name), workloads.DEFAULT_DATA
    return _context(queue_capacity).load_scene_json(path, data)


def _desc(c, seed):
    return capi.render_desc(c["width"], c["height"], depth=c["depth"], samples=c["samples"], shadow=c["shadow"],
                            spectral=c.get("spectral", True), hero=c.get("hero", 4), mis=c.get("mis", False),
                            russian=c.get("russian", False), stratified=c.get("stratified", False),
                            aa=c.get("aa", 1), adaptive=c.get("adaptive", False), aces=c.get("aces", False),
                            denoise=c.get("denoise", False), terminate=c.get("terminate", False), seed=seed)


def _requests(c):
    """The batch's requests without seeds: (scene, width, height, depth, samples, shadow)."""
    rng = np.random.default_rng(c["layout"])
    names = workloads.VARIANTS if c["scenes"] == "variants" else ["ico59-diffuse", "ico59-glass"]
    out = []
    for i in range(c["requests"]):
        side = int(round(math.exp(rng.uniform(math.log(c["res_lo"]), math.log(c["res_hi"])))))
        spp = int(round(math.exp(rng.uniform(0.0, math.log(c["spp_hi"])))))
        name = names[i % 2] if c["scenes"] == "mesh" else names[int(rng.integers(len(names)))]
        out.append((name, side, side, int(rng.integers(2, c["depth_hi"] + 1)), spp,
                    int(rng.integers(1, c["shadow_hi"] + 1))))
    return out


def _rays(n, seed):
    """Rays that start inside the box, in all directions."""
    rng = np.random.default_rng(seed)
    o = np.stack([rng.uniform(-1.9, 1.9, n), rng.uniform(-1.9, 1.9, n), rng.uniform(-5.9, -0.1, n)], 1)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


def _mesh(n, seed):
    """n triangles of a bumpy closed surface, in scan order (as a modeller writes them)."""
    rng = np.random.default_rng(seed)
    rows = max(1, int(math.sqrt(n / 4)))
    cols = max(3, -(-n // (2 * rows)))
    th = np.linspace(0.0, math.pi, rows + 1)[:, None]
    ph = np.linspace(0.0, 2 * math.pi, cols + 1)[None, :]
    k = rng.integers(1, 9, (6, 2))
    a = rng.uniform(0, 2 * math.pi, 6)
    r = 0.8 + sum(0.02 * np.sin(k[i, 0] * th + a[i]) * np.cos(k[i, 1] * ph) for i in range(6))
    p = np.stack([r * np.sin(th) * np.cos(ph), r * np.cos(th) * np.ones_like(ph), r * np.sin(th) * np.sin(ph)], -1)
    p = p + rng.normal(0.0, 1e-3, p.shape)
    q = np.stack([np.concatenate([p[:-1, :-1], p[1:, :-1], p[:-1, 1:]], -1),
                  np.concatenate([p[1:, :-1], p[1:, 1:], p[:-1, 1:]], -1)], 2)
    return np.ascontiguousarray(q.reshape(-1, 9)[:n], np.float32)


def prepare(case, seed):
    kind = case["kind"]
    render_seed = 1 + (seed * 2654435761) % (2 ** 31 - 1)
    s = {"case": case, "kind": kind}
    if kind in ("plain", "noalloc"):
        s["ctx"], s["sid"] = _context(0), _scene(0, case["scene"])
        s["desc"] = _desc(case, render_seed)
        if kind == "noalloc":
            s["hdr"] = torch.zeros(case["height"], case["width"], 3, dtype=torch.float32, device="cuda")
            s["rgb"] = torch.zeros(case["height"], case["width"], 3, dtype=torch.uint8, device="cuda")
    elif kind == "batch":
        q = 1 << 22
        s["ctx"], s["jobs"] = _context(q), []
        for i, (name, w, h, depth, spp, shadow) in enumerate(_requests(case)):
            d = capi.render_desc(w, h, depth=depth, samples=spp, shadow=shadow, seed=render_seed + i)
            s["jobs"].append((_scene(q, name), d, np.zeros((h, w, 3), np.float32), np.zeros((h, w, 3), np.uint8)))
    elif kind == "rays":
        s["ctx"], s["sid"] = _context(0), _scene(0, case["scene"])
        s["rays"] = _rays(case["rays"], seed)
        if case["what"] == "shadow":
            s["dist2"] = np.random.default_rng(seed + 1).uniform(0.05, 16.0, case["rays"]).astype(np.float32)
    elif kind == "bvh":
        s["ctx"], s["tris"] = _context(0), _mesh(case["triangles"], seed)
    else:
        s["ctx"] = _context(0)
        rng = np.random.default_rng(seed)
        y, x = np.mgrid[0:case["height"], 0:case["width"]].astype(np.float32)
        base = 0.6 + 0.5 * np.sin(x / 90.0 + rng.uniform(0, 6)) * np.cos(y / 70.0 + rng.uniform(0, 6))
        img = base[..., None] * np.array([1.0, 0.8, 0.6], np.float32)
        s["hdr"] = (img * rng.gamma(8.0, 1.0 / 8.0, img.shape)).astype(np.float32)   # Monte-Carlo noise
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "plain":
        hdr, rgb, _ = ctx.render(s["sid"], s["desc"])
        return hdr, rgb
    if kind == "noalloc":
        ctx.render_noalloc(s["sid"], s["desc"], s["hdr"].data_ptr(), s["rgb"].data_ptr())
        return s["hdr"], s["rgb"]
    if kind == "batch":
        ids = [ctx.submit(sid, d) for sid, d, _, _ in s["jobs"]]
        ctx.run_until_idle()
        for rid, (_, _, hdr, rgb) in zip(ids, s["jobs"]):
            ctx.fetch(rid, hdr_out=hdr, rgb_out=rgb)
        return [[hdr, rgb] for _, _, hdr, rgb in s["jobs"]]
    if kind == "rays":
        if s["case"]["what"] == "closest":
            return ctx.trace_closest(s["sid"], s["rays"])
        if s["case"]["what"] == "bvh":
            return ctx.trace_bvh(s["sid"], s["rays"])
        return ctx.trace_shadow(s["sid"], s["rays"], s["dist2"])
    if kind == "bvh":
        nodes, order = ctx.build_bvh(s["tris"])
        # rows for the most nodes a tree of n triangles can have; the last three words of a node are integers
        pad = np.zeros((2 * len(order) - 1, 9), np.float32)
        pad[:len(nodes)] = nodes
        return pad[:, :6], pad.view(np.int32)[:, 6:], order
    return ctx.tonemap(s["hdr"], aces=s["case"]["aces"], denoise=s["case"]["denoise"])


# ------------------------------------------------------------------ what a pass cannot do without
PLANE_FLOPS = 25       # one quad test: two 3-vector products, a quotient, the quad's projections
SCENE_TESTS = 10       # quad or sphere tests a ray needs in the box scenes
MEAN_VERTICES = 3.0    # vertices of a path that is not cut by its depth
MESH_FLOPS = 600       # a ray through a binary SAH tree of 70k triangles: about 20 nodes and 6 triangles


def _render_work(c, mesh):
    paths = c["width"] * c["height"] * c["samples"] * c.get("aa", 1)
    rays = paths * min(c["depth"], MEAN_VERTICES) * (1 + c["shadow"])
    flops = rays * (PLANE_FLOPS * SCENE_TESTS + (MESH_FLOPS if mesh else 0))
    return 15 * c["width"] * c["height"], flops


def work(case):
    kind = case["kind"]
    if kind in ("plain", "noalloc"):
        b, f = _render_work(case, case["scene"] in MESH_SCENES)
    elif kind == "batch":
        b = f = 0
        for name, w, h, depth, spp, shadow in _requests(case):
            x = _render_work({"width": w, "height": h, "depth": depth, "samples": spp, "shadow": shadow},
                             name in MESH_SCENES)
            b, f = b + x[0], f + x[1]
    elif kind == "rays":
        n, mesh = case["rays"], case["scene"] in MESH_SCENES
        b = n * {"closest": 24 + 12, "bvh": 24 + 8, "shadow": 28 + 4}[case["what"]]
        f = n * (PLANE_FLOPS * SCENE_TESTS + (MESH_FLOPS if mesh else 0))
    elif kind == "bvh":
        n = case["triangles"]
        # vertices in; nodes and order out; binning of three axes once per level
        b, f = n * (36 + 36 + 4), n * max(1.0, math.log2(max(2, n))) * 3 * 12
    else:
        px = case["width"] * case["height"]
        b, f = px * 15, px * (20 + (2 * 25 * 20 if case["denoise"] else 0))
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------ values in 64 bits
def _scene_arrays(name):
    h = capi.HostScene(workloads.scene_path(name), workloads.DEFAULT_DATA)
    planes, spheres = h.planes().astype(np.float64), h.spheres().astype(np.float64)
    h.close()
    return planes, spheres


def exact(case, seed):
    if case["kind"] != "rays" or case["what"] != "closest" or case["scene"] not in PLANE_SCENES:
        return None
    planes, spheres = _scene_arrays(case["scene"])
    r = torch.from_numpy(_rays(case["rays"], seed)).double()
    o, d = r[:, :3], r[:, 3:]
    best = torch.full((r.shape[0],), math.inf, dtype=torch.float64)
    for p in spheres:
        cp = torch.from_numpy(p[:3]) - o
        b = (d * cp).sum(1)
        q = (cp * cp).sum(1) - b * b
        half = torch.sqrt(torch.clamp(p[3] ** 2 - q, min=0.0))
        t = torch.where(b - half < 0, b + half, b - half)
        best = torch.where((q <= p[3] ** 2) & (t >= 0) & (t < best), t, best)
    for p in planes:
        po, u, v, n = (torch.from_numpy(p[i:i + 3]) for i in (0, 3, 6, 9))
        den = d @ n
        t = ((po - o) @ n) / den
        lh = o + d * t[:, None] - po
        a, b = (lh @ u) / (u @ u), (lh @ v) / (v @ v)
        ok = (den.abs() > 1e-6) & (t > 1e-6) & (a >= 0) & (a <= 1) & (b >= 0) & (b <= 1) & (t < best)
        best = torch.where(ok, t, best)
    t = torch.where(torch.isfinite(best), best, torch.zeros_like(best))
    return None, None, t.numpy()
