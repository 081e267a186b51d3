"""The estimate pass of the analytic trace (flat_closest, flat_blocked) against
the exact tests.

The pass takes scenes whose quads are axis-aligned rectangles or boxes.  Each
scene here is loaded twice: as it is, and with one far, tiny, slanted quad
added, which sends every ray through the exact tests.  Ids and t must agree
bit for bit, shadow answers too, and both with the oracle.  Rays: random ones,
ones aimed at the quads' borders and corners and at sphere silhouettes,
axis-parallel and nearly axis-parallel ones, origins on and next to surfaces
and far outside the scene, and directions that are not of unit length.
"""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _quad(o, u, v, material="grey", light=False):
    q = {"type": "plane", "origin": [float(x) for x in o], "u": [float(x) for x in u], "v": [float(x) for x in v],
         "material": material}
    if light:
        q["light"] = True
    return q


def _box(rng, c, half, angle, material="grey", digits=4, gap=0.0):
    """Six quads of a box turned about y, coordinates rounded as in a scene file."""
    ca, sa = np.cos(angle), np.sin(angle)
    ax = [np.array([ca, 0, -sa]) * 2 * half[0], np.array([0.0, 1, 0]) * 2 * half[1], np.array([sa, 0, ca]) * 2 * half[2]]
    p = np.asarray(c) - 0.5 * (ax[0] + ax[1] + ax[2])
    out = []
    for k in range(3):
        u, v = ax[(k + 1) % 3], ax[(k + 2) % 3]
        out.append(_quad(np.round(p, digits), np.round(u, digits), np.round(v, digits), material))
        out.append(_quad(np.round(p + ax[k] * (1 + gap), digits), np.round(u, digits), np.round(v, digits), material))
    return out


def _scene(kind, seed):
    rng = np.random.default_rng(seed)
    s = {"large": 60.0, "small": 0.05}.get(kind, 1.0)
    c = np.array([7.0, -3.0, 5.0]) * s if kind == "shifted" else np.zeros(3)
    prims = [_quad(c + np.array([-2, 2, -6]) * s, [4 * s, 0, 0], [0, 0, 7 * s]),          # ceiling
             _quad(c + np.array([2, 2, -6]) * s, [-6 * s, 0, 0], [0, -6 * s, 0]),         # back
             _quad(c + np.array([2, -2, 0]) * s, [0, 0, -7 * s], [-4 * s, 0, 0], "red"),  # floor
             _quad(c + np.array([2, -2, 0]) * s, [0, 4 * s, 0], [0, 0, -6 * s], "red"),
             _quad(c + np.array([-2, -2, -6]) * s, [0, 4 * s, 0], [0, 0, 6 * s]),
             # two more quads of the floor's plane, one over the other
             _quad(c + np.array([-1.5, -2, -3]) * s, [1 * s, 0, 0], [0, 0, 1 * s], "grey"),
             _quad(c + np.array([-1, -2, -2.5]) * s, [1 * s, 0, 0], [0, 0, 1 * s], "red")]
    prims += _box(rng, c + np.array([-0.9, -0.8, -4.0]) * s, np.array([0.6, 1.2, 0.6]) * s, 0.32)
    prims += _box(rng, c + np.array([0.9, -1.4, -2.8]) * s, np.array([0.6, 0.6, 0.6]) * s, -0.32, "red",
                  gap=0.02 if kind == "gap" else 0.0)
    if kind == "many":
        for k in range(70):
            o = np.round(rng.uniform(-1.8, 1.8, 3) + np.array([0, 0, -3]), 3)
            prims.append(_quad(o, [0.1, 0, 0], [0, 0.1, 0]))
    spheres = [{"type": "sphere", "center": [float(x) for x in c + np.array(p) * s], "radius": float(r * s), "material": m}
               for p, r, m in (((0.2, 0.9, -3.2), 0.5, "grey"), ((-1.2, 1.2, -2.0), 0.03, "red"),
                               ((1.1, 0.6, -4.5), 0.4, "glow" if kind == "glow" else "grey"))]
    prims.append(_quad(c + np.array([-0.375, 2, -4.25]) * s, [0.75 * s, 0, 0], [0, 0, 0.4 * s], "light", True))
    return {"schema": "1.0", "name": kind, "version": "1.0.0",
            "camera": {"position": [float(x) for x in c], "fov": 65},
            "materials": {"grey": {"albedo": [0.7, 0.7, 0.7]}, "red": {"albedo": [0.6, 0.1, 0.1]},
                          "glow": {"emissive": [2.0, 2.0, 1.0]}, "light": {"emissive": [80.0, 68.0, 48.0]}},
            "primitives": prims + spheres}, s, c


def _rays(sc, s, c, n, seed):
    rng = np.random.default_rng(seed)
    def inside(m):
        return np.stack([rng.uniform(-1.95, 1.95, m), rng.uniform(-1.95, 1.95, m), rng.uniform(-5.95, -0.05, m)], 1) * s + c
    o = inside(n)
    quads = [p for p in sc["primitives"] if p["type"] == "plane"]
    Q = np.array([p["origin"] + p["u"] + p["v"] for p in quads])
    k = rng.integers(0, len(quads), n)
    a, b = rng.uniform(0, 1, n), rng.uniform(0, 1, n)
    edge = rng.integers(0, 4, n)
    a = np.where(edge == 0, np.round(a), a)
    b = np.where(edge == 1, np.round(b), np.where(edge == 2, np.round(b * 2) / 2, b))
    target = Q[k, :3] + Q[k, 3:6] * a[:, None] + Q[k, 6:9] * b[:, None]
    d = rng.normal(size=(n, 3))
    sel = np.arange(n) % 3 == 0
    d[sel] = (target - o)[sel]
    # sphere silhouettes: aim at points r from the centre, across the view
    sp = [p for p in sc["primitives"] if p["type"] == "sphere"]
    S = np.array([p["center"] + [p["radius"]] for p in sp])
    sel = np.arange(n) % 17 == 1
    j = rng.integers(0, len(sp), n)
    w = S[j, :3] - o
    x = np.cross(w, rng.normal(size=(n, 3)))
    x /= np.maximum(np.linalg.norm(x, axis=1, keepdims=True), 1e-30)
    d[sel] = (w + x * S[j, 3:4] * (1 + rng.normal(0, 3e-4, (n, 1))))[sel]
    # starts on and next to surfaces
    sel = np.arange(n) % 5 == 2
    o[sel] = (target + rng.normal(0, 1, (n, 3)) * s * rng.choice([0.0, 1e-6, 1e-4, 1e-3], (n, 1)))[sel]
    # far origins
    sel = np.arange(n) % 31 == 3
    far = target + rng.normal(size=(n, 3)) * 40 * s
    o[sel], d[sel] = far[sel], (target - far)[sel]
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)
    # axis-parallel, nearly so, and other lengths
    sel = np.arange(n) % 11 == 4
    ax = rng.integers(0, 3, n)
    eps = rng.choice([0.0, 1e-7, 1e-6, 2e-6, 5e-6, 1e-4], n) * rng.choice([-1, 1], n)
    dd = np.tile(eps[:, None], (1, 3))
    dd[np.arange(n), ax] = rng.choice([-1, 1], n)
    d[sel] = dd[sel]
    sel = np.arange(n) % 41 == 5
    d[sel] *= rng.choice([0.3, 0.98, 1.004, 1.02, 7.0], (n, 1))[sel]
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.fixture(scope="module")
def ctx():
    from pcr_b200 import capi
    c = capi.Context(device=0, queue_capacity=1 << 17)
    yield c
    c.close()


@pytest.mark.parametrize("kind", ["plain", "large", "small", "shifted", "gap", "glow", "many"])
def test_estimates_agree_with_exact_tests(ctx, tmp_path, kind):
    from oracle import oracle as O
    O.build()
    sc, s, c = _scene(kind, 3)
    extra = json.loads(json.dumps(sc))
    at = c + np.array([0, 0, 900.0]) * s
    extra["primitives"].append(_quad(at, np.array([1e-3, 1e-3, 0]) * s, np.array([0, 1e-3, 1e-3]) * s))
    paths = []
    for name, x in (("fast", sc), ("exact", extra)):
        paths.append(str(tmp_path / f"{name}.json"))
        with open(paths[-1], "w") as f:
            json.dump(x, f)
    fast, exact = (ctx.load_scene_json(p, str(tmp_path)) for p in paths)
    n = 300_000
    rays = _rays(sc, s, c, n, 17)
    m0, p0, t0 = ctx.trace_closest(fast, rays)
    m1, p1, t1 = ctx.trace_closest(exact, rays)
    assert np.array_equal(p0, p1) and np.array_equal(m0, m1)
    assert np.array_equal(t0.view(np.uint32), t1.view(np.uint32))
    assert 0.3 < (p0 != 0).mean()
    omat, _ = O.scene_intersect(O.load_scene(paths[0], str(tmp_path)), rays)
    assert np.array_equal(m0, omat)
    # shadow segments: the ray's length to some point, on a light for a third of them
    rng = np.random.default_rng(5)
    light = [p for p in sc["primitives"] if p.get("light")][0]
    L = (np.array(light["origin"]) + np.array(light["u"]) * rng.uniform(0, 1, (n, 1))
         + np.array(light["v"]) * rng.uniform(0, 1, (n, 1)))
    to = (L - rays[:, :3]).astype(np.float32)
    d2 = (rng.uniform(0.01, 5, n) ** 2 * s * s).astype(np.float32)
    sel = np.arange(n) % 3 == 0
    sel &= (to * to).sum(1) > 1e-8
    d2[sel] = (to[sel] * to[sel]).sum(1, dtype=np.float32)
    rays[sel, 3:] = to[sel] / np.sqrt(d2[sel])[:, None]
    b0, b1 = ctx.trace_shadow(fast, rays, d2), ctx.trace_shadow(exact, rays, d2)
    assert np.array_equal(b0, b1)
    assert 0.02 < b0.mean() < 0.98
    for sid in (fast, exact):
        ctx.release_scene(sid)


@pytest.mark.parametrize("scene,kw", [
    ("cornell", dict(depth=1, samples=1, shadow=1, spectral=False)),
    ("cornell", dict(depth=6, samples=5, shadow=3, spectral=True, hero=1)),
    ("cornell-spheres", dict(depth=4, samples=4, shadow=2, spectral=False, mis=True, russian=True, stratified=True, aa=2)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, spectral=True, hero=3)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, spectral=True, terminate=True)),
    ("closed-cornell-glass", dict(depth=8, samples=2, shadow=8, spectral=True)),
])
@pytest.mark.parametrize("size", [(1, 1), (33, 7), (128, 96)])
def test_whole_paths_equal_queue_stages(ctx, tmp_path, scene, kw, size):
    """The whole-path kernel (scenes without a mesh) against the queue stages:
    the same scene with a triangle far behind the camera goes through the
    queues and must give the same image (each sample's value is the same;
    only the FP64 summation order differs)."""
    from conftest import GOLDEN, scene_path
    from pcr_b200 import capi, workloads
    sc = workloads.read_scene_json(scene_path(scene))
    (tmp_path / "tri.obj").write_text("v 0 0 0\nv 0.001 0 0\nv 0 0.001 0\nf 1 2 3\n")
    sc["primitives"].insert(0, {"type": "mesh", "file": "tri.obj", "position": [0, 0, 5000.0],
                                "material": next(k for k, m in sc["materials"].items() if "emissive" not in m)})
    p = tmp_path / "queue.json"
    p.write_text(json.dumps(sc))
    import shutil, os
    if os.path.isdir(os.path.join(GOLDEN, "spd")):
        shutil.copytree(os.path.join(GOLDEN, "spd"), tmp_path / "spd")
    a, b = ctx.load_scene_json(scene_path(scene), GOLDEN), ctx.load_scene_json(str(p), str(tmp_path))
    d = capi.render_desc(size[0], size[1], seed=11, **kw)
    whole, queue = ctx.render(a, d), ctx.render(b, d)
    assert np.allclose(whole[0], queue[0], rtol=1e-6, atol=1e-7)
    ids = [ctx.submit(s, d) for s in (a, b)]
    ctx.run_until_idle()
    for rid in ids:
        assert np.allclose(ctx.fetch(rid)[0], whole[0], rtol=1e-6, atol=1e-7)
    for sid in (a, b):
        ctx.release_scene(sid)
