"""Ray queries that start on a sphere, or as close to it as a float can say.

There the sign of |centre - origin|^2 - radius^2 is inside its own rounding
error, and the reference's operations may answer t = 0 as well as the far
root.  The estimate pass must leave such rays to the exact tests.  Every scene
is loaded twice, as it is and with one far, tiny, slanted quad that sends each
ray through the exact tests: ids, t and shadow answers must agree bit for bit,
and the materials with the oracle's.
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


def _room(spheres, light_y=2.0):
    prims = [_quad([-2, 2, -6], [4, 0, 0], [0, 0, 7]), _quad([2, 2, -6], [-6, 0, 0], [0, -6, 0]),
             _quad([2, -2, 0], [0, 0, -7], [-4, 0, 0], "red"), _quad([2, -2, 0], [0, 4, 0], [0, 0, -6], "red"),
             _quad([-2, -2, -6], [0, 4, 0], [0, 0, 6]),
             _quad([-0.375, light_y, -4.0], [0.75, 0, 0], [0, 0, 0.5], "light", True)]
    prims += [{"type": "sphere", "center": list(c), "radius": r, "material": m} for c, r, m in spheres]
    return {"schema": "1.0", "name": "room", "version": "1.0.0", "camera": {"position": [0.0, 0.0, 0.0], "fov": 65},
            "materials": {"grey": {"albedo": [0.7, 0.7, 0.7]}, "red": {"albedo": [0.6, 0.1, 0.1]},
                          "glow": {"emissive": [2.0, 2.0, 1.0]}, "light": {"emissive": [80.0, 68.0, 48.0]}},
            "primitives": prims}


ROOMS = {
    "free": _room([((0.2, 0.9, -3.2), 0.5, "grey"), ((1.1, -0.6, -4.5), 0.4, "red")]),
    # cut by the floor, and by one another
    "sunk": _room([((0.2, -1.9, -3.2), 0.5, "grey"), ((1.0, 0.6, -4.5), 0.4, "red"), ((1.3, 0.6, -4.5), 0.4, "grey")]),
    "light-inside": _room([((0.0, 1.0, -3.75), 0.9, "grey"), ((1.1, -0.6, -4.5), 0.4, "red")], light_y=1.0),
    "emissive": _room([((0.2, -0.9, -3.2), 0.5, "glow"), ((0.2, -1.5, -3.2), 0.5, "grey")]),
}


def _starts(spheres, n, rng):
    """Origins inside the room, three quarters of them on or next to a sphere."""
    o = np.stack([rng.uniform(-1.95, 1.95, n), rng.uniform(-1.95, 1.95, n), rng.uniform(-5.95, -0.05, n)], 1)
    S = np.array([list(s["center"]) + [abs(s["radius"])] for s in spheres])
    j = rng.integers(0, len(S), n)
    w = rng.normal(size=(n, 3))
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    off = np.where(np.arange(n) % 4 == 1, 0.0, rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-8, -3, n))
    on = S[j, :3] + w * (S[j, 3] + off)[:, None]
    return np.where((np.arange(n) % 4 == 0)[:, None], o, on).astype(np.float32)


def _agree(ctx, tmp_path, sc, seed):
    from oracle import oracle as O
    O.build()
    exact = json.loads(json.dumps(sc))
    exact["primitives"].append(_quad([0, 0, 900.0], [1e-3, 1e-3, 0], [0, 1e-3, 1e-3]))
    paths = []
    for name, x in (("fast", sc), ("exact", exact)):
        paths.append(str(tmp_path / f"{name}.json"))
        with open(paths[-1], "w") as f:
            json.dump(x, f)
    sids = [ctx.load_scene_json(p, str(tmp_path)) for p in paths]
    rng = np.random.default_rng(seed)
    n = 1_000_000
    spheres = [p for p in sc["primitives"] if p["type"] == "sphere"]
    o = _starts(spheres, n, rng)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d.astype(np.float32)], 1)
    (m0, p0, t0), (m1, p1, t1) = (ctx.trace_closest(s, rays) for s in sids)
    assert np.array_equal(p0, p1) and np.array_equal(m0, m1), f"{(p0 != p1).sum()} hits differ"
    assert np.array_equal(t0.view(np.uint32), t1.view(np.uint32))
    omat, _ = O.scene_intersect(O.load_scene(paths[0], str(tmp_path)), rays)
    assert np.array_equal(m0, omat)
    # shadow segments of any length, to the light, and to points inside the spheres
    light = [p for p in sc["primitives"] if p.get("light")][0]
    to = (np.array(light["origin"]) + np.array(light["u"]) * rng.uniform(0, 1, (n, 1))
          + np.array(light["v"]) * rng.uniform(0, 1, (n, 1)) - o)
    S = np.array([list(s["center"]) + [s["radius"]] for s in spheres])
    j = rng.integers(0, len(S), n)
    sel = np.arange(n) % 3 == 1
    to[sel] = (S[j, :3] + rng.uniform(-0.5, 0.5, (n, 3)) * S[j, 3:] - o)[sel]
    to = to.astype(np.float32)
    d2 = (to * to).sum(1, dtype=np.float32)
    sel = (np.arange(n) % 3 == 2) | (d2 < 1e-8)
    aimed = rays.copy()
    aimed[~sel, 3:] = to[~sel] / np.sqrt(d2[~sel])[:, None]
    d2[sel] = rng.uniform(0.01, 5, sel.sum()).astype(np.float32) ** 2
    b0, b1 = (ctx.trace_shadow(s, aimed, d2) for s in sids)
    assert np.array_equal(b0, b1), f"{(b0 != b1).sum()} shadow answers differ"
    assert 0.02 < b0.mean() < 0.98
    for s in sids:
        ctx.release_scene(s)


@pytest.fixture(scope="module")
def ctx():
    from pcr_b200 import capi
    c = capi.Context(device=0, queue_capacity=1 << 17)
    yield c
    c.close()


@pytest.mark.parametrize("kind", list(ROOMS))
def test_rays_that_start_on_a_sphere(ctx, tmp_path, kind):
    _agree(ctx, tmp_path, ROOMS[kind], 7)


@pytest.mark.parametrize("radii", [(0.0, 1e-5, 1.99), (-0.5, -1.4, 0.3), (-300.0, 0.5, 0.0)])
def test_spheres_of_zero_and_negative_radius(ctx, tmp_path, radii):
    """The intersection only uses the radius's square: a point sphere is met
    from its centre, a negative radius counts as its magnitude."""
    a, b, c = radii
    _agree(ctx, tmp_path, _room([((0.2, -1.9, -3.2), a, "grey"), ((1.1, -0.6, -4.5), b, "red"),
                                 ((0.0, 0.0, -3.0), c, "grey")]), 11)
