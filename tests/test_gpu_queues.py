"""Paths and shadow rays that go through the queues.

A path waits in the path queue, and a shadow ray becomes a record, where it
meets the box of the scene's triangle mesh.  Each scene here is rendered as it
is and with a mesh of two tiny triangles far outside opposite corners, whose
box holds the whole room while no ray meets a triangle: every path then waits
at every vertex and every lit shadow ray is a record, and images (up to the
order of the FP64 sums), ray counts and shadow-ray counts must stay the same.
"""
import json
import os
import shutil

import numpy as np
import pytest

from conftest import GOLDEN, scene_path

pytestmark = pytest.mark.gpu

OBJ = "v -50 -50 -50\nv -49.999 -50 -50\nv -50 -49.999 -50\nv 50 50 50\nv 49.999 50 50\nv 50 49.999 50\nf 1 2 3\nf 4 5 6\n"


def _boxed(tmp_path, scene):
    """The scene's file with the two-triangle mesh added, and its data root."""
    from pcr_b200 import workloads
    sc = workloads.read_scene_json(scene_path(scene))
    root = tmp_path / scene
    root.mkdir()
    (root / "corners.obj").write_text(OBJ)
    if os.path.isdir(os.path.join(GOLDEN, "spd")):
        shutil.copytree(os.path.join(GOLDEN, "spd"), root / "spd")
    sc["primitives"].insert(0, {"type": "mesh", "file": "corners.obj", "position": [0, 0, 0],
                                "material": next(k for k, m in sc["materials"].items() if "emissive" not in m)})
    path = root / "boxed.json"
    path.write_text(json.dumps(sc))
    return str(path), str(root)


def _counts(ctx, sid, desc):
    ctx.reset_stats()
    images = ctx.render(sid, desc)[:2]
    st = ctx.stats()
    return images, (st["paths"], st["rays"], st["shadow_rays"]), st


@pytest.mark.parametrize("capacity", [1 << 10, 1 << 17])
@pytest.mark.parametrize("scene,kw", [
    ("cornell", dict(depth=1, samples=2, shadow=1, spectral=False)),
    ("cornell", dict(depth=5, samples=4, shadow=3, russian=True)),
    ("cornell-glass", dict(depth=6, samples=3, shadow=2)),
])
def test_ray_counts_do_not_depend_on_the_queue(tmp_path, capacity, scene, kw):
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=capacity)
    a = ctx.load_scene_json(scene_path(scene), GOLDEN)
    b = ctx.load_scene_json(*_boxed(tmp_path, scene))
    d = capi.render_desc(70, 41, seed=23, **kw)
    assert _counts(ctx, b, d)[1] == _counts(ctx, a, d)[1]
    ctx.close()
