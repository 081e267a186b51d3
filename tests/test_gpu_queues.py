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
    root.mkdir(parents=True)
    (root / "corners.obj").write_text(OBJ)
    if os.path.isdir(os.path.join(GOLDEN, "spd")):
        shutil.copytree(os.path.join(GOLDEN, "spd"), root / "spd")
    sc["primitives"].insert(0, {"type": "mesh", "file": "corners.obj", "position": [0, 0, 0],
                                "material": next(k for k, m in sc["materials"].items() if "emissive" not in m)})
    path = root / "boxed.json"
    path.write_text(json.dumps(sc))
    return str(path), str(root)


def _counts(ctx, sid, desc, batch=False):
    """A render's images, its path and ray counts, and the stats.  batch: in
    one with a request of more paths than are staged (on the scene alone, so
    that the path kernel of mesh scenes follows both); its counts are left
    out."""
    from pcr_b200 import capi
    if batch:
        big = capi.render_desc(300, 250, depth=1, samples=1, shadow=1, seed=77, spectral=False)
        alone = _counts(ctx, sid, big)[1]
    ctx.reset_stats()
    if batch:
        rid, other = ctx.submit(sid, desc), ctx.submit(sid, big)
        ctx.run_until_idle()
        images = ctx.fetch(rid)[:2]
        ctx.fetch(other)
    else:
        images = ctx.render(sid, desc)[:2]
    st = ctx.stats()
    counts = (st["paths"], st["rays"], st["shadow_rays"])
    return images, tuple(x - y for x, y in zip(counts, alone)) if batch else counts, st


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
    counts = _counts(ctx, a, d)[1]
    # (few paths are staged; in the batch they are not)
    assert _counts(ctx, b, d)[1] == counts
    assert _counts(ctx, b, d, batch=True)[1] == counts
    ctx.close()


@pytest.mark.parametrize("depth", [1, 4, 5])
def test_a_small_plain_render_launches_what_it_needs(tmp_path, depth):
    """A plain render of few paths on a mesh scene: `depth` iterations after
    the camera rays', no kernel for adaptive rounds, none to restore the
    queues' order."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0)
    sid = ctx.load_scene_json(*_boxed(tmp_path, "cornell"))
    st = _counts(ctx, sid, capi.render_desc(64, depth=depth, samples=1, shadow=2, seed=5))[2]
    assert st["iterations"] == 1 + depth
    assert st["stage_launches"]["status"] == st["iterations"], st["stage_launches"]
    ctx.close()


def _slanted(tmp_path, scene, n=100):
    """The scene's file with tiny slanted quads far behind the camera: the
    estimates do not take them, and with many its rays are traced in full by
    the stages."""
    from pcr_b200 import workloads
    sc = workloads.read_scene_json(scene_path(scene))
    sc["primitives"] += [{"type": "plane", "origin": [0, k, 900.0], "u": [1e-3, 1e-3, 0], "v": [0, 1e-3, 1e-3],
                          "material": next(k for k, m in sc["materials"].items() if "emissive" not in m)} for k in range(n)]
    path = tmp_path / f"{scene}-slanted{n}.json"
    path.write_text(json.dumps(sc))
    return str(path), GOLDEN


@pytest.mark.parametrize("scene,kw", [
    ("cornell", dict(depth=1, samples=1, shadow=1, spectral=False)),
    ("cornell", dict(depth=5, samples=4, shadow=3, russian=True)),
    ("cornell-spheres", dict(depth=4, samples=4, shadow=9, spectral=False, mis=True, stratified=True, aa=2)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, hero=3)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, terminate=True)),
    ("closed-cornell-glass", dict(depth=8, samples=2, shadow=8)),
    ("cornell-large-light", dict(depth=3, samples=2, shadow=2, aa=9, adaptive=True)),
])
@pytest.mark.parametrize("size", [(1, 1), (33, 7), (128, 96)])
def test_staged_scenes_give_the_same_images(tmp_path, scene, kw, size):
    """Scenes that the estimates do not take: the same images and counts, with
    the rays traced by the extend and shadow stages and not by the path kernel
    of mesh-free scenes."""
    from pcr_b200 import capi
    d = capi.render_desc(*size, seed=11, **kw)
    for capacity in (1 << 9, 1 << 17):
        ctx = capi.Context(device=0, queue_capacity=capacity)
        a, b = ctx.load_scene_json(scene_path(scene), GOLDEN), ctx.load_scene_json(*_slanted(tmp_path, scene))
        whole, counts, _ = _counts(ctx, a, d)
        staged, staged_counts, st = _counts(ctx, b, d)
        if not kw.get("adaptive"):  # (a converged pixel's last bits may decide its number of rounds)
            assert staged_counts == counts
            assert np.allclose(staged[0], whole[0], rtol=1e-6, atol=1e-7)
        else:
            assert np.allclose(staged[0], whole[0], rtol=1e-4, atol=1e-5)
        assert st["stage_launches"]["extend"] > 0 and st["stage_launches"]["shadow"] > 0, st["stage_launches"]
        assert st["stage_launches"]["other"] == 0, st["stage_launches"]
        ctx.close()


def test_few_exact_tests_stay_in_one_launch(tmp_path):
    """One slanted quad, few shadow rays, few paths: the whole path in one
    launch, plain and batched; more shadow rays are staged.  Same images."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=1 << 14)
    a, b = ctx.load_scene_json(scene_path("cornell"), GOLDEN), ctx.load_scene_json(*_slanted(tmp_path, "cornell", 1))
    for shadow, whole in ((1, True), (4, True), (16, False)):
        d = capi.render_desc(61, 47, depth=5, samples=3, shadow=shadow, seed=41)
        want, counts, _ = _counts(ctx, a, d)
        got, got_counts, st = _counts(ctx, b, d)
        assert got_counts == counts and np.allclose(got[0], want[0], rtol=1e-6, atol=1e-7)
        assert (st["stage_launches"]["other"] > 0) == whole and (st["stage_launches"]["extend"] == 0) == whole
        rid = ctx.submit(b, d)
        ctx.run_until_idle()
        assert np.allclose(ctx.fetch(rid)[0], want[0], rtol=1e-6, atol=1e-7)
    ctx.close()


def test_one_batch_of_all_kinds_of_scenes(tmp_path):
    """Requests on scenes without a mesh, with one, and staged (the last two
    share the queues), in one wavefront: each as if alone."""
    from pcr_b200 import capi
    for capacity in (1 << 12, 1 << 18):
        ctx = capi.Context(device=0, queue_capacity=capacity)
        sids = [ctx.load_scene_json(*x) for x in (
            (scene_path("cornell"), GOLDEN), _boxed(tmp_path / str(capacity), "cornell-glass"),
            _slanted(tmp_path, "cornell-spheres"), (scene_path("cornell-mesh-light"), GOLDEN),
            _boxed(tmp_path / str(capacity), "cornell"), _slanted(tmp_path, "cornell-glass"))]
        descs = [capi.render_desc(w, h, depth=depth, samples=spp, shadow=s, seed=60 + k, spectral=spectral)
                 for k, (w, h, depth, spp, s, spectral) in enumerate([
                     (64, 48, 4, 4, 2, True), (50, 31, 7, 3, 3, True), (71, 40, 3, 5, 1, False),
                     (48, 48, 4, 4, 4, True), (33, 90, 5, 2, 10, True), (40, 40, 6, 6, 2, True)])]
        alone = [ctx.render(s, d)[0] for s, d in zip(sids, descs)]
        ids = [ctx.submit(s, d) for s, d in zip(sids, descs)]
        ctx.run_until_idle()
        for rid, image in zip(ids, alone):
            assert np.allclose(ctx.fetch(rid)[0], image, rtol=1e-6, atol=1e-7)
        ctx.close()


@pytest.mark.parametrize("capacity", [1 << 9, 1 << 17])
@pytest.mark.parametrize("scene,kw", [
    ("cornell", dict(depth=1, samples=1, shadow=1, spectral=False)),
    ("cornell", dict(depth=6, samples=5, shadow=20, hero=1)),
    ("cornell-spheres", dict(depth=4, samples=4, shadow=2, spectral=False, mis=True, russian=True, stratified=True, aa=2)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, hero=2)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, hero=3)),
    ("cornell-glass", dict(depth=8, samples=3, shadow=2, terminate=True)),
    ("closed-cornell-glass", dict(depth=8, samples=2, shadow=8)),
])
@pytest.mark.parametrize("size", [(1, 1), (33, 7), (128, 96)])
def test_waiting_paths_give_the_same_images(tmp_path, capacity, scene, kw, size):
    """Batched, so that the path kernel of mesh scenes follows the paths: they
    are resumed after every vertex, with their weights, hits and pending forks.
    The queue of the small context holds fewer shadow records than its warps
    reserve, so that shadow rays are also walked in place."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=capacity)
    a, b = ctx.load_scene_json(scene_path(scene), GOLDEN), ctx.load_scene_json(*_boxed(tmp_path, scene))
    d = capi.render_desc(*size, seed=11, **kw)
    whole, counts, _ = _counts(ctx, a, d)
    waited, waited_counts, st = _counts(ctx, b, d, batch=True)
    assert waited_counts == counts
    assert st["stage_launches"]["extend"] > 0 and st["stage_launches"]["other"] == 0
    assert np.allclose(waited[0], whole[0], rtol=1e-6, atol=1e-7)
    ctx.close()


def test_a_large_plain_render_waits_too(tmp_path):
    """A plain render of more paths than are staged, in several fills of the
    queue."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=1 << 14)
    a, b = ctx.load_scene_json(scene_path("cornell-glass"), GOLDEN), ctx.load_scene_json(*_boxed(tmp_path, "cornell-glass"))
    d = capi.render_desc(160, 120, depth=6, samples=7, shadow=3, seed=12)
    whole, counts, _ = _counts(ctx, a, d)
    waited, waited_counts, _ = _counts(ctx, b, d)
    assert waited_counts == counts and counts[0] > 1 << 16
    assert np.allclose(waited[0], whole[0], rtol=1e-6, atol=1e-7)
    ctx.close()


def test_many_shadow_samples_grow_the_queue_of_a_mesh_scene(tmp_path):
    """More than 8 shadow samples per hit on a scene whose shadow rays become
    records: the queue grows, plain, batched and between the two."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=1 << 12)
    a, b = ctx.load_scene_json(scene_path("cornell"), GOLDEN), ctx.load_scene_json(*_boxed(tmp_path, "cornell"))
    before = ctx.stats()["device_bytes"]
    for shadow, w in ((40, 48), (64, 300), (3, 48)):
        d = capi.render_desc(w, 48, depth=3, samples=8, shadow=shadow, seed=91)
        want = ctx.render(a, d)[0]
        rid = ctx.submit(b, d)
        ctx.run_until_idle()
        assert np.allclose(ctx.fetch(rid)[0], want, rtol=1e-6, atol=1e-7)
        assert np.allclose(ctx.render(b, d)[0], want, rtol=1e-6, atol=1e-7)
    assert ctx.stats()["device_bytes"] >= before
    with pytest.raises(capi.PcrError):
        ctx.render(b, capi.render_desc(16, samples=1, shadow=65))
    ctx.close()


def test_few_paths_are_staged_in_a_batch_too(tmp_path):
    """One small request on a mesh scene: the staged form, as in a plain
    render, and the same image beside requests that are not."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=1 << 14)
    a, b = ctx.load_scene_json(scene_path("cornell-glass"), GOLDEN), ctx.load_scene_json(*_boxed(tmp_path, "cornell-glass"))
    d = capi.render_desc(61, 47, depth=7, samples=3, shadow=5, seed=31)
    want = ctx.render(a, d)[0]
    for n in (1, 3):
        ids = [ctx.submit(b, d) for _ in range(n)]
        ctx.run_until_idle()
        for i in ids:
            assert np.allclose(ctx.fetch(i)[0], want, rtol=1e-6, atol=1e-7)
    # staged ones first, others join them while they run
    ctx.serve_start()
    ids = [ctx.submit(b, d)]
    ids += [ctx.submit(b, capi.render_desc(300, 200, depth=4, samples=4, shadow=3, seed=k)) for k in range(3)]
    ids += [ctx.submit(a, d), ctx.submit(b, d)]
    for i in ids:
        ctx.wait(i, 30000)
    for i in (ids[0], ids[4], ids[5]):
        assert np.allclose(ctx.fetch(i)[0], want, rtol=1e-6, atol=1e-7)
    ctx.serve_stop()
    ctx.close()
