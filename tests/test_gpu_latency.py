"""What a deep render lets others wait for.

A mesh-free path is followed to its end in the iteration it starts in, so an
iteration's work has to be bounded by the vertices its paths may have and not by
their number alone: a cancel, a newly admitted request and a finished result
are only seen between blocks of iterations.
"""
import time

import pytest

from conftest import GOLDEN, scene_path

pytestmark = pytest.mark.gpu

DEEP = dict(depth=64, shadow=16)
VERTICES_PER_SLOT = 64
WAVE = 2 * 148 * 4 * 128


@pytest.mark.parametrize("scene", ["closed-cornell-spec", "closed-cornell-glass"])
def test_an_iteration_of_deep_paths_is_bounded(scene):
    from pcr_b200 import capi
    fill = 1 << 20
    ctx = capi.Context(device=0, queue_capacity=fill)
    sid = ctx.load_scene_json(scene_path(scene), GOLDEN)
    depth, paths = 255, 2 * 256 * 256 * 160
    most = max(VERTICES_PER_SLOT * fill, WAVE * depth) // depth  # new paths of an iteration
    ids = [ctx.submit(sid, capi.render_desc(256, samples=160, depth=depth, shadow=1, seed=3 + k)) for k in range(2)]
    ctx.reset_stats()
    ctx.run_until_idle()
    st = ctx.stats()
    assert st["paths"] == paths
    assert st["iterations"] >= paths // most, (st["iterations"], most)
    for i in ids:
        ctx.fetch(i)
    # shallow paths are not cut: a block of iterations or two is enough
    rid = ctx.submit(sid, capi.render_desc(256, samples=32, depth=6, shadow=4, seed=9))
    ctx.reset_stats()
    ctx.run_until_idle()
    assert ctx.stats()["iterations"] <= 32
    ctx.fetch(rid)
    ctx.close()


def test_cancel_and_small_requests_beside_a_deep_render():
    """A small request is done, and a cancel ends the deep one, long before
    the seconds that blocks of whole deep paths took."""
    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=1 << 20)
    sid = ctx.load_scene_json(scene_path("closed-cornell-spec"), GOLDEN)
    ctx.serve_start()
    try:
        deep = ctx.submit(sid, capi.render_desc(1024, samples=4096, seed=1, **DEEP))
        time.sleep(0.3)
        start = time.perf_counter()
        small = ctx.submit(sid, capi.render_desc(32, depth=2, samples=1, shadow=1))
        ctx.wait(small, 30000)
        ctx.fetch(small)
        beside = time.perf_counter() - start
        time.sleep(0.3)
        start = time.perf_counter()
        ctx.cancel(deep)
        with pytest.raises(capi.PcrError) as e:
            ctx.wait(deep, 30000)
        assert e.value.status == 7
        cancelled = time.perf_counter() - start
        assert beside < 0.6 and cancelled < 0.6, (beside, cancelled)
    finally:
        ctx.serve_stop()
        ctx.close()
