"""Results into any memory a caller may name: ordinary and pinned host arrays,
and device memory (a GPU program's own buffers)."""
import ctypes as C

import numpy as np
import pytest

from conftest import GOLDEN, scene_path

pytestmark = pytest.mark.gpu


def test_results_in_pageable_pinned_and_device_memory():
    import torch

    from pcr_b200 import capi
    ctx = capi.Context(device=0, queue_capacity=1 << 12)
    sid = ctx.load_scene_json(scene_path("cornell"), GOLDEN)
    L, n, w, h = ctx.L, 5003, 37, 23
    rng = np.random.default_rng(1)
    rays = np.concatenate([rng.uniform(-1, 1, (n, 3)) - [0, 0, 3], rng.normal(size=(n, 3))], 1).astype(np.float32)
    rays[:, 3:] /= np.linalg.norm(rays[:, 3:], axis=1, keepdims=True)
    dist2 = rng.uniform(0.1, 9, n).astype(np.float32)
    image = rng.gamma(2.0, 0.5, (h, w, 3)).astype(np.float32)
    desc = capi.render_desc(w, h, depth=3, samples=2, shadow=2, seed=4)
    mat, prim, t = ctx.trace_closest(sid, rays)
    want = {"mat": mat, "prim": prim, "t": t, "shadow": ctx.trace_shadow(sid, rays, dist2), "tone": ctx.tonemap(image)}
    want["hdr"], want["rgb"], _ = ctx.render(sid, desc)
    r, d2 = capi._fp(rays), capi._fp(dist2)

    def ptr(x, ctype):
        return C.cast(x.data_ptr(), C.POINTER(ctype))

    # one kind of memory for all results of a call, and a mixture
    for place in (("pageable",) * 3, ("pinned",) * 3, ("device",) * 3, ("device", "pageable", "device"),
                  ("pageable", "device", "pinned")):
        def buf(i, shape, dtype):
            x = torch.zeros(shape, dtype=dtype, device="cuda:0" if place[i] == "device" else "cpu")
            return x.pin_memory() if place[i] == "pinned" else x
        m, p, tt = buf(0, n, torch.int32), buf(1, n, torch.int32), buf(2, n, torch.float32)
        assert L.pcr_trace_closest(ctx.h, sid, r, n, ptr(m, C.c_int32), ptr(p, C.c_int32), ptr(tt, C.c_float)) == 0
        got = {"mat": m, "prim": p, "t": tt}
        got["shadow"] = buf(0, n, torch.int32)
        assert L.pcr_trace_shadow(ctx.h, sid, r, d2, n, ptr(got["shadow"], C.c_int32)) == 0
        got["tone"] = buf(1, (h, w, 3), torch.uint8)
        assert L.pcr_tonemap(ctx.h, capi._fp(image), w, h, 0, 0, ptr(got["tone"], C.c_uint8)) == 0
        got["hdr"], got["rgb"] = buf(0, (h, w, 3), torch.float32), buf(1, (h, w, 3), torch.uint8)
        assert L.pcr_render(ctx.h, sid, C.byref(desc), ptr(got["hdr"], C.c_float), ptr(got["rgb"], C.c_uint8), None) == 0
        torch.cuda.synchronize()
        for k, x in got.items():
            x = x.cpu().numpy()
            if k == "hdr":
                assert np.allclose(x, want[k], rtol=1e-6, atol=1e-7), (k, place)
            elif k == "rgb":
                assert np.abs(x.astype(int) - want[k].astype(int)).max() <= 1, (k, place)
            else:
                assert np.array_equal(x, np.asarray(want[k]).reshape(x.shape)), (k, place)
    ctx.close()
