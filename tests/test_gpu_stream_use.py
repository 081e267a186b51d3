"""A caller's own use of the context's stream while the engine serves.

The launch graphs are captured when a combination of scene kinds first runs,
at any time of serving.  Meanwhile other threads may query, wait on or record
events on the stream (pcr_ctx_stream is there for that): neither side may fail.
"""
import threading

import numpy as np
import pytest

from conftest import GOLDEN, scene_path
from test_gpu_queues import _boxed, _slanted

pytestmark = pytest.mark.gpu


def test_stream_queries_and_events_while_graphs_are_captured(tmp_path):
    import torch

    from pcr_b200 import capi
    desc = capi.render_desc(48, depth=3, samples=2, shadow=2, seed=8)
    for turn in range(3):
        ctx = capi.Context(device=0, queue_capacity=1 << 12)
        sids = [ctx.load_scene_json(*x) for x in ((scene_path("cornell"), GOLDEN),
                                                  _boxed(tmp_path / str(turn), "cornell"), _slanted(tmp_path, "cornell"))]
        want = ctx.render(sids[0], desc)[0]
        stream = torch.cuda.ExternalStream(ctx.stream(), device="cuda:0")
        stop, errors = threading.Event(), []

        def use():
            try:
                while not stop.is_set():
                    stream.query()
                    e = torch.cuda.Event()
                    e.record(stream)
                    e.query()
            except Exception as x:  # noqa: BLE001
                errors.append(x)

        threads = [threading.Thread(target=use) for _ in range(3)]
        for th in threads:
            th.start()
        ctx.serve_start()
        try:
            for group in ([0], [1], [2], [0, 1], [1, 2], [0, 2], [0, 1, 2]):
                ids = [ctx.submit(sids[k], desc) for k in group]
                for i in ids:
                    ctx.wait(i, 20000)
                    assert np.allclose(ctx.fetch(i)[0], want, rtol=1e-6, atol=1e-7)
        finally:
            stop.set()
            for th in threads:
                th.join()
            ctx.serve_stop()
        assert not errors, errors[:1]
        ctx.close()
