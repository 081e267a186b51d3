"""pcr_render_noalloc on scenes with a mesh (named to run last, as
test_zz_no_alloc.py): its queues in the fixed scratch, path forks, and shadow
records past the scratch's queue, against pcr_render."""
import numpy as np
import pytest

from conftest import GOLDEN, scene_path
from test_gpu_queues import _boxed

pytestmark = pytest.mark.gpu


def _render_both(ctx, sid, desc):
    import torch
    w, h = desc.width, desc.height
    hdr = torch.full((h, w, 3), float("nan"), dtype=torch.float32, device="cuda:0")
    rgb = torch.zeros(h, w, 3, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx.render_noalloc(sid, desc, hdr.data_ptr(), rgb.data_ptr())
    torch.cuda.synchronize()
    freed = torch.cuda.mem_get_info()[0] - free
    ref_hdr, ref_rgb, _ = ctx.render(sid, desc)
    assert np.allclose(hdr.cpu().numpy(), ref_hdr, rtol=1e-6, atol=1e-7)
    assert np.abs(rgb.cpu().numpy().astype(int) - ref_rgb.astype(int)).max() <= 1
    return freed


# 256x256 with 8 shadow rays: the vertices of an iteration want more records
# than the scratch holds, and wait; in glass, forks fill the path queue
@pytest.mark.parametrize("scene", ["cornell-bunny", "cornell-mesh-light", "cornell", "cornell-glass"])
def test_noalloc_on_mesh_scenes(tmp_path, scene):
    from pcr_b200 import capi
    ctx = capi.Context(device=0)
    where = (scene_path(scene), GOLDEN) if "mesh" in scene or "bunny" in scene else _boxed(tmp_path, scene)
    sid = ctx.load_scene_json(*where)
    small = capi.render_desc(40, 31, depth=5, samples=3, shadow=3, seed=5)
    big = capi.render_desc(256, depth=6, samples=6, shadow=8, seed=6, mis=True, russian=True)
    _render_both(ctx, sid, small)  # (loads the kernels)
    _render_both(ctx, sid, big)
    assert _render_both(ctx, sid, small) == 0, "the call changed the device's free memory"
    _render_both(ctx, sid, capi.render_desc(200, 180, depth=4, samples=2, shadow=8, spectral=False, seed=7))
    ctx.close()
