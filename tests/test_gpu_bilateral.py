"""The bilateral filter's tabulated weights against the filter computed in
numpy with the same float operations, on images that reach both ends of the
table: flat areas (colour distance 0), hard black / white and colour edges
(distances past the last entry, weight zero), and sizes below the window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bilateral(src):
    f = np.float32
    inv_s, inv_c = f(1) / (f(2) * f(1.5) * f(1.5)), f(1) / (f(2) * f(10) * f(10))
    h, w, _ = src.shape
    sums = np.zeros((h, w, 4), f)
    c = src.astype(np.int64)
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
            if y0 >= y1 or x0 >= x1:
                continue
            n = c[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
            d2 = ((n - c[y0:y1, x0:x1]) ** 2).sum(-1)
            e = f(dx * dx + dy * dy) * inv_s + d2.astype(f) * inv_c
            wt = np.exp(-e.astype(np.float64)).astype(f)
            sums[y0:y1, x0:x1, 0] += wt
            for k in range(3):
                sums[y0:y1, x0:x1, 1 + k] += wt * n[..., k].astype(f)
    return np.minimum(f(255), sums[..., 1:] / sums[..., :1] + f(0.5)).astype(np.uint8)


@pytest.mark.parametrize("w,h", [(1, 1), (2, 3), (5, 4), (130, 67)])
@pytest.mark.parametrize("kind", ["flat", "edges", "noise"])
def test_tabulated_weights_match_filter(w, h, kind):
    from pcr_b200 import capi
    rng = np.random.default_rng(w * 7 + h)
    if kind == "flat":
        hdr = np.full((h, w, 3), 0.5, np.float32)
    elif kind == "edges":   # tone-mapped bytes 0 and about 255, per channel
        hdr = np.where(rng.uniform(size=(h, w, 3)) < 0.5, 0.0, 1000.0).astype(np.float32)
    else:
        hdr = rng.gamma(2.0, 0.4, (h, w, 3)).astype(np.float32)
    ctx = capi.Context(device=0, queue_capacity=1 << 17)
    try:
        want = _bilateral(_bilateral(ctx.tonemap(hdr)))
        got = ctx.tonemap(hdr, denoise=True)
    finally:
        ctx.close()
    # numpy's and CUDA's double exponentials may differ in the last bit
    diff = np.abs(got.astype(int) - want.astype(int))
    assert diff.max() <= 1 and (diff > 0).mean() <= 1e-3
