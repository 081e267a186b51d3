"""The spectra as renders evaluate them: divisions by 150 and 5 from a rounded
reciprocal and one correction.  Every float32 wavelength of 400..700 nm, bit
for bit against the same operations in NumPy's IEEE float32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from pcr_b200 import capi
    c = capi.Context(device=0, queue_capacity=1 << 10)
    yield c
    c.close()


def _visible():
    lo, hi = np.array([400.0, 700.0], np.float32).view(np.uint32)
    lam = np.arange(lo, hi + 1, dtype=np.uint32).view(np.float32)
    return np.concatenate([lam, np.array([0.0, 399.99997, 700.00006, 1000.0], np.float32)])


@pytest.mark.parametrize("fit", [(1.5, -2.0, 0.75, 1.0), (-6.0, 30.0, -11.0, 2.5), (0.0, 0.0, 0.0, 0.3)])
def test_sigmoid_at_every_visible_wavelength(ctx, fit):
    lam = _visible()
    c0, c1, c2, scale = (np.float32(x) for x in fit)
    L = (lam - np.float32(550)) / np.float32(150)
    p = c0 + L * (c1 + L * c2)
    want = (np.float32(0.5) + p / (np.float32(2) * np.sqrt(np.float32(1) + p * p))) * scale
    got = ctx.eval_stage(0, lam, np.array(fit, np.float32))[:, 0]
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def test_table_at_every_visible_wavelength(ctx):
    lam = _visible()
    table = np.random.default_rng(3).uniform(0, 1, 61).astype(np.float32)
    t = (lam - np.float32(400)) / np.float32(5)
    i = np.clip(t.astype(np.int32), 0, 59)
    f = t - i.astype(np.float32)
    want = table[i] * (np.float32(1) - f) + table[i + 1] * f
    want[lam == 700] = table[60]
    want[(lam < 400) | (lam > 700)] = 0
    got = ctx.eval_stage(1, lam, table)[:, 0]
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
