"""Rounding of a pole sum, up to 64 poles with a division per term and beyond with shared ones: no
larger than with a division per term, one after the other. Both are compared with 64-bit-mantissa sums over many frequencies; the division per term is restated
here, its fused multiply-adds rounded once from the wider type."""
import numpy as np
import pytest

from ed_lattice_b200 import _edgpu_lib as L
from ed_lattice_b200.edlat import eval_poles

pytestmark = pytest.mark.gpu

W = np.longdouble


def _division_per_term(p, w, z):
    x, y = z.real, z.imag
    re, im = np.zeros(z.size), np.zeros(z.size)
    for pk, wk in zip(p, w):
        d = x - pk
        a = (W(d) * d + y * y).astype(float)
        s = wk / a
        re = (W(s) * d + re).astype(float)
        im = (im - W(s) * y).astype(float)
    return re, im


@pytest.mark.parametrize("npoles", [8, 16, 64, 65, 150, 1200])
def test_rounding_of_shared_divisions(npoles):
    r = np.random.default_rng(npoles)
    z = r.uniform(-10, 10, 20000) + 1j * r.choice([0.02, 0.15, 1.0, 6.0], 20000)
    p, w = r.uniform(-9, 9, npoles), r.exponential(1.0, npoles) / npoles
    d = W(z.real)[:, None] - p
    a = d * d + (W(z.imag) ** 2)[:, None]
    ref = (w * d / a).sum(1), -(w * W(z.imag)[:, None] / a).sum(1)
    size = (w * np.hypot(d, W(z.imag)[:, None]) / a).sum(1)
    g = eval_poles(p, w, z)
    rms = lambda v: float(np.sqrt(np.mean((sum((np.abs(c - q) / size) ** 2 for c, q in zip(v, ref))))))  # noqa: E731
    # 20,000 frequencies: the two rms values are known to about 1 %
    assert rms((g.real, g.imag)) <= 1.03 * rms(_division_per_term(p, w, z))


@pytest.mark.parametrize("npoles", [37, 77])
def test_large_and_infinite_weights(npoles):
    """Weights near the end of the range; an infinite one stays an infinity of its sign."""
    r = np.random.default_rng(1)
    p, w, z = r.uniform(-9, 9, npoles), r.uniform(0.5, 1.0, npoles), r.uniform(-10, 10, 50) + 0.1j
    for scale in (1e250, 1e300):
        ref = (w / (z[:, None] - p)).sum(1)
        size = (w / np.abs(z[:, None] - p)).sum(1)
        assert np.all(np.abs(eval_poles(p, w * scale, z) / scale - ref) <= 1e-14 * size)
    w[5] = np.inf
    zr, zi, re, im = z.real.copy(), z.imag.copy(), np.zeros(z.size), np.zeros(z.size)  # (re + 1j * im: inf * 0)
    q = lambda v: v.ctypes.data_as(L._pd)  # noqa: E731
    L.check(L.lib().edg_eval_poles(p.size, q(p), q(w), z.size, q(zr), q(zi), q(re), q(im)), "poles")
    assert np.array_equal(re, np.sign(zr - p[5]) * np.inf) and np.all(im == -np.inf)
