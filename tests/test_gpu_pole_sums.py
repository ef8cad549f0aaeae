"""Pole sums against numpy at the sizes where the eight-pole groups and the chunks can go wrong,
and where a group's shared division does not apply: denominators far apart, very large and very
small, a frequency on a pole. Each term carries a few roundings of 1.1e-16 and the terms of one
sum are added in chunks: 1e-14 of the sum of magnitudes."""
import numpy as np
import pytest

from ed_lattice_b200.edlat import eval_poles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npoles", [1, 2, 7, 8, 9, 15, 16, 17, 63, 1023, 4099, 70001])
@pytest.mark.parametrize("nz", [1, 255, 257, 513])
def test_pole_sums(npoles, nz):
    r = np.random.default_rng(npoles * 1000 + nz)
    p, w = r.uniform(-9, 9, npoles), r.normal(size=npoles)
    z = r.uniform(-10, 10, nz) + 1j * r.choice([0.05, 1.0, -3.0], nz)
    d = z[:, None] - p[None, :] if npoles * nz < 2e7 else None
    if d is None:
        ref = np.array([(w / (x - p)).sum() for x in z])
        size = np.array([np.abs(w / (x - p)).sum() for x in z])
    else:
        ref, size = (w / d).sum(1), np.abs(w / d).sum(1)
    assert np.all(np.abs(eval_poles(p, w, z) - ref) <= 1e-14 * size)


@pytest.mark.parametrize("scale", [1e-100, 1e-40, 1e40, 1e100, 1e150])
def test_pole_sums_scaled(scale):
    r = np.random.default_rng(5)
    p, w = r.uniform(1, 9, 37) * scale, r.normal(size=37)
    p[::5] /= scale  # groups of very different denominators
    z = (r.uniform(-10, -1, 19) + 1j) * scale
    ref, size = (w / (z[:, None] - p)).sum(1), np.abs(w / (z[:, None] - p)).sum(1)
    assert np.all(np.abs(eval_poles(p, w, z) - ref) <= 1e-14 * size)


def test_frequency_on_a_pole():
    """1/0 stays with its own frequency."""
    p, w = np.arange(8.0), np.ones(8)
    g = eval_poles(p, w, np.array([3.0 + 0j, 3.5 + 0j]))
    assert not np.isfinite(g[0]) and abs(g[1].real - (1 / (3.5 - p)).sum()) < 1e-13
