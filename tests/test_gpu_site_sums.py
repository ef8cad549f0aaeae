"""Observables and energies of a state against the oracle at the sizes where the column-wise site
sums can go wrong: one column, one row, columns short of and past a block's 512 (256 above 16
sites), row chunks with a remainder, every site-count template, complex vectors. The sums are
of at most 10^6 positive terms: 1e-12 relative; ekin is a difference of sums of order U N."""
import numpy as np
import pytest

import ed_lattice_b200 as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [(8, 1, 0, 4), (8, 1, 4, 0), (8, 1, 1, 7), (3, 3, 4, 5), (11, 1, 5, 6), (3, 4, 6, 3), (7, 2, 4, 6), (5, 3, 7, 2),
         (4, 4, 5, 2), (17, 1, 3, 2), (9, 2, 2, 4), (11, 2, 1, 4)]


@pytest.mark.parametrize("flux", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%d_%d_%d" % c)
def test_site_sums(case, flux):
    lx, ly, nup, ndw = case
    h = E.square_lattice(lx, ly)
    h[np.diag_indices(lx * ly)] = np.round(np.random.default_rng(1).uniform(-1, 1, lx * ly) * 64) / 64
    if flux:
        h = h.astype(complex)
        h[0, 1], h[1, 0] = 1j, -1j
    for hf in (False, True):
        om = O.Model(h, uloc=4.0, xmu=1.0, hfmode=hf)
        s = E.Sector(E.Model(h, uloc=4.0, xmu=1.0, hfmode=hf), nup, ndw)
        v = O.random_vector(3, s.dim) + (1j * O.random_vector(4, s.dim) if flux else 0.0)
        v /= np.linalg.norm(v)
        s.set_state(v)
        got = s.observables(0.5)
        # |psi|^2 per configuration: densities and double occupancies by the definition
        mu, md = s.maps()
        ns = lx * ly
        bu = ((mu[:, None] >> np.arange(ns)) & 1).astype(float)
        bd = ((md[:, None] >> np.arange(ns)) & 1).astype(float)
        p = (np.abs(v) ** 2).reshape(s.dimdw, s.dimup)
        up, dw, dd = p.sum(0) @ bu, p.sum(1) @ bd, (bd * (p @ bu)).sum(0)
        for key, ref in (("dens_up", up), ("dens_dw", dw), ("dens", up + dw), ("docc", dd), ("magz", up - dw)):
            assert np.allclose(got[key], 0.5 * ref, rtol=0, atol=1e-12), key
        e = s.energy(2.0)
        hv = O.Stored(om, nup, ndw).matvec_z(v) if flux else O.Stored(om, nup, ndw).matvec_d(v)
        eps = np.real(np.diag(h)) - 1.0 - (2.0 if hf else 0.0)
        ekin = np.vdot(v, hv).real - eps @ (up + dw) - 4.0 * dd.sum()
        ehar = -2.0 * (up + dw).sum() if hf else 0.0
        for key, ref in (("ekin", ekin), ("epot", 4.0 * dd.sum() + ehar), ("eknot", np.real(np.diag(h)) @ (up + dw)),
                         ("ehartree", ehar)):
            assert abs(e[key] - 2.0 * ref) <= 1e-11, (key, e[key], 2.0 * ref)
        s.delete()
