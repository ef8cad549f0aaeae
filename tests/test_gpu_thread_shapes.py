"""Sectors of different sizes worked on in several host threads at once: a kernel that wants more
than 48 KB of shared memory for its rows or coefficients takes a different amount of it in each
thread. Every thread gets what it gets alone, bit for bit."""
import threading

import numpy as np
import pytest

import ed_lattice_b200 as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sector(lx, ly, nup, ndw, cplx=False):
    h = E.square_lattice(lx, ly)
    h[np.diag_indices(lx * ly)] = np.random.default_rng(4).uniform(-1, 1, lx * ly)
    if cplx:
        h = h.astype(complex)
        h[0, 1], h[1, 0] = 1j, -1j
    return E.Sector(E.Model(h, uloc=4.0, xmu=1.0, hfmode=False), nup, ndw)


def _in_threads(jobs, rounds):
    alone = [f() for f in jobs]
    errors, start = [], threading.Barrier(len(jobs))

    def work(i):
        try:
            start.wait()
            for _ in range(rounds):
                got = jobs[i]()
                assert all(np.array_equal(g, a) for g, a in zip(got, alone[i]))
        except Exception as e:  # noqa: BLE001
            errors.append((i, e))

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors


def test_row_lengths():
    """Tiles of 48 and 55 KB (DimUp 3003 and 3432), chains of launches without host work between."""
    jobs = []
    for nup, ndw in ((6, 2), (7, 2), (6, 3), (7, 3)):
        s = _sector(7, 2, nup, ndw)
        v = O.random_vector(3 + nup, s.dim)
        jobs.append(lambda s=s, v=v: E.tridiag_Hv_sector(s, v, 60)[:2])
    _in_threads(jobs, 12)


def test_many_levels():
    """Sixteen levels of sectors of 400 to 560 states, from the whole Krylov basis (a tolerance that
    nothing meets): 51 to 72 KB of Ritz coefficients."""
    jobs = []
    for lx, ly, nup, ndw, cplx in ((6, 1, 3, 3, False), (8, 1, 1, 4, False), (8, 1, 1, 3, True), (5, 2, 1, 2, False)):
        s = _sector(lx, ly, nup, ndw, cplx)
        jobs.append(lambda s=s: s.lowest_k(16, seed=5, maxit=1024, tol=1e-300)[:2])
    _in_threads(jobs, 12)
