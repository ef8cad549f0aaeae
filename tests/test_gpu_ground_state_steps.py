"""Ground-state Lanczos steps queued ahead of the host's convergence test: chains that end at a
step limit on either side of the shortest one that is estimated (16 steps), a start vector that
spans an invariant subspace (a vanishing b with a step already queued), and runs in several
threads. Against the dense spectrum to the 1e-10 of the convergence contract; a chain cut at a
limit against the eigenvalue of its own tridiagonal, whose coefficients it shares, to 1e-12."""
import threading

import numpy as np
import pytest

import ed_lattice_b200 as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _sector(lx, ly, nup, ndw):
    h = E.square_lattice(lx, ly)
    h[np.diag_indices(lx * ly)] = np.random.default_rng(2).uniform(-1, 1, lx * ly)
    kw = dict(uloc=4.0, xmu=1.0, hfmode=False)
    return E.Sector(E.Model(h, **kw), nup, ndw), O.dense_h(O.Model(h, **kw), nup, ndw)


@pytest.mark.parametrize("mode", [E.EDG_GS_F64, E.EDG_GS_F32_REFINE], ids=["f64", "refine"])
@pytest.mark.parametrize("case", [(2, 1, 1, 1), (4, 1, 2, 1), (3, 2, 3, 3), (8, 1, 2, 2)], ids=lambda c: "%dx%d_%d_%d" % c)
def test_limits_and_exhaustion(case, mode):
    s, H = _sector(*case)
    w, V = np.linalg.eigh(H)
    v0 = O.random_vector(3, s.dim)
    e0, _, n = E.sp_lanc_eigh(s, v0=v0, maxit=300, tol=1e-12, mode=mode)
    assert abs(e0 - w[0]) <= 1e-10 * abs(w[0])
    for k in (1, 2, 15, 16, 17, 18):
        if mode != E.EDG_GS_F64 or k > s.dim // 2:
            continue
        a, b, _, _ = E.tridiag_Hv_sector(s, v0, k)
        wk = np.linalg.eigvalsh(np.diag(a) + np.diag(b[1:k], 1) + np.diag(b[1:k], -1))
        ek, _, nk = E.sp_lanc_eigh(s, v0=v0, maxit=k, tol=1e-15, mode=mode, want_vector=False)
        assert nk == k and abs(ek - wk[0]) <= 1e-12 * abs(wk[0])
    # two eigenvectors: the Krylov space has two dimensions
    x = V[:, 0] + 0.5 * V[:, -1]
    ex, vx, _ = E.sp_lanc_eigh(s, v0=x, maxit=300, tol=1e-12, mode=mode)
    assert abs(ex - w[0]) <= 1e-10 * abs(w[0])
    assert abs(np.linalg.norm(vx) - 1.0) <= 1e-10


def test_runs_in_threads():
    secs = [_sector(8, 1, 2, 2)[0], _sector(3, 2, 3, 3)[0], _sector(8, 1, 2, 2)[0], _sector(3, 2, 3, 2)[0]]
    run = lambda s: E.sp_lanc_eigh(s, seed=7, maxit=200, tol=1e-12, want_vector=False)  # noqa: E731
    alone = [run(s) for s in secs]
    got = [None] * len(secs)

    def work(i):
        for _ in range(5):
            got[i] = run(secs[i])

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(secs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert got == alone
