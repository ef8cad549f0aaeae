"""The row-tile H x v (16-byte slots, 16-bit schedule) against the oracle where it can go wrong:
one column, one row, columns and rows that do not fill a slice or a tile, odd DimUp, tiles of
two and of one CTA per SM, column parts, one hopping value (sign bits) and several (palette).
Hopping values are powers of two, so every product is exact and the FP64 result carries the
bits of the oracle's sums in the same order. FP32: the bound of the other H x v tests, 2e-6 of
the largest element (about 20 terms of 6e-8 each). Chains: FP64 coefficients to 1e-9 over 20
steps, as in the other Lanczos tests."""
import ctypes as C

import numpy as np
import pytest

import ed_lattice_b200 as E
from ed_lattice_b200 import _edgpu_lib as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lattice(lx, ly, tp=0.0):
    h = E.square_lattice(lx, ly)
    if tp:
        for y in range(ly):
            for x in range(lx):
                for dx in (1, -1):
                    i, j = x + lx * y, (x + dx) % lx + lx * ((y + 1) % ly)
                    if i != j and h[i, j] == 0.0:
                        h[i, j] = h[j, i] = -tp
    return h


# lx, ly, nup, ndw, tp
CASES = [
    (8, 1, 0, 4, 0.0),    # one column
    (8, 1, 4, 0, 0.0),    # one row
    (8, 1, 1, 7, 0.0),    # 8 columns, 8 rows
    (3, 3, 4, 5, 0.0),    # 126 x 126: part slices, even rows
    (11, 1, 5, 4, 0.0),   # 462 x 330: single pass by tiles in FP64
    (11, 1, 5, 5, 0.0),   # 462 x 462: and in FP32
    (13, 1, 3, 3, 0.125),  # 286 x 286: nine slices, fewer than the resident warps
    (3, 4, 1, 6, 0.0),    # 12 x 924: a third of a slice, many tiles
    (3, 4, 6, 1, 0.0),    # 924 x 12: few tiles, column parts
    (3, 4, 5, 6, 0.25),   # 792 x 924, two hopping values
    (7, 2, 7, 3, 0.0),    # 3432 columns: over 48 KB, four CTAs per SM or two
    (13, 1, 6, 3, 0.0),   # 1716 x 286
    (5, 3, 7, 2, 0.0),    # 6435 columns (odd): two CTAs per SM
    (5, 3, 7, 2, 0.125),  # the same with a palette
    (4, 4, 8, 2, 0.0),    # 12870 columns: one CTA per SM
    (4, 4, 8, 1, 0.25),   # the same with a palette, 16 rows
]


@pytest.mark.parametrize("case", CASES, ids=["%dx%d_%d_%d_%g" % c for c in CASES])
def test_hxv_tile_vs_oracle(case):
    import torch
    lx, ly, nup, ndw, tp = case
    h = lattice(lx, ly, tp)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    st = O.Stored(O.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw)
    v = O.random_vector(3, s.dim)
    ref = st.matvec_d(v)
    scale = np.abs(ref).max()
    x64 = torch.from_numpy(v).cuda()
    for x, prec, fn, cands in ((x64, E.EDG_PREC_F64, L.lib().edg_hxv_dev_f64, (0, 3)),
                               (x64.float(), E.EDG_PREC_F32, L.lib().edg_hxv_dev_f32, (0, 12))):
        for cand in cands:
            s.set_kernels(cand, prec)
            y = torch.full_like(x, float("nan"))
            L.check(fn(s.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), "hxv")
            y = y.cpu().numpy()
            if prec == E.EDG_PREC_F64:
                assert np.array_equal(y, ref), (cand, np.abs(y - ref).max())
            else:
                assert np.abs(y - ref).max() <= 2e-6 * scale, (cand, np.abs(y - ref).max() / scale)
    n = min(20, s.dim)
    ao, bo, _, no = st.tridiag(v, n)
    for cand in (0, 3):
        s.set_kernels(cand, E.EDG_PREC_F64)
        a, b, _, m = E.tridiag_Hv_sector(s, v, n)
        m = min(m, no) - (1 if min(m, no) < n else 0)  # up to the step where the Krylov space ends
        assert np.allclose(a[:m], ao[:m], rtol=1e-9, atol=1e-9) and np.allclose(b[:m], bo[:m], rtol=1e-9, atol=1e-9)
    s.delete()


@pytest.mark.parametrize("case", CASES + [(4, 4, 5, 4, 0.0)], ids=lambda c: "%dx%d_%d_%d_%g" % c)
def test_hxv_tile_direct(case):
    """The direct form's order (diag, UP, DW), whole (up to 12,000,000 FP64 and 4,000,000 FP32
    states) and, last case in FP32, as two passes."""
    import torch
    lx, ly, nup, ndw, tp = case
    h = lattice(lx, ly, tp)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw, E.EDG_FORM_DIRECT)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    v = O.random_vector(3, s.dim)
    ref = O.direct_matvec_d(O.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw, v)
    x = torch.from_numpy(v).cuda()
    y = torch.full_like(x, float("nan"))
    L.check(L.lib().edg_hxv_dev_f64(s.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), "hxv")
    assert np.array_equal(y.cpu().numpy(), ref)
    x = x.float()
    y = torch.full_like(x, float("nan"))
    L.check(L.lib().edg_hxv_dev_f32(s.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), "hxv")
    assert np.abs(y.cpu().numpy() - ref).max() <= 2e-6 * np.abs(ref).max()
    s.delete()


def test_infinities_stay_where_they_belong():
    """An infinite element of v reaches only the rows that H connects to it: idle slots and the
    repeated reads of short hop lists add nothing."""
    import torch
    h = lattice(11, 1)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), 5, 5)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    v = O.random_vector(5, s.dim)
    v[s.dim // 2] = np.inf
    ref = O.Stored(O.Model(h, uloc=4.0, xmu=2.0, hfmode=False), 5, 5).matvec_d(v)
    x = torch.from_numpy(v).cuda()
    for cand in (0, 3):
        s.set_kernels(cand, E.EDG_PREC_F64)
        y = torch.empty_like(x)
        L.check(L.lib().edg_hxv_dev_f64(s.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), "hxv")
        assert np.array_equal(y.cpu().numpy(), ref)
    s.delete()


def flux_lattice(lx, ly, flux):
    """Nearest-neighbour hopping with a phase per x bond: several complex values, both signs."""
    h = E.square_lattice(lx, ly).astype(complex)
    for y in range(ly):
        for x in range(lx):
            i, j = x + lx * y, (x + 1) % lx + lx * y
            if i != j:
                h[i, j] = -np.exp(2j * np.pi * flux * (y + 1))
                h[j, i] = np.conj(h[i, j])
    return h


@pytest.mark.parametrize("case", [(8, 1, 0, 4), (8, 1, 4, 0), (3, 3, 4, 5), (11, 1, 5, 4), (3, 4, 6, 5), (7, 2, 7, 3),
                                  (5, 3, 7, 2), (4, 4, 8, 1), (7, 2, 7, 7)], ids=lambda c: "%dx%d_%d_%d" % c)
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("form", [E.EDG_FORM_STORED, E.EDG_FORM_DIRECT], ids=["stored", "direct"])
def test_hxv_tile_complex(case, prec, form):
    """Complex Hij: one launch up to 10,000,000 states, down pass and row tiles beyond (the last
    case). FP64 to 1e-13 of the largest element, FP32 to 2e-6."""
    import torch
    lx, ly, nup, ndw = case
    if nup == ndw == 7 and (prec == "f32") != (form == E.EDG_FORM_DIRECT):
        pytest.skip("the oracle takes a minute: two passes as stored FP64 and direct FP32 only")
    h = flux_lattice(lx, ly, 0.25)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw, form)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    v = O.random_vector(3, s.dim) + 1j * O.random_vector(4, s.dim)
    om = O.Model(h, uloc=4.0, xmu=2.0, hfmode=False)
    ref = O.Stored(om, nup, ndw).matvec_z(v) if form == E.EDG_FORM_STORED else O.direct_matvec_z(om, nup, ndw, v)
    x = torch.from_numpy(v).cuda().to(torch.complex128 if prec == "f64" else torch.complex64)
    y = torch.full_like(x, float("nan"))
    fn = L.lib().edg_hxv_dev_f64 if prec == "f64" else L.lib().edg_hxv_dev_f32
    L.check(fn(s.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), "hxv")
    d = np.abs(y.cpu().numpy() - ref).max() / np.abs(ref).max()
    assert d <= (1e-13 if prec == "f64" else 2e-6), d
    s.delete()


@pytest.mark.parametrize("case", [(10, 1, 5, 5, 20, "f64"),  # 252 columns: one slice per warp against two
                                  (3, 4, 4, 4, 12, "f64"), (3, 4, 5, 6, 12, "f32"), (4, 4, 3, 4, 3, "f64"),
                                  (7, 2, 4, 7, 2, "f64")], ids=lambda c: "%dx%d_%d_%d_x%d_%s" % c)
def test_many_columns_are_single_chains(case):
    """Blocks whose tiles go to CTAs of four warps: the coefficients of each column are those of
    a chain of its own, whose CTAs have eight, bit for bit."""
    import torch
    lx, ly, nup, ndw, k, prec = case
    p = E.EDG_PREC_F64 if prec == "f64" else E.EDG_PREC_F32
    s = E.Sector(E.Model(lattice(lx, ly), uloc=4.0, xmu=2.0, hfmode=False), nup, ndw)
    X = torch.tensor(np.stack([O.random_vector(50 + c, s.dim) for c in range(k)]), dtype=torch.float64, device="cuda")
    n, pd, pi = 20, L._pd, L._pi
    a, b, n2, ns = np.zeros((k, n)), np.zeros((k, n)), np.zeros(k), np.zeros(k, dtype=np.int32)
    L.check(L.lib().edg_tridiag_block_dev(s.handle, k, C.c_void_p(X.data_ptr()), n, 1e-9, p, a.ctypes.data_as(pd),
                                          b.ctypes.data_as(pd), n2.ctypes.data_as(pd), ns.ctypes.data_as(pi)), "block")
    for c in (0, k // 2, k - 1):
        a1, b1, n21, ns1 = np.zeros(n), np.zeros(n), C.c_double(), C.c_int()
        L.check(L.lib().edg_tridiag_dev_f64(s.handle, C.c_void_p(X[c].data_ptr()), n, 1e-9, p, a1.ctypes.data_as(pd),
                                            b1.ctypes.data_as(pd), C.byref(n21), C.byref(ns1)), "single")
        assert ns[c] == ns1.value == n and n2[c] == n21.value
        assert np.array_equal(a[c], a1) and np.array_equal(b[c], b1), c
    s.delete()
