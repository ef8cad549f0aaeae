"""Host-side rules of csrc/limits.h (which sectors a kernel or a table can take), compiled here with
the host compiler: dimensions, hop counts and shared-memory sizes are arithmetic and need no GPU."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

import ed_lattice_b200 as E
from oracle import oracle as O
from tests.exact_columns import Columns

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include "limits.h"
using namespace edg;
extern "C" {
int down_index(int64_t dim) { return tile_down_index(dim); }
int64_t groups(int64_t dim, int64_t resident, int real, int W) { return dw_group_count(dim, resident, real, W); }
int64_t group_most(int real, int W) { return dw_group_most(real, W); }
int64_t group_smem(int64_t rows, int real, int W) { return dw_group_smem(rows, real, W); }
int pays(int cplx, int real, int64_t dimup, int64_t dimdw, double hops) {
  return tile_pays(cplx != 0, real, dimup, dimdw, hops);
}
int one_pass(int64_t dimup, int64_t dimdw, int64_t most, int tiles) {
  return single_pass_default(dimup, dimdw, most, tiles != 0);
}
uint64_t hops(int ns, int nel, int64_t bonds) { return hop_total(ns, nel, bonds); }
int fits(uint64_t n) { return table_fits(n); }
int direct(int64_t dimup, int64_t dimdw, uint64_t hu, uint64_t hd, int cplx) {
  return direct_tables(dimup, dimdw, hu, hd, cplx != 0);
}
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("limits")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "ed_lattice_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    r = C.CDLL(str(lib))
    r.down_index.argtypes = [C.c_int64]
    r.hops.argtypes, r.hops.restype = [C.c_int, C.c_int, C.c_int64], C.c_uint64
    r.groups.argtypes, r.groups.restype = [C.c_int64, C.c_int64, C.c_int, C.c_int], C.c_int64
    r.group_most.argtypes, r.group_most.restype = [C.c_int, C.c_int], C.c_int64
    r.group_smem.argtypes, r.group_smem.restype = [C.c_int64, C.c_int, C.c_int], C.c_int64
    r.one_pass.argtypes = [C.c_int64, C.c_int64, C.c_int64, C.c_int]
    r.pays.argtypes = [C.c_int, C.c_int, C.c_int64, C.c_int64, C.c_double]
    r.fits.argtypes = [C.c_uint64]
    r.direct.argtypes = [C.c_int64, C.c_int64, C.c_uint64, C.c_uint64, C.c_int]
    return r


def test_columns_are_the_oracles():
    """The columns that the large-sector tests compare with, against the oracle's H x v."""
    h = E.square_lattice(3, 2).astype(complex)
    h[0, 1], h[1, 0] = 1j, -1j
    for hij in (E.square_lattice(3, 2), h):
        om = O.Model(hij, uloc=4.0, xmu=2.0, hfmode=False)
        for stored in (True, False):
            cols = Columns(hij, 2, 3, 4.0, 2.0, stored)
            st = O.Stored(om, 2, 3)
            for i in range(0, st.dim, 7):
                e = np.zeros(st.dim, dtype=complex)
                e[i] = 1.0
                ref = st.matvec_z(e) if stored else O.direct_matvec_z(om, 2, 3, e)
                got = np.zeros(st.dim, dtype=complex)
                for j, v in cols(i).items():
                    got[j] = v
                assert np.array_equal(got, ref), (stored, i)


def test_tile_down_hops_fit_their_index(rules):
    """Down hops of the tiles' whole product are 32-bit element indices, one bit of them a sign."""
    for ns, nup, ndw, fits in ((14, 6, 7, True), (24, 3, 9, False), (22, 4, 11, False), (22, 4, 8, False)):
        dim = math.comb(ns, nup) * math.comb(ns, ndw)
        last = (math.comb(ns, ndw) - 1) * math.comb(ns, nup)  # the last row's first element
        assert bool(rules.down_index(dim)) == fits == (last < 2**31)


def _bonds(h):
    return np.count_nonzero(h) - np.count_nonzero(np.diag(h))


def test_hop_totals(rules):
    """The 64-bit count against the tables that the oracle builds, and past 2^32 by the binomials."""
    for lx, ly in ((1, 1), (2, 1), (8, 1), (3, 3)):
        h = E.square_lattice(lx, ly) if lx * ly > 1 else np.zeros((1, 1))
        ns = lx * ly
        for nel in range(ns + 1):
            assert rules.hops(ns, nel, _bonds(h)) == O.hop_csr(O.Model(h), 1, nel)[1].size
    n = rules.hops(30, 15, _bonds(E.square_lattice(5, 6)))
    assert n == 120 * math.comb(28, 14) and not rules.fits(n)
    assert rules.fits(2**32 - 2) and not rules.fits(2**32 - 1) and not rules.fits(2**32)


@pytest.mark.parametrize("case", [(5, 6, 15, 0, 0, False), (5, 6, 0, 15, 1, False),  # 4.8e9 hops of a spin
                                  (30, 1, 15, 1, 0, False), (30, 1, 1, 15, 0, False),  # 37 GB of tables
                                  (22, 1, 1, 11, 0, False), (22, 1, 1, 11, 1, False),  # more than the vector
                                  (9, 2, 9, 2, 0, False), (9, 2, 9, 2, 1, False),  # rows beyond the tiles
                                  (4, 4, 6, 6, 0, True), (4, 4, 8, 8, 1, True), (8, 1, 4, 4, 0, True),
                                  (9, 2, 2, 9, 1, True), (9, 2, 0, 9, 0, True), (3, 4, 6, 6, 0, True)])
def test_direct_form_tables(rules, case):
    lx, ly, nup, ndw, cplx, want = case
    ns, nb = lx * ly, _bonds(E.square_lattice(lx, ly))
    assert bool(rules.direct(math.comb(ns, nup), math.comb(ns, ndw), rules.hops(ns, nup, nb),
                             rules.hops(ns, ndw, nb), cplx)) == want


@pytest.mark.parametrize("W", [1, 2])
@pytest.mark.parametrize("real", [4, 8])
def test_row_groups_fit_shared_memory(rules, real, W):
    """Every number of down configurations has room in its groups, and four blocks with a group each
    and 4 KB of static arrays in an SM's 228 KB (1 KB of it reserved per block)."""
    most = rules.group_most(real, W)
    assert 4 * (rules.group_smem(most, real, W) + 4096 + 1024) <= 228 * 1024
    dims = {math.comb(n, k) for n in range(1, 31) for k in range(n + 1)}
    dims |= {592 * k * most + d for k in (1, 2, 15) for d in (-1, 0, 1)} | {206_600, 335_700}
    for dim in dims:
        g = rules.groups(dim, 592, real, W)
        assert 1 <= g <= dim and (g % 592 == 0 or g == dim < 592)
        assert g * most >= dim


@pytest.mark.parametrize("case", [(924, 924, 12_000_000, 1, True), (924, 924, 12_000_000, 0, False),
                                  (560, 560, 12_000_000, 0, True),  # 313,600 states
                                  (4368, 1820, 12_000_000, 0, False), (4368, 1820, 4_000_000, 1, False),
                                  (6188, 680, 12_000_000, 0, False), (11440, 120, 12_000_000, 0, True),
                                  (24310, 136, 12_000_000, 0, True), (17550, 351, 12_000_000, 0, True),
                                  (24310, 680, 12_000_000, 0, False)])
def test_single_pass_is_the_default_where_its_kernel_wins(rules, case):
    assert bool(rules.one_pass(*case[:4])) == case[4]


# complex, bytes per real, lattice, nup, ndw; measured on both sides
@pytest.mark.parametrize("case", [(0, 8, 15, 1, 1, 6, False), (0, 8, 18, 1, 15, 1, False), (0, 8, 9, 2, 1, 6, False),
                                  (0, 8, 18, 1, 1, 9, True), (0, 8, 10, 1, 5, 5, True), (0, 8, 4, 4, 8, 1, True),
                                  (0, 8, 5, 3, 7, 1, True), (0, 4, 17, 1, 11, 1, False), (0, 4, 4, 3, 4, 4, True),
                                  (0, 4, 5, 3, 5, 2, True), (0, 4, 19, 1, 1, 12, True), (1, 8, 18, 1, 1, 6, False),
                                  (1, 8, 5, 4, 1, 10, False), (1, 8, 15, 1, 6, 1, False), (1, 8, 4, 4, 5, 1, True),
                                  (1, 8, 8, 1, 4, 4, True), (1, 8, 21, 1, 2, 10, False), (1, 8, 19, 1, 3, 9, True),
                                  (1, 4, 9, 1, 3, 3, False), (1, 4, 4, 3, 6, 2, True), (1, 4, 17, 1, 1, 7, False),
                                  (1, 4, 21, 1, 2, 10, True)])
def test_tiles_run_where_they_win(rules, case):
    cplx, real, lx, ly, nup, ndw, want = case
    ns, nb = lx * ly, _bonds(E.square_lattice(lx, ly))
    up, dw = math.comb(ns, nup), math.comb(ns, ndw)
    hops = rules.hops(ns, nup, nb) / up + rules.hops(ns, ndw, nb) / dw
    assert bool(rules.pays(cplx, real, up, dw, hops)) == want
