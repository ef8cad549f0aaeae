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
