"""Direct-form sectors whose hop tables nothing would read or would not fit: they keep none and are
applied from the bitstrings, as sectors of any size were; a stored sector with such a table is
refused. Exact columns, or the oracle where it can."""
import ctypes as C

import numpy as np
import pytest

import ed_lattice_b200 as E
from ed_lattice_b200 import _edgpu_lib as L
from oracle import oracle as O
from tests.exact_columns import Columns

pytestmark = pytest.mark.gpu


def _quarter_turn(h):
    h = h.astype(complex)
    i, j = np.argwhere(np.triu(h))[0]
    h[i, j], h[j, i] = 1j, -1j
    return h


def _run(s, prec):
    fn = L.lib().edg_hxv_dev_f64 if prec == "f64" else L.lib().edg_hxv_dev_f32
    return lambda a, b: L.check(fn(s.handle, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())), "hxv")


# lattice, nup, ndw, complex, precision
@pytest.mark.parametrize("case", [(5, 6, 0, 15, False, "f64"),   # 4.8e9 hops of the down spin, one column
                                  (5, 6, 0, 15, True, "f32"),
                                  (22, 1, 1, 11, False, "f64"),  # tables larger than the vector
                                  (9, 2, 9, 2, False, "f32")],   # rows beyond the tiles
                         ids=lambda c: "%dx%d_%d_%d_%s_%s" % (*c[:4], "complex" if c[4] else "real", c[5]))
def test_direct_columns(case):
    import torch
    lx, ly, nup, ndw, cplx, prec = case
    h = E.square_lattice(lx, ly)
    if cplx:
        h = _quarter_turn(h)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw, E.EDG_FORM_DIRECT)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    dt = {("f64", True): torch.complex128, ("f32", True): torch.complex64, ("f64", False): torch.float64,
          ("f32", False): torch.float32}[prec, cplx]
    x = torch.zeros(s.dim, dtype=dt, device="cuda")
    y = torch.empty_like(x)
    r = np.random.default_rng(2)
    cols = Columns(h, nup, ndw, 4.0, 2.0, stored=False)
    cols.check(_run(s, prec), x, y, [0, s.dim - 1] + [int(i) for i in r.integers(0, s.dim, 3)])
    s.delete()
    del x, y
    torch.cuda.empty_cache()


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
def test_direct_rows_beyond_the_tiles(cplx):
    import torch
    h = E.square_lattice(17, 1)
    if cplx:
        h = _quarter_turn(h)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), 8, 1, E.EDG_FORM_DIRECT)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    om = O.Model(h, uloc=4.0, xmu=2.0, hfmode=False)
    v = O.random_vector(3, s.dim) + (1j * O.random_vector(4, s.dim) if cplx else 0.0)
    ref = O.direct_matvec_z(om, 8, 1, v) if cplx else O.direct_matvec_d(om, 8, 1, v)
    x = torch.from_numpy(v).cuda()
    y = torch.empty_like(x)
    _run(s, "f64")(x, y)
    got = y.cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max() if cplx else np.array_equal(got, ref)
    s.delete()


def test_stored_table_past_uint32_is_refused():
    with pytest.raises(E.EdgError) as e:
        E.Sector(E.Model(E.square_lattice(5, 6), uloc=4.0, xmu=2.0, hfmode=False), 15, 0)
    assert e.value.status == L.EDG_ERR_UNSUPPORTED
