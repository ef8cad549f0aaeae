"""Sectors of more down configurations than one row group per resident block holds in shared memory:
the grouped down pass behind the complex and direct forms and the stored one, by exact
columns; and the Lanczos-fused step, whose <v, H v> is formed from the same product in torch
(sums of 74 M terms in another order: 1e-12)."""
import ctypes as C

import numpy as np
import pytest

import ed_lattice_b200 as E
from ed_lattice_b200 import _edgpu_lib as L
from tests.exact_columns import Columns

pytestmark = pytest.mark.gpu

# sites of the ring, nup, ndw, complex, form, precision: DimDw = 352,716 (21) and 705,432 (22)
CASES = [(21, 2, 10, True, "stored", "f64"), (21, 3, 10, True, "stored", "f64"), (21, 2, 10, True, "direct", "f32"), (21, 2, 10, False, "direct", "f64"),
         (22, 2, 11, False, "direct", "f32"), (21, 2, 10, False, "stored", "f64"), (22, 2, 11, False, "stored", "f32")]


def _ring(ns, cplx):
    h = E.ring(ns)
    if cplx:
        h = h.astype(complex)
        for i in range(0, ns, 2):  # a quarter turn on every other bond: exact values
            j = (i + 1) % ns
            h[i, j], h[j, i] = 1j, -1j
    return h


@pytest.mark.parametrize("case", CASES, ids=lambda c: "ring%d_%d_%d_%s_%s_%s" % (*c[:3], "complex" if c[3] else "real", *c[4:]))
def test_columns(case):
    import torch
    ns, nup, ndw, cplx, form, prec = case
    h = _ring(ns, cplx)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw,
                 E.EDG_FORM_STORED if form == "stored" else E.EDG_FORM_DIRECT)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    dt = {("f64", True): torch.complex128, ("f32", True): torch.complex64, ("f64", False): torch.float64,
          ("f32", False): torch.float32}[prec, cplx]
    fn = L.lib().edg_hxv_dev_f64 if prec == "f64" else L.lib().edg_hxv_dev_f32
    x = torch.zeros(s.dim, dtype=dt, device="cuda")
    y = torch.empty_like(x)
    run = lambda a, b: L.check(fn(s.handle, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())), "hxv")  # noqa: E731
    cols = Columns(h, nup, ndw, 4.0, 2.0, form == "stored")
    r = np.random.default_rng(1)
    cols.check(run, x, y, [0, s.dim - 1] + [int(i) for i in r.integers(0, s.dim, 4)])
    if form == "stored" and not cplx and prec == "f64":
        v = torch.randn(s.dim, dtype=dt, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
        n, pd = 2, L._pd
        a, b, n2, m = np.zeros(n), np.zeros(n), C.c_double(), C.c_int()
        L.check(L.lib().edg_tridiag_dev_f64(s.handle, C.c_void_p(v.data_ptr()), n, 1e-9, E.EDG_PREC_F64,
                                            a.ctypes.data_as(pd), b.ctypes.data_as(pd), C.byref(n2), C.byref(m)), "chain")
        v /= torch.linalg.vector_norm(v)
        run(v, y)
        a0 = torch.dot(v, y).item()
        b1 = torch.linalg.vector_norm(y - a0 * v).item()
        assert abs(a[0] - a0) <= 1e-12 * abs(a0) and abs(b[1] - b1) <= 1e-12 * b1
    s.delete()
    del x, y
    torch.cuda.empty_cache()
