"""The tiles' whole product on the sectors of more than 500,000 states with rows shorter than a slice
(one column, 18 columns) and with few rows, plain by exact columns and Lanczos-fused against the
two passes (20 coefficients to 1e-9, as in the other Lanczos tests)."""
import ctypes as C

import numpy as np
import pytest

import ed_lattice_b200 as E
from ed_lattice_b200 import _edgpu_lib as L
from tests.exact_columns import Columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(22, 1, 0, 10), (9, 2, 1, 9), (5, 3, 7, 2), (4, 4, 8, 2)], ids=lambda c: "%dx%d_%d_%d" % c)
def test_single_pass_by_tiles(case):
    import torch
    lx, ly, nup, ndw = case
    h = E.square_lattice(lx, ly)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw)
    assert s.dim > 500_000
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    cols = Columns(h, nup, ndw, 4.0, 2.0)
    which = [0, s.dim - 1] + [int(i) for i in np.random.default_rng(6).integers(0, s.dim, 6)]
    for dt, fn in ((torch.float64, L.lib().edg_hxv_dev_f64), (torch.float32, L.lib().edg_hxv_dev_f32)):
        x = torch.zeros(s.dim, dtype=dt, device="cuda")
        run = lambda a, b: L.check(fn(s.handle, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())), "hxv")  # noqa: E731
        cols.check(run, x, torch.empty_like(x), which)
    v = E.random_vector(9, s.dim)
    a3, b3, _, _ = E.tridiag_Hv_sector(s, v, 20)
    s.set_kernels(0, E.EDG_PREC_F64)
    a0, b0, _, _ = E.tridiag_Hv_sector(s, v, 20)
    assert np.allclose(a3, a0, rtol=1e-9, atol=1e-9) and np.allclose(b3, b0, rtol=1e-9, atol=1e-9)
    s.delete()
