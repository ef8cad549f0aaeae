"""The single-pass H x v (down choice 3) on a sector of more than 2^31 states with short rows, whose
up rows the tile kernels would take: exact columns at rows whose first element lies past 2^31."""
import ctypes as C

import pytest

import ed_lattice_b200 as E
from ed_lattice_b200 import _edgpu_lib as L
from tests.exact_columns import Columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [E.EDG_PREC_F32, E.EDG_PREC_F64], ids=["f32", "f64"])
def test_single_pass_past_int32(prec):
    import torch
    h = E.ring(22)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), 4, 8)
    assert s.dim > 2**31 and s.dimup == 7315
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    f32 = prec == E.EDG_PREC_F32
    s.set_kernels(12 if f32 else 3, prec)
    fn = L.lib().edg_hxv_dev_f32 if f32 else L.lib().edg_hxv_dev_f64
    x = torch.zeros(s.dim, dtype=torch.float32 if f32 else torch.float64, device="cuda")
    y = torch.empty_like(x)
    cols = Columns(h, 4, 8, 4.0, 2.0)
    run = lambda a, b: L.check(fn(s.handle, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())), "hxv")  # noqa: E731
    cols.check(run, x, y, (0, 2**31 - 1, 2**31 + 12_345, s.dim - s.dimup + 17, s.dim - 1))
    s.delete()
    del x, y
    torch.cuda.empty_cache()
