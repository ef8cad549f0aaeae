"""Default H x v of sectors whose whole product the row tiles do not take: one |value| of up hops and
several of down hops, rows beyond a tile. Default, two passes and the single pass against the
oracle; hopping values are powers of two, so FP64 carries the oracle's bits (FP32: 2e-6 of the
largest element)."""
import ctypes as C

import numpy as np
import pytest

import ed_lattice_b200 as E
from ed_lattice_b200 import _edgpu_lib as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _two_values(lx, ly):
    """Nearest neighbours for the up spin, next-nearest ones too for the down spin."""
    h = E.square_lattice(lx, ly)
    d = h.copy()
    for y in range(ly):
        for x in range(lx):
            for dx in (1, -1):
                i, j = x + lx * y, (x + dx) % lx + lx * ((y + 1) % ly)
                if i != j and d[i, j] == 0.0:
                    d[i, j] = d[j, i] = -0.25
    return np.stack([h, d])


@pytest.mark.parametrize("case", [(3, 4, 6, 6), (3, 4, 6, 3), (4, 4, 5, 2), (17, 1, 8, 2)], ids=lambda c: "%dx%d_%d_%d" % c)
def test_default_two_passes_and_single_pass(case):
    import torch
    lx, ly, nup, ndw = case
    h = E.square_lattice(lx, ly) if ly == 1 else _two_values(lx, ly)
    om = O.Model(h, uloc=4.0, xmu=2.0, hfmode=False)
    s = E.Sector(E.Model(h, uloc=4.0, xmu=2.0, hfmode=False), nup, ndw)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    v = O.random_vector(3, s.dim)
    ref = O.Stored(om, nup, ndw).matvec_d(v)
    x64 = torch.from_numpy(v).cuda()
    for x, prec, fn, single in ((x64, E.EDG_PREC_F64, L.lib().edg_hxv_dev_f64, 3),
                                (x64.float(), E.EDG_PREC_F32, L.lib().edg_hxv_dev_f32, 12)):
        for cand in (None, 0, single):
            if cand is not None:
                s.set_kernels(cand, prec)
            y = torch.full_like(x, float("nan"))
            L.check(fn(s.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())), "hxv")
            d = np.abs(y.cpu().numpy() - ref).max()
            assert d == 0.0 if prec == E.EDG_PREC_F64 else d <= 2e-6 * np.abs(ref).max(), (cand, d)
    s.delete()
