"""Columns H e_i of a sector by the definition, for sectors too large for the oracle's H x v: the
hops of one bitstring pair, with hopping values that products and sums keep exact."""
import math

import numpy as np


def _rank(m):
    """Place of the bitstring m among those with as many bits, ascending."""
    bits = [b for b in range(m.bit_length()) if (m >> b) & 1]
    return sum(math.comb(b, k + 1) for k, b in enumerate(bits))


def _state(r, ns, n):
    """The bitstring of rank r among those of n bits in ns."""
    m = 0
    for k in range(n, 0, -1):
        b = max(c for c in range(ns) if math.comb(c, k) <= r)
        m |= 1 << b
        r -= math.comb(b, k)
    return m


def _hops(h, m, conj):
    """(rank of the target, value) of sum_ab h[a, b] c+_a c_b on the bitstring m."""
    ns = h.shape[0]
    out = []
    for a in range(ns):
        for b in range(ns):
            if a == b or h[a, b] == 0 or not (m >> b) & 1 or (m >> a) & 1:
                continue
            lo, hi = min(a, b), max(a, b)
            between = (m >> (lo + 1)) & ((1 << (hi - lo - 1)) - 1)
            t = m - (1 << b) + (1 << a)
            v = h[a, b].conjugate() if conj else h[a, b]
            out.append((_rank(t), -v if bin(between).count("1") & 1 else v))
    return out


class Columns:
    """Columns of H = sum h c+c (both spins) + U n_up n_dw - xmu n, zero on-site energies. The
    stored form keeps conjg(Hij), the direct form applies Hij."""

    def __init__(self, h, nup, ndw, uloc, xmu, stored=True):
        self.h, self.u, self.xmu, self.stored = h, uloc, xmu, stored
        self.ns, self.nup, self.ndw = h.shape[0], nup, ndw
        self.dimup = math.comb(self.ns, nup)

    def __call__(self, i):
        iup, idw = i % self.dimup, i // self.dimup
        mu, md = _state(iup, self.ns, self.nup), _state(idw, self.ns, self.ndw)
        conj = self.stored and np.iscomplexobj(self.h)
        col = {i: self.u * bin(mu & md).count("1") - self.xmu * (self.nup + self.ndw)}
        for t, v in _hops(self.h, mu, conj):
            j = t + idw * self.dimup
            col[j] = col.get(j, 0) + v
        for t, v in _hops(self.h, md, conj):
            j = iup + t * self.dimup
            col[j] = col.get(j, 0) + v
        return {j: v for j, v in col.items() if v != 0}

    def check(self, hxv, x, y, which):
        """hxv(x, y) on e_i, for each i of `which`: x is zero before and after."""
        import torch
        for i in which:
            x[i] = 1.0
            y.fill_(float("nan"))
            hxv(x, y)
            x[i] = 0.0
            want = self(i)
            idx = torch.tensor(sorted(want), dtype=torch.int64, device=y.device)
            got = y[idx].cpu().numpy()
            assert np.array_equal(got, np.array([want[j] for j in sorted(want)], dtype=got.dtype)), i
            assert int(torch.count_nonzero(y)) == len(want), i
