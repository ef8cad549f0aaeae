"""The sector-Lanczos work whose speed is measured, one case per way the engine is used.

A case is a dict of plain values. `prepare` builds the model and the sector (which a program
keeps for as long as it works on that sector) and the inputs; `run` is one call a program
makes; `exact` is the same result from torch's sparse and dense FP64 operations alone.

Kinds:
  hxv      H x v on a device vector (edg_hxv_dev_*): the callback under every Krylov method
  gf       the Green's function of all sites from one state: chain block, then the pole sums
  chi      spin susceptibility chains of several momenta from one state, then the pole sums
  lowest   the lowest levels and vectors of one sector (the finite-temperature sector solve)
  e0       the ground-state energy of one sector, FP32 vectors with FP64 refinement
  static   observables and energies of one state
  poles    pole sums over a whole state list on the Matsubara and the real axis
"""
import ctypes as C
import math

import numpy as np
import torch

import ed_lattice_b200 as E
from ed_lattice_b200 import edlat

DEV = "cuda"


def listed():
    return [
        # the half-filled 4x4 Hubbard lattice, the largest sector that one works on every day:
        # FP32 H x v, vectors far larger than L2
        {"name": "hxv_f32_4x4", "kind": "hxv", "lx": 4, "ly": 4, "nup": 8, "ndw": 8, "u": 8.0, "prec": "f32"},
        # FP64 H x v of an odd lattice away from even rows: DimUp = 6435 is odd
        {"name": "hxv_f64_5x3", "kind": "hxv", "lx": 5, "ly": 3, "nup": 7, "ndw": 8, "u": 6.0, "prec": "f64"},
        # FP64 H x v of the largest sector of a finite-temperature list, vectors inside L2
        {"name": "hxv_f64_3x4", "kind": "hxv", "lx": 3, "ly": 4, "nup": 6, "ndw": 6, "u": 4.0, "prec": "f64"},
        # the smallest everyday sector: one call is launch latency
        {"name": "hxv_f64_ring8", "kind": "hxv", "lx": 8, "ly": 1, "nup": 4, "ndw": 4, "u": 4.0, "prec": "f64"},
        # the on-the-fly form (ed_sparse_H=F), which keeps no hop tables
        {"name": "hxv_direct_4x4", "kind": "hxv", "lx": 4, "ly": 4, "nup": 6, "ndw": 6, "u": 8.0, "prec": "f64",
         "form": "direct"},
        # a lattice in a magnetic flux: complex Hij and complex vectors
        {"name": "hxv_flux_4x4", "kind": "hxv", "lx": 4, "ly": 4, "nup": 5, "ndw": 5, "u": 8.0, "prec": "f64",
         "flux": 0.25},
        # Green's function of every site from one state of a finite-temperature list
        {"name": "gf_f64_3x4", "kind": "gf", "lx": 3, "ly": 4, "nup": 6, "ndw": 6, "u": 4.0, "prec": "f64",
         "nchain": 12, "nlanc": 150},
        # spin susceptibility of four momenta on a large sector, FP32 vectors
        {"name": "chi_f32_4x4", "kind": "chi", "lx": 4, "ly": 4, "nup": 6, "ndw": 6, "u": 8.0, "prec": "f32",
         "nchain": 4, "nlanc": 100},
        # the finite-temperature sector solve: lowest 4 levels and their vectors
        {"name": "lowest4_3x4", "kind": "lowest", "lx": 3, "ly": 4, "nup": 6, "ndw": 6, "u": 4.0, "k": 4},
        # ground-state energy of a large sector
        {"name": "e0_refine_4x4", "kind": "e0", "lx": 4, "ly": 4, "nup": 6, "ndw": 6, "u": 8.0},
        # observables and energies of a ground state
        {"name": "static_4x4", "kind": "static", "lx": 4, "ly": 4, "nup": 7, "ndw": 7, "u": 8.0},
        # the Green's function of a whole state list on both axes
        {"name": "poles_120k", "kind": "poles", "npoles": 120000, "nmats": 4096, "nreal": 5000},
    ]


# Lattices of the drawn cases: rings, ladders and square clusters of 8 to 16 sites.
LATTICES = [(8, 1), (2, 4), (9, 1), (3, 3), (10, 1), (5, 2), (11, 1), (4, 3), (3, 4), (13, 1), (7, 2), (5, 3), (4, 4)]


def _sector_near(rng, lo, hi, lattices=LATTICES):
    """A sector whose dimension is near a size drawn evenly over the logarithm of [lo, hi]."""
    every = []
    for lx, ly in lattices:
        ns = lx * ly
        for nup in range(2, ns - 1):
            for ndw in range(2, ns - 1):
                d = math.comb(ns, nup) * math.comb(ns, ndw)
                if lo <= d <= hi:
                    every.append((d, lx, ly, nup, ndw))
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    every.sort(key=lambda s: abs(math.log(s[0] / want)))
    _, lx, ly, nup, ndw = rng.choice(every[:12])
    return {"lx": lx, "ly": ly, "nup": nup, "ndw": ndw}


def draw(rng):
    kind = rng.choice(["hxv", "hxv", "hxv", "hxv", "gf", "gf", "chi", "lowest", "e0", "static", "poles"])
    u = rng.choice([2.0, 4.0, 6.0, 8.0, 10.0])
    if kind == "hxv":
        how = rng.choice(["plain", "plain", "plain", "tp", "direct", "flux"])
        c = {"kind": kind, **_sector_near(rng, 4000, {"direct": 6.5e7, "flux": 2e7}.get(how, 1.66e8)), "u": u,
             "prec": rng.choice(["f32", "f64"])}
        if how == "tp":  # next-nearest hopping: longer hop lists, two hopping values
            c["tp"] = rng.choice([0.125, 0.25, -0.25])
        if how == "direct":
            c["form"] = "direct"
        if how == "flux":
            c["flux"] = rng.choice([0.125, 0.25, 0.375])
        return c
    if kind == "poles":
        return {"kind": kind, "npoles": int(math.exp(rng.uniform(math.log(600), math.log(120000)))),
                "nmats": rng.randrange(500, 4097), "nreal": rng.randrange(500, 5001)}
    if kind == "gf":
        c = {"kind": kind, **_sector_near(rng, 4000, 860000), "u": u, "prec": rng.choice(["f32", "f64"])}
        c["nchain"] = rng.randrange(1, 1 + min(12, c["lx"] * c["ly"]))
        c["nlanc"] = rng.randrange(80, 151)
        return c
    if kind == "chi":
        c = {"kind": kind, **_sector_near(rng, 4000, 2e7), "u": u, "prec": rng.choice(["f32", "f64"])}
        c["nchain"] = rng.randrange(1, min(5, c["lx"] * c["ly"]))
        c["nlanc"] = rng.randrange(60, 101)
        return c
    if kind == "lowest":
        return {"kind": kind, **_sector_near(rng, 4000, 860000), "u": u, "k": rng.randrange(1, 5)}
    if kind == "e0":
        return {"kind": kind, **_sector_near(rng, 1e5, 6.5e7), "u": u}
    return {"kind": kind, **_sector_near(rng, 4000, 1.31e8), "u": u}


# ------------------------------------------------------------------------------- inputs
def _disorder(case, seed):
    """On-site energies, multiples of 2^-16 as in the repository's disordered 3x4 lattice."""
    eps = np.random.default_rng(seed).uniform(-1.0, 1.0, case["lx"] * case["ly"])
    return np.round(eps * 65536) / 65536


def _hij(case, seed):
    """Nearest-neighbour -1 (periodic), next-nearest tp on both diagonals, a Peierls phase per x bond."""
    lx, ly = case["lx"], case["ly"]
    flux, tp = case.get("flux", 0.0), case.get("tp", 0.0)
    H = np.zeros((lx * ly, lx * ly), dtype=np.complex128 if flux else np.float64)

    def bond(i, j, h):
        if i != j:
            H[i, j] = h
            H[j, i] = np.conj(h)

    for y in range(ly):
        for x in range(lx):
            i, xp, yp, xm = x + lx * y, (x + 1) % lx, (y + 1) % ly, (x - 1) % lx
            if tp and ly > 1:
                bond(i, xp + lx * yp, -tp)
                bond(i, xm + lx * yp, -tp)
            elif tp:
                bond(i, (x + 2) % lx, -tp)
    for y in range(ly):
        for x in range(lx):
            i = x + lx * y
            bond(i, (x + 1) % lx + lx * y, -np.exp(2j * np.pi * flux * (y + 1)) if flux else -1.0)
            bond(i, x + lx * ((y + 1) % ly), -1.0)
    if case["kind"] in ("gf", "lowest", "e0"):
        H[np.diag_indices(lx * ly)] = _disorder(case, seed)
    return H


def _vector(case, seed, dim, dtype):
    """A normalised random vector: a Lanczos start, or the typical thermal state of a sector."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    v = torch.randn(dim, generator=g, device=DEV, dtype=dtype)
    return v / torch.linalg.vector_norm(v)


def _dim(case, dup=0):
    ns = case["lx"] * case["ly"]
    return math.comb(ns, case["nup"] + dup) * math.comb(ns, case["ndw"])


def _dtype(case):
    if case.get("flux"):
        return torch.complex128 if case["prec"] == "f64" else torch.complex64
    return torch.float64 if case.get("prec", "f64") == "f64" else torch.float32


def _qcos(case):
    """Site weights cos(q.r) of the first `nchain` momenta after q = 0."""
    lx, ly = case["lx"], case["ly"]
    x, y = np.arange(lx * ly) % lx, np.arange(lx * ly) // lx
    return np.array([np.cos(2 * np.pi * ((q % lx) * x / lx + (q // lx) * y / ly)) for q in range(1, case["nchain"] + 1)])


def _pole_inputs(case, seed):
    r = np.random.default_rng(seed)
    p = r.uniform(-12.0, 12.0, case["npoles"])
    w = r.exponential(1.0, case["npoles"]) / case["npoles"]
    wm, _, wr, _, _ = edlat.grids(0.05, lmats=case["nmats"], lreal=case["nreal"])
    return p, w, np.concatenate([1j * wm, wr + 0.02j])


def _energy_below(case, seed):
    """The energy the chains' poles are counted from: that of free electrons, which U only raises."""
    eps = np.linalg.eigvalsh(_hij(case, seed))
    up = case["nup"] + (1 if case["kind"] == "gf" else 0)
    return float(eps[:up].sum() + eps[: case["ndw"]].sum() - case["u"] / 2 * (up + case["ndw"]))


def _matsubara():
    return 1j * np.pi * 0.05 * (2 * np.arange(1, 1025) - 1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poles":
        p, w, z = _pole_inputs(case, seed)
        return {"case": case, "p": p, "w": w, "z": z}
    model = E.Model(_hij(case, seed), uloc=case["u"], xmu=case["u"] / 2, hfmode=False)
    form = E.EDG_FORM_DIRECT if case.get("form") == "direct" else E.EDG_FORM_STORED
    sec = E.Sector(model, case["nup"], case["ndw"], form)
    st = {"case": case, "model": model, "sector": sec, "seed": seed}
    if kind == "hxv":
        sec.set_stream(torch.cuda.current_stream().cuda_stream)
        st["v"] = _vector(case, seed, sec.dim, _dtype(case))
        st["hv"] = torch.empty_like(st["v"])
    if kind in ("gf", "chi", "static"):
        sec.set_state(_vector(case, seed, sec.dim, torch.float64).cpu().numpy())
    if kind in ("gf", "chi"):
        st["ei"] = _energy_below(case, seed)
        st["z"] = _matsubara()
    if kind == "gf":
        st["target"] = E.Sector(model, case["nup"] + 1, case["ndw"])
    if kind == "chi":
        st["qcos"] = _qcos(case)
    return st


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "hxv":
        fn = E.lib().edg_hxv_dev_f64 if case["prec"] == "f64" else E.lib().edg_hxv_dev_f32
        status = fn(state["sector"].handle, C.c_void_p(state["v"].data_ptr()), C.c_void_p(state["hv"].data_ptr()))
        if status != 0:
            raise E.EdgError(status, "spHtimesV", E.lib().edg_last_error().decode())
        return state["hv"]
    if kind == "poles":
        return edlat.eval_poles(state["p"], state["w"], state["z"])
    sec = state["sector"]
    if kind in ("gf", "chi"):
        prec = E.EDG_PREC_F64 if case["prec"] == "f64" else E.EDG_PREC_F32
        if kind == "gf":
            chains = E.gf_chain_block(sec, state["target"], +1, range(1, case["nchain"] + 1), 1, case["nlanc"],
                                      state["ei"], precision=prec)
        else:
            chains = E.chi_chain_block(sec, case["nlanc"], state["ei"], kind=0, qcos=state["qcos"], precision=prec)
        g = np.array([edlat.eval_poles(c.poles, c.weight, state["z"]) for c in chains])
        return g if case["prec"] == "f64" else g.astype(np.complex64)  # FP32 vectors: FP32 results
    if kind == "lowest":
        # the vectors enter thermal averages: converged well below what those are printed to
        ev, vecs, _, _ = sec.lowest_k(case["k"], seed=state["seed"], maxit=1024, tol=1e-12)
        return {"evals": ev, "vectors": vecs}
    if kind == "e0":
        e0, _, _ = E.sp_lanc_eigh(sec, seed=state["seed"], maxit=150, tol=1e-10, mode=E.EDG_GS_F32_REFINE,
                                  want_vector=False)
        return e0
    return {"observables": sec.observables(), "energy": sec.energy()}


# --------------------------------------------------------------------------------- work
def _hops(case, dup=0):
    """Mean hops per configuration, both spins."""
    ns = case["lx"] * case["ly"]
    H = _hij(case, 0)
    nb = np.count_nonzero(H) - np.count_nonzero(np.diag(H))
    return sum(nb * n * (ns - n) / (ns * (ns - 1)) for n in (case["nup"] + dup, case["ndw"]))


def work(case):
    kind = case["kind"]
    if kind == "poles":
        nz = case["nmats"] + case["nreal"]
        return {"bytes": 16.0 * (case["npoles"] + 2 * nz), "flops": 8.0 * case["npoles"] * nz}
    dup = 1 if kind == "gf" else 0
    d, real = _dim(case, dup), 2 if case.get("flux") else 1
    step = d * (2.0 * _hops(case, dup) + 4.0) * real * real
    size = 8 if case.get("prec", "f64") == "f64" else 4
    if kind == "hxv":
        return {"bytes": 2.0 * d * real * size, "flops": step}
    if kind in ("gf", "chi"):
        steps = case["nchain"] * case["nlanc"]
        return {"bytes": 8.0 * _dim(case) + 16.0 * 1024 * case["nchain"], "flops": steps * (step + 8.0 * d)}
    if kind == "lowest":  # about 50 steps per level, each orthogonalised against 25 vectors
        return {"bytes": 8.0 * d * case["k"], "flops": 50.0 * case["k"] * (step + 100.0 * d)}
    if kind == "e0":  # about 100 steps
        return {"bytes": 8.0 * d, "flops": 100.0 * (step + 8.0 * d)}
    return {"bytes": 8.0 * d, "flops": step + d * (2.0 * case["lx"] * case["ly"] + 6.0)}


# ------------------------------------------------------------- the same results, in torch
class _Torch:
    """H of one sector as sparse matrices per spin and a dense diagonal, FP64 or complex128."""

    def __init__(self, case, seed, dup=0):
        ns = case["lx"] * case["ly"]
        H = _hij(case, seed)
        if np.iscomplexobj(H) and case.get("form") != "direct":
            H = H.conj()  # the stored form keeps conjg(Hij), as the reference's does
        self.dtype = torch.complex128 if np.iscomplexobj(H) else torch.float64
        every = np.arange(1 << ns, dtype=np.int64)
        count = sum((every >> b) & 1 for b in range(ns))
        self.mats, self.occ, loc = [], [], []
        for n in (case["nup"] + dup, case["ndw"]):
            m = every[count == n]
            rank = np.full(1 << ns, -1, dtype=np.int64)
            rank[m] = np.arange(m.size)
            rows, cols, vals = [], [], []
            for a in range(ns):
                for b in range(ns):
                    if a == b or H[a, b] == 0:
                        continue
                    t = np.flatnonzero(((m >> a) & 1) & (1 - ((m >> b) & 1)))
                    lo, hi = min(a, b), max(a, b)
                    between = m[t] & (((1 << hi) - 1) & ~((2 << lo) - 1))
                    sign = 1 - 2 * (count[between] & 1)
                    rows.append(t)
                    cols.append(rank[m[t] - (1 << a) + (1 << b)])
                    vals.append(H[a, b] * sign)
            rows, cols, vals = (np.concatenate(x) for x in (rows, cols, vals))
            coo = torch.sparse_coo_tensor(torch.tensor(np.stack([rows, cols])), torch.tensor(vals, dtype=self.dtype),
                                          (m.size, m.size))
            self.mats.append(coo.coalesce().to_sparse_csr().to(DEV))
            occ = np.stack([(m >> b) & 1 for b in range(ns)], 1).astype(np.float64)
            self.occ.append(torch.tensor(occ, device=DEV))
            loc.append(self.occ[-1] @ torch.tensor(np.real(np.diag(H)) - case["u"] / 2, device=DEV))
        self.diag = loc[1][:, None] + loc[0][None, :]
        self.diag.addmm_(self.occ[1], self.occ[0].T, alpha=case["u"])
        self.shape = tuple(self.diag.shape)

    def hop(self, v):
        """The hopping part of H v, v as [DimDw, DimUp]."""
        out = torch.sparse.mm(self.mats[0], v.T.contiguous()).T.contiguous()
        return out.add_(torch.sparse.mm(self.mats[1], v))

    def mul(self, v):
        v = v.reshape(self.shape)
        return self.hop(v).add_(self.diag * v).reshape(-1)


def _lanczos(h, v, steps, keep):
    """Coefficients of the recurrence from v; `keep`: orthogonalised against every vector before."""
    a, b = [], []
    basis = torch.empty((steps if keep else 0, v.numel()), dtype=v.dtype, device=v.device)
    prev, beta = None, 0.0
    for j in range(steps):
        w = h.mul(v)
        alpha = torch.dot(v, w)
        w.sub_(v * alpha)
        if prev is not None:
            w.sub_(prev * beta)
        if keep:
            basis[j] = v
            q = basis[: j + 1]
            for _ in range(2):
                w.sub_(q.T @ (q @ w))
        a.append(float(alpha))
        beta = torch.linalg.vector_norm(w)
        prev, v = v, w / beta
        b.append(float(beta))
        if b[-1] < 1e-9:
            break
    return np.array(a), np.array(b)


def _tridiagonal(a, b):
    return np.linalg.eigh(np.diag(a) + np.diag(b[: a.size - 1], 1) + np.diag(b[: a.size - 1], -1))


def _green(h, v, steps, z):
    """<v| (z - H)^-1 |v> from `steps` Lanczos steps."""
    n2 = float(torch.dot(v, v))
    if n2 == 0.0:
        return np.zeros(z.size, dtype=np.complex128)
    a, b = _lanczos(h, v / math.sqrt(n2), steps, keep=h.diag.numel() < 2e6)
    th, s = _tridiagonal(a, b)
    return (n2 * s[0] ** 2 / (z[:, None] - th[None, :])).sum(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "poles":
        p, w, z = (torch.tensor(x, device=DEV) for x in _pole_inputs(case, seed))
        out = torch.zeros_like(z)
        for k in range(0, p.numel(), 4096):
            out += (w[None, k:k + 4096] / (z[:, None] - p[None, k:k + 4096])).sum(1)
        return out
    if kind in ("hxv", "static"):
        h = _Torch(case, seed)
        v = _vector(case, seed, _dim(case), _dtype(case)).to(h.dtype)
        if kind == "hxv":
            return h.mul(v)
        v = v.reshape(h.shape)
        p = v * v
        nd, nu = h.occ[1].T @ p.sum(1), h.occ[0].T @ p.sum(0)
        docc = (h.occ[1] * (p @ h.occ[0])).sum(0)
        return {"observables": {"dens": nu + nd, "dens_up": nu, "dens_dw": nd, "docc": docc, "magz": nu - nd},
                "energy": {"ekin": (v * h.hop(v)).sum().item(), "epot": case["u"] * docc.sum().item(),
                           "eknot": 0.0, "ehartree": 0.0}}
    if kind == "lowest":
        if _dim(case) < 2000:
            return None
        h = _Torch(case, seed)
        a, b = _lanczos(h, _vector(case, 1, _dim(case), torch.float64), min(400, _dim(case) // 2), keep=True)
        return {"evals": _tridiagonal(a, b)[0][: case["k"]], "vectors": None}
    if kind == "e0":
        h = _Torch(case, seed)
        a, b = _lanczos(h, _vector(case, 1, _dim(case), torch.float64), 220, keep=False)
        return float(_tridiagonal(a, b)[0][0])
    z = _matsubara() + _energy_below(case, seed)
    frm = _Torch(case, seed)
    psi = _vector(case, seed, _dim(case), torch.float64).reshape(frm.shape)
    if kind == "chi":
        out = []
        for q in _qcos(case):
            f = [o @ torch.tensor(q, device=DEV) for o in frm.occ]
            out.append(_green(frm, ((f[0][None, :] - f[1][:, None]) / 2 * psi).reshape(-1), case["nlanc"], z))
        return np.array(out)
    to, ns, out = _Torch(case, seed, dup=1), case["lx"] * case["ly"], []
    every = np.arange(1 << ns, dtype=np.int64)
    count = sum((every >> b) & 1 for b in range(ns))
    src, tgt = every[count == case["nup"]], every[count == case["nup"] + 1]
    rank = np.full(1 << ns, -1, dtype=np.int64)
    rank[src] = np.arange(src.size)
    for i in range(case["nchain"]):
        t = np.flatnonzero((tgt >> i) & 1)
        s = tgt[t] - (1 << i)
        sign = torch.tensor(1.0 - 2.0 * (count[s & ((1 << i) - 1)] & 1), device=DEV)
        v = torch.zeros(to.shape, dtype=torch.float64, device=DEV)
        v[:, torch.tensor(t, device=DEV)] = psi[:, torch.tensor(rank[s], device=DEV)] * sign
        out.append(_green(to, v.reshape(-1), case["nlanc"], z))
    return np.array(out)
