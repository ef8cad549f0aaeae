// excite.cu -- excitation operators and static observables on device vectors.
//
//  c^+ / c   : apply_op_CDG / apply_op_C (src/SECTOR.f90:217-268) over a whole vector as in
//              lanc_build_gf_electrons_diag (src/GF/GF_ELECTRONS.f90:241-245,267-271). In the
//              spin-factorised layout they are a signed permutation along one index: along iup
//              (within rows) for spin up, of whole rows for spin down.
//  S^z / N   : apply_op_Sz / apply_op_N (src/SECTOR.f90:271-341), diagonal scalings, with an
//              optional real site-weight vector for momentum combinations (cos(q.r)).
//  J         : the current of lanc_ed_build_oc (src/OC/OC_ELECTRONS.f90:139-205).
//  observables: lanc_observables (src/OBSERVABLES.f90:127-152), per-site moments of |psi|^2.
// Vectors of a complex-Hij sector hold complex elements interleaved (re, im): the kernels take
// the element width W (1 real, 2 complex) as a template argument.
#include <algorithm>

#include "common.cuh"

namespace edg {
namespace {

__device__ __forceinline__ uint32_t rank_c(uint32_t s, const uint32_t* C) {
  uint32_t r = 0;
  int i = 1;
  while (s) {
    int p = __ffs(s) - 1;
    r += C[p * kBinomN + i];
    ++i;
    s &= s - 1;
  }
  return r;
}

// For every target configuration (rank jr in the destination basis of one spin): source
// rank in the origin basis (or -1) and the fermionic sign of c^+/c at `pos` (0-based).
__global__ void k_cop_table(const uint32_t* mapJ, int64_t dimJ, int pos, int op, const uint32_t* C, int64_t* srcI,
                            double* sgn) {
  int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (j >= dimJ) return;
  const uint32_t t = mapJ[j];
  const uint32_t bit = 1u << pos;
  uint32_t s;
  if (op > 0) {  // t = cdg(pos) s : t has pos set, s has it clear
    if (!(t & bit)) { srcI[j] = -1; sgn[j] = 0.0; return; }
    s = t & ~bit;
  } else {  // t = c(pos) s : t has pos clear, s has it set
    if (t & bit) { srcI[j] = -1; sgn[j] = 0.0; return; }
    s = t | bit;
  }
  srcI[j] = int64_t(rank_c(s, C));
  sgn[j] = (__popc(s & (bit - 1u)) & 1) ? -1.0 : 1.0;  // bits below pos (src/AUX_FUNX.f90:84-86)
}

// spin up: out[jdw][jup] (+)= coef * sgn[jup] * in[jdw][src[jup]], elements of W reals
template <int W>
__global__ void k_cop_up(const double* __restrict__ in, double* __restrict__ out, int64_t dupI, int64_t dupJ,
                         int64_t ddw, const int64_t* __restrict__ src, const double* __restrict__ sg, double coef,
                         int accumulate) {
  for (int64_t row = blockIdx.x; row < ddw; row += gridDim.x) {
    const double* ir = in + row * dupI * W;
    double* orow = out + row * dupJ * W;
    for (int64_t j = threadIdx.x; j < dupJ; j += blockDim.x) {
      const int64_t sidx = src[j];
#pragma unroll
      for (int c = 0; c < W; ++c) {
        const double v = sidx >= 0 ? coef * sg[j] * ir[sidx * W + c] : 0.0;
        if (accumulate) orow[j * W + c] += v; else orow[j * W + c] = v;
      }
    }
  }
}

// spin down: out[jdw][:] (+)= coef * sgn[jdw] * in[src[jdw]][:]
__global__ void k_cop_dw(const double* __restrict__ in, double* __restrict__ out, int64_t dup, int64_t ddwJ,
                         const int64_t* __restrict__ src, const double* __restrict__ sg, double coef, int accumulate) {
  for (int64_t row = blockIdx.x; row < ddwJ; row += gridDim.x) {
    const int64_t sidx = src[row];
    const double f = sidx >= 0 ? coef * sg[row] : 0.0;
    const double* ir = in + (sidx >= 0 ? sidx : 0) * dup;
    double* orow = out + row * dup;
    for (int64_t j = threadIdx.x; j < dup; j += blockDim.x) {
      const double v = sidx >= 0 ? f * ir[j] : 0.0;
      if (accumulate) orow[j] += v; else orow[j] = v;
    }
  }
}

// per-configuration site sums f[r] = sum_i w_i n_i(map[r])
__global__ void k_site_sum(const uint32_t* map, int64_t dim, const double* w, int ns, double* f) {
  int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (r >= dim) return;
  uint32_t s = map[r];
  double acc = 0.0;
  for (int i = 0; i < ns; ++i)
    if ((s >> i) & 1u) acc += w[i];
  f[r] = acc;
}

// out = (kind 0: (fu - fd)/2 ; kind 1: fu + fd) * in, elements of W reals
template <int W>
__global__ void k_diagop(const double* __restrict__ in, double* __restrict__ out, int64_t dup, int64_t ddw,
                         const double* __restrict__ fu, const double* __restrict__ fd, int kind) {
  for (int64_t row = blockIdx.x; row < ddw; row += gridDim.x) {
    const double d = fd[row];
    for (int64_t j = threadIdx.x; j < dup; j += blockDim.x) {
      const double f = kind == 0 ? (fu[j] - d) / 2.0 : fu[j] + d;
#pragma unroll
      for (int c = 0; c < W; ++c) out[(row * dup + j) * W + c] = f * in[(row * dup + j) * W + c];
    }
  }
}

// Signed hop operator sum_k coef_k T(a_k <- b_k) of one spin, gather form (J of the OC builder).
struct HopOp {
  int nb;
  int a[2 * kMaxSites];
  int b[2 * kMaxSites];
  double c[2 * kMaxSites];
  double ci[2 * kMaxSites];  // imaginary parts (complex Hij)
};

__device__ __forceinline__ int parity_between(uint32_t t, int a, int b) {
  int lo = a < b ? a : b, hi = a < b ? b : a;
  uint32_t mask = ((1u << hi) - 1u) & ~((2u << lo) - 1u);
  return __popc(t & mask) & 1;
}

// acc += (c + i ci) * x for W = 2 (complex elements), acc += c * x for W = 1
template <int W>
__device__ __forceinline__ void hop_acc(double c, double ci, const double* x, double* acc) {
  if (W == 1) {
    acc[0] += c * x[0];
  } else {
    acc[0] += c * x[0] - ci * x[W - 1];
    acc[W - 1] += c * x[W - 1] + ci * x[0];
  }
}

template <int W>
__global__ void k_hopop(const double* __restrict__ in, double* __restrict__ out, int64_t dup, int64_t ddw,
                        const uint32_t* mup, const uint32_t* mdw, const uint32_t* C, HopOp hu, HopOp hd) {
  const int64_t n = dup * ddw;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t idw = e / dup, iup = e - idw * dup;
    const uint32_t tu = mup[iup], td = mdw[idw];
    double acc[W];
#pragma unroll
    for (int c = 0; c < W; ++c) acc[c] = 0.0;
    for (int k = 0; k < hu.nb; ++k) {
      const int a = hu.a[k], b = hu.b[k];
      if (((tu >> a) & 1u) && !((tu >> b) & 1u)) {
        const uint32_t s = (tu & ~(1u << a)) | (1u << b);
        const double sg = parity_between(tu, a, b) ? -1.0 : 1.0;
        hop_acc<W>(hu.c[k] * sg, hu.ci[k] * sg, in + (idw * dup + rank_c(s, C)) * W, acc);
      }
    }
    for (int k = 0; k < hd.nb; ++k) {
      const int a = hd.a[k], b = hd.b[k];
      if (((td >> a) & 1u) && !((td >> b) & 1u)) {
        const uint32_t s = (td & ~(1u << a)) | (1u << b);
        const double sg = parity_between(td, a, b) ? -1.0 : 1.0;
        hop_acc<W>(hd.c[k] * sg, hd.ci[k] * sg, in + (int64_t(rank_c(s, C)) * dup + iup) * W, acc);
      }
    }
#pragma unroll
    for (int c = 0; c < W; ++c) out[e * W + c] = acc[c];
  }
}

// Observables: per-site sums of |psi|^2. A thread owns C columns (fixed up bits) and walks the
// rows of its block's chunk: per row one sum for each low site that the row's down configuration
// occupies (the same test for every thread) and one for all rows since the high half of the
// configuration changed (rows ascend, so every few tens of rows), which then joins the total and
// the sums of the high sites it occupies. The up bits enter once, at the end: dens_up_i = sum
// over columns with bit i of the totals, docc_i the same of the site sums, dens_dw_i the site
// sums over all columns. One row per CTA with a test and a 64-bit select for each of 30 sites
// and element took 1205 us on the 4x4 (7,7) sector (1.05 GB). partial[block][3][kMaxSites].
template <int NS, int W, int C>
__global__ void __launch_bounds__(256) k_obs_cols(const double* __restrict__ psi, int64_t dup, int64_t ddw,
                                                  const uint32_t* __restrict__ mup, const uint32_t* __restrict__ mdw,
                                                  int rows_per, double* __restrict__ partial) {
  extern __shared__ uint32_t s_md[];
  __shared__ double s_sum[8][3 * NS];
  const int64_t r0 = int64_t(blockIdx.y) * rows_per;
  const int nr = int(ddw - r0 < rows_per ? ddw - r0 : rows_per);
  for (int i = threadIdx.x; i < nr; i += blockDim.x) s_md[i] = mdw[r0 + i];
  __syncthreads();
  constexpr int M = NS / 2;  // low sites
  double tot[C], blk[C], x[C][NS];
  int64_t col[C];
#pragma unroll
  for (int k = 0; k < C; ++k) {
    col[k] = int64_t(blockIdx.x) * (256 * C) + k * 256 + threadIdx.x;
    tot[k] = blk[k] = 0.0;
#pragma unroll
    for (int i = 0; i < NS; ++i) x[k][i] = 0.0;
  }
  uint32_t high = s_md[0] >> M;  // the rows' high part; blk sums the rows since it changed
  auto flush = [&] {
#pragma unroll
    for (int i = M; i < NS; ++i)
      if ((high >> (i - M)) & 1u) {
#pragma unroll
        for (int k = 0; k < C; ++k) x[k][i] += blk[k];
      }
#pragma unroll
    for (int k = 0; k < C; ++k) {
      tot[k] += blk[k];
      blk[k] = 0.0;
    }
  };
  constexpr int U = 4;  // rows whose elements are loaded together
  for (int r = 0; r < nr; r += U) {
    double p[U][C], q[U][C];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int k = 0; k < C; ++k) {
        p[u][k] = q[u][k] = 0.0;
        if (r + u < nr && col[k] < dup) {
          const double* e = psi + ((r0 + r + u) * dup + col[k]) * W;
          p[u][k] = __ldcs(e);
          if (W == 2) q[u][k] = __ldcs(e + W - 1);
        }
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t d = s_md[min(r + u, nr - 1)];  // past the chunk: zero elements of its last row
      if ((d >> M) != high) {
        flush();
        high = d >> M;
      }
      double w[C];
#pragma unroll
      for (int k = 0; k < C; ++k) {
        w[k] = W == 1 ? p[u][k] * p[u][k] : __fma_rn(q[u][k], q[u][k], p[u][k] * p[u][k]);
        blk[k] += w[k];
      }
#pragma unroll
      for (int i = 0; i < M; ++i)
        if ((d >> i) & 1u) {
#pragma unroll
          for (int k = 0; k < C; ++k) x[k][i] += w[k];
        }
    }
  }
  flush();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t up[C];
#pragma unroll
  for (int k = 0; k < C; ++k) up[k] = col[k] < dup ? mup[col[k]] : 0u;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < C; ++k) {
      const bool on = (up[k] >> i) & 1u;
      v[0] += on ? tot[k] : 0.0;
      v[1] += x[k][i];
      v[2] += on ? x[k][i] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      for (int o = 16; o > 0; o >>= 1) v[t] += __shfl_down_sync(0xffffffffu, v[t], o);
      if (lane == 0) s_sum[wid][t * NS + i] = v[t];
    }
  }
  __syncthreads();
  double* out = partial + (int64_t(blockIdx.y) * gridDim.x + blockIdx.x) * 3 * kMaxSites;
  for (int j = threadIdx.x; j < 3 * NS; j += blockDim.x)
    if (j % NS < kMaxSites) {
      double t = 0.0;
      for (int w = 0; w < 8; ++w) t += s_sum[w][j];
      out[j / NS * kMaxSites + j % NS] = t;
    }
}

// out[v] = sum over blocks of partial[block][v], v < gridDim.x, fixed order
__global__ void __launch_bounds__(256) k_obs_sum(const double* __restrict__ partial, int nblk, double* __restrict__ out) {
  __shared__ double sh[8];
  double t = 0.0;
  for (int b = threadIdx.x; b < nblk; b += 256) t += partial[int64_t(b) * 3 * kMaxSites + blockIdx.x];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    t = 0.0;
    for (int w = 0; w < 8; ++w) t += sh[w];
    out[blockIdx.x] = t;
  }
}

template <int NS, int W>
int launch_obs(const edg_sector_s* s, const double* psi, DevBuf<double>& part, double* sums, cudaStream_t st) {
  constexpr int C = NS <= 16 ? 2 : 1;
  const int64_t gx = (s->up.dim + 256 * C - 1) / (256 * C);
  // about 8 blocks per SM, at least 8 rows each (the closing reduction costs as much as 10 rows)
  int64_t gy = std::max<int64_t>(1, std::min<int64_t>((s->dw.dim + 7) / 8, (148 * 8 + gx - 1) / gx));
  int64_t per = (s->dw.dim + gy - 1) / gy;
  if (per > 10240) per = 10240;  // row masks in shared memory
  gy = (s->dw.dim + per - 1) / per;
  const int64_t nblk = gx * gy;
  EDG_CHECK(part.alloc(size_t(nblk + 1) * 3 * kMaxSites, st, "observable partials"));
  EDG_CUDA(cudaMemsetAsync(part.p, 0, size_t(nblk + 1) * 3 * kMaxSites * sizeof(double), st));
  k_obs_cols<NS, W, C><<<dim3(unsigned(gx), unsigned(gy)), 256, size_t(per) * sizeof(uint32_t), st>>>(
      psi, s->up.dim, s->dw.dim, s->up.map.p, s->dw.map.p, int(per), part.p);
  double* out = part.p + size_t(nblk) * 3 * kMaxSites;
  k_obs_sum<<<3 * kMaxSites, 256, 0, st>>>(part.p, int(nblk), out);
  EDG_CUDA(cudaGetLastError());
  EDG_CUDA(cudaMemcpyAsync(sums, out, 3 * kMaxSites * sizeof(double), cudaMemcpyDeviceToHost, st));
  EDG_CUDA(cudaStreamSynchronize(st));
  return EDG_OK;
}

// sums[0][i], [1][i], [2][i]: up density, down density and double occupancy of site i in psi
template <int W>
int site_sums(const edg_sector_s* s, const double* psi, double (*sums)[kMaxSites], cudaStream_t st) {
  DevBuf<double> part;
  const int ns = s->model.ns;
  if (ns <= 8) return launch_obs<8, W>(s, psi, part, sums[0], st);
  if (ns <= 12) return launch_obs<12, W>(s, psi, part, sums[0], st);
  if (ns <= 16) return launch_obs<16, W>(s, psi, part, sums[0], st);
  if (ns <= 20) return launch_obs<20, W>(s, psi, part, sums[0], st);
  return launch_obs<32, W>(s, psi, part, sums[0], st);
}

int grid_rows(int64_t rows) { return int(rows < 148 * 8 ? (rows < 1 ? 1 : rows) : 148 * 8); }

}  // namespace

int apply_cop(const edg_sector_s* from, const edg_sector_s* to, int op, int site, int spin, double coef,
              int accumulate, const double* din, double* dout, cudaStream_t st) {
  const int pos = site - 1;
  const SpinBasis& BJ = spin == 1 ? to->up : to->dw;
  DevBuf<int64_t> src;
  DevBuf<double> sg;
  EDG_CHECK(src.alloc(BJ.dim, st, "c-op table"));
  EDG_CHECK(sg.alloc(BJ.dim, st, "c-op table"));
  k_cop_table<<<int((BJ.dim + 255) / 256), 256, 0, st>>>(BJ.map.p, BJ.dim, pos, op, to->binom.p, src.p, sg.p);
  EDG_CUDA(cudaGetLastError());
  const int W = to->cplx ? 2 : 1;
  if (spin == 1) {
    if (W == 2)
      k_cop_up<2><<<grid_rows(to->dw.dim), 256, 0, st>>>(din, dout, from->up.dim, to->up.dim, to->dw.dim, src.p,
                                                         sg.p, coef, accumulate);
    else
      k_cop_up<1><<<grid_rows(to->dw.dim), 256, 0, st>>>(din, dout, from->up.dim, to->up.dim, to->dw.dim, src.p,
                                                         sg.p, coef, accumulate);
  } else {  // whole rows move: a row of W * DimUp reals
    k_cop_dw<<<grid_rows(to->dw.dim), 256, 0, st>>>(din, dout, W * to->up.dim, to->dw.dim, src.p, sg.p, coef,
                                                    accumulate);
  }
  EDG_CUDA(cudaGetLastError());
  EDG_CUDA(cudaStreamSynchronize(st));  // tables are freed on return
  return EDG_OK;
}

int apply_diagop(const edg_sector_s* s, int kind, const double* wsite, const double* din, double* dout,
                 cudaStream_t st) {
  const int ns = s->model.ns;
  DevBuf<double> w, fu, fd;
  EDG_CHECK(w.alloc(ns, st, "site weights"));
  EDG_CHECK(fu.alloc(s->up.dim, st, "site sums"));
  EDG_CHECK(fd.alloc(s->dw.dim, st, "site sums"));
  EDG_CUDA(cudaMemcpyAsync(w.p, wsite, ns * sizeof(double), cudaMemcpyHostToDevice, st));
  k_site_sum<<<int((s->up.dim + 255) / 256), 256, 0, st>>>(s->up.map.p, s->up.dim, w.p, ns, fu.p);
  k_site_sum<<<int((s->dw.dim + 255) / 256), 256, 0, st>>>(s->dw.map.p, s->dw.dim, w.p, ns, fd.p);
  if (s->cplx)
    k_diagop<2><<<grid_rows(s->dw.dim), 256, 0, st>>>(din, dout, s->up.dim, s->dw.dim, fu.p, fd.p, kind);
  else
    k_diagop<1><<<grid_rows(s->dw.dim), 256, 0, st>>>(din, dout, s->up.dim, s->dw.dim, fu.p, fd.p, kind);
  EDG_CUDA(cudaGetLastError());
  EDG_CUDA(cudaStreamSynchronize(st));
  return EDG_OK;
}

// J along the site chain 1-2-...-Ns-1 (Norb=1): for each isite, jsite=isite+1 (periodic),
// + Hij(isite,jsite) c^+_isite c_jsite - conjg(Hij(jsite,isite)) c^+_jsite c_isite, per spin,
// skipped where Hij is zero (src/OC/OC_ELECTRONS.f90:153-198). Returns r with J|psi> = i r
// (complex r for complex Hij).
int apply_current(const edg_sector_s* s, const double* din, double* dout, cudaStream_t st) {
  const edg_model_s& m = s->model;
  const int ns = m.ns;
  HopOp h[2];
  for (int sp = 0; sp < 2; ++sp) {
    const int idx = (m.nspin == 2) ? sp : 0;
    h[sp].nb = 0;
    auto im = [&](int io, int jo) { return m.him[idx].empty() ? 0.0 : m.him[idx][io * ns + jo]; };
    for (int isite = 0; isite < ns; ++isite) {
      const int jsite = (isite + 1 == ns) ? 0 : isite + 1;
      // Hij(io=isite, jo=jsite)
      const double t1 = m.hre[idx][isite * ns + jsite], t1i = im(isite, jsite);
      if (t1 != 0.0 || t1i != 0.0) {
        const int k = h[sp].nb++;
        h[sp].a[k] = isite;
        h[sp].b[k] = jsite;
        h[sp].c[k] = t1;
        h[sp].ci[k] = t1i;
      }
      // -conjg(Hij(io=jsite, jo=isite))
      const double t2 = m.hre[idx][jsite * ns + isite], t2i = im(jsite, isite);
      if (t2 != 0.0 || t2i != 0.0) {
        const int k = h[sp].nb++;
        h[sp].a[k] = jsite;
        h[sp].b[k] = isite;
        h[sp].c[k] = -t2;
        h[sp].ci[k] = t2i;
      }
    }
  }
  const int64_t n = s->dim;
  int g = int((n + 255) / 256);
  if (g > 148 * 8) g = 148 * 8;
  if (s->cplx)
    k_hopop<2><<<g, 256, 0, st>>>(din, dout, s->up.dim, s->dw.dim, s->up.map.p, s->dw.map.p, s->binom.p, h[0], h[1]);
  else
    k_hopop<1><<<g, 256, 0, st>>>(din, dout, s->up.dim, s->dw.dim, s->up.map.p, s->dw.map.p, s->binom.p, h[0], h[1]);
  EDG_CUDA(cudaGetLastError());
  EDG_CUDA(cudaStreamSynchronize(st));
  return EDG_OK;
}

int observables(const edg_sector_s* s, const double* psi, double weight, double* dens, double* dens_up,
                double* dens_dw, double* docc, double* magz, cudaStream_t st) {
  double q[3][kMaxSites];
  EDG_CHECK(s->cplx ? site_sums<2>(s, psi, q, st) : site_sums<1>(s, psi, q, st));
  for (int i = 0; i < s->model.ns; ++i) {
    const double u = q[0][i], d = q[1][i], dd = q[2][i];
    if (dens_up) dens_up[i] += weight * u;
    if (dens_dw) dens_dw[i] += weight * d;
    if (dens) dens[i] += weight * (u + d);
    if (docc) docc[i] += weight * dd;
    if (magz) magz[i] += weight * (u - d);
  }
  return EDG_OK;
}

// lanc_energy (src/ENERGY.f90:118-226, Norb=1 terms) for one state:
//  ekin = <psi|H|psi> - <psi|diag(H)|psi> (the off-diagonal part is exactly the hopping), with
//  diag(H) from the site sums: sum_i eps_i n_i per spin + U docc_i, eps_i the one-body energies
//  that the H x v applies (SpinBasis::eps),
//  eknot from the Hij diagonal and the site densities, epot = U sum_i docc_i plus the Hartree
//  term -U/2 sum_i n_i when HFMODE (reported also on its own, as ENERGY.f90:343 adds it).
int energy(edg_sector_s* s, const double* psi, double weight, double* ekin, double* epot, double* eknot,
           double* ehartree) {
  const int ns = s->model.ns;
  const int64_t n = s->vlen;  // <psi|H psi> over reals = Re <psi|H|psi> for complex psi
  cudaStream_t st = s->stream;
  EDG_CHECK(s->w64[0].alloc(n, st, "energy work vector"));
  double* hv = s->w64[0].p;
  DevBuf<double> part;
  EDG_CHECK(part.alloc(size_t(kRedSlots) + 4, st, "energy partials"));
  double* out = part.p + kRedSlots;
  EDG_CHECK(red_scratch_reset(st, part.p));
  if (hxv_lz_available(s, sizeof(double))) {
    // the Lanczos-fused product at step 0 with unit scale: w = H psi - 0 * psi and <psi, w>
    const double one = 1.0;
    EDG_CUDA(cudaMemcpyAsync(out + 1, &one, sizeof(double), cudaMemcpyHostToDevice, st));
    EDG_CHECK(hxv_apply_lz<double>(s, psi, psi, hv, out + 1, 0, part.p, out));
  } else {
    EDG_CHECK(hxv_apply<double>(s, psi, hv));
    EDG_CHECK(dot_dev<double>(st, psi, hv, n, part.p, out));
  }
  double h = 0.0;
  EDG_CUDA(cudaMemcpyAsync(&h, out, sizeof(double), cudaMemcpyDeviceToHost, st));
  double q[3][kMaxSites];  // (the site sums wait for the stream: h and `one` are settled after)
  EDG_CHECK(s->cplx ? site_sums<2>(s, psi, q, st) : site_sums<1>(s, psi, q, st));
  const std::vector<double>& h1 = s->model.hre[0];
  const std::vector<double>& h2 = s->model.nspin == 2 ? s->model.hre[1] : s->model.hre[0];
  double kn = 0.0, ep = 0.0, eh = 0.0, dg = 0.0;
  for (int i = 0; i < ns; ++i) {
    const double nu = q[0][i], nd = q[1][i], dd = q[2][i];
    kn += h1[size_t(i) * ns + i] * nu + h2[size_t(i) * ns + i] * nd;
    ep += s->model.uloc * dd;
    dg += s->up.eps[i] * nu + s->dw.eps[i] * nd + s->U * dd;
    if (s->model.hfmode) eh -= 0.5 * s->model.uloc * (nu + nd);
  }
  if (ekin) *ekin += weight * (h - dg);
  if (eknot) *eknot += weight * kn;
  if (epot) *epot += weight * (ep + eh);
  if (ehartree) *ehartree += weight * eh;
  return EDG_OK;
}

}  // namespace edg
