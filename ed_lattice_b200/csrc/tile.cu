// tile.cu -- the H x v over row tiles held in shared memory as 16-byte slots.
//
// A CTA stages the RT rows idw of a tile (4 FP32, 2 FP64, 2 complex64 or 1 complex128) column
// by column: slot iup holds the RT values of column iup, so one 16-byte shared load per up hop
// feeds RT rows. The up hops of 32 consecutive columns (a slice, one per lane) run slot by slot
// over a 16-bit schedule (SpinBasis::t16_*, k_sched16 in basis.cu). Forms:
//  * kUpAdd: hv already holds diag*v and the down hops; hv += (I x H_up) v. The up pass of
//    large stored sectors.
//  * kDwUp: the whole product, the diagonal, then the row's down hops (one list per row, the
//    same for every lane: coalesced reads of the source rows), then the up hops. One launch and
//    one write of hv; the source rows come from L2, so it is the H x v of sectors whose vectors
//    sit there.
//  * kUpDw, kUp: the direct form's order, diag, UP, DW: whole, or without the down hops, which
//    the down pass then adds.
// Sources come ascending inside each spin part, so FP64 results carry the bits of spMatVec's
// and directMatVec's restatements.
//
// What bounds it: the shared-memory data path, 128 bytes per clock and SM. A slot of a slice
// takes 4 wavefronts (one per 8 lanes) and half a wavefront of entries; in source order without
// a schedule bank conflicts took 36-39 wavefronts per 8 lanes and 16-17 hops on the 4x4
// lattice, with it 22-23. Where a tile fills an SM, staging it is next (a fifth of the pass
// from HBM; the next tile's rows are therefore fetched into L2 ahead). A slice ends at a pair of
// slots: ending at four cost 5 % more slots (24.0 against 22.9 on that lattice, any order) and
// 1-3 % of the product.
// Measured, before (32-bit SELL entries, two FP32 or two FP64 rows) and now, us:
//   up pass, 4x4 (8,8)  FP32  1025 -> 808     4x4 (7,7) FP64  1862 -> 1294
//   up pass, 5x3 (7,8)  FP64   570 -> 397     fused Lanczos 4x4 (6,6) FP64  1084 -> 804
//   whole product, 3x4 (6,6) FP64: two passes 44.0 -> 21.9; 12 Lanczos columns 491 -> 187
//   complex128 4x4 (5,5): 2433 (one thread per element, L1 gathers) -> 923 in two passes;
//   3x4 (6,6) 81 -> 44, 4x4 (4,5) 825 -> 326 in one launch
#include <algorithm>
#include <type_traits>

#include "hxv.cuh"
#include "reduce.cuh"

namespace edg {
namespace {

template <typename T, int W>
struct TileArgs {
  const uint4* __restrict__ ent;       // eight 16-bit entries per lane and batch
  const uint2* __restrict__ code;      // eight palette codes per lane and batch (PAL)
  const uint32_t* __restrict__ off;    // [nsl] first batch of a slice << 9 | its slot pairs
  const double* __restrict__ pal;      // palette: W doubles per code (PAL)
  T h;                                 // value of sign bit 0 (!PAL)
  T h_dw = T(0);                       // the same of the down hops
  bool two = false;                    // each warp stands for two of the sum <v, w>
  int npal = 0;
  int nsl = 0, ntile = 0;
  int csplit = 1;                      // column parts of a tile, each its own work item
  int cap = 0;                         // down hops kept per row (down form)
  const T* __restrict__ vi_dw = nullptr;  // imaginary parts of the down values (W == 2)
};

// One element: W reals.
template <typename T, int W>
struct alignas(sizeof(T) * W) Elem {
  T x[W];
};

// The 16-byte slot at byte offset `at` of the tile and acc += h * slot. The slot is read as
// two 64-bit halves so that FP32 pairs feed the packed FMA without repacking.
template <typename T, int W>
struct SlotAcc;
template <>
struct SlotAcc<float, 1> {  // four rows, two packed pairs
  uint64_t a[2];
  __device__ __forceinline__ void set(const float* x) {
    a[0] = (uint64_t(__float_as_uint(x[1])) << 32) | __float_as_uint(x[0]);
    a[1] = (uint64_t(__float_as_uint(x[3])) << 32) | __float_as_uint(x[2]);
  }
  __device__ __forceinline__ float get(int i) const { return __uint_as_float(uint32_t(a[i >> 1] >> (32 * (i & 1)))); }
  __device__ __forceinline__ void fma(const float* h, ulonglong2 q) {
    const uint64_t hh = (uint64_t(__float_as_uint(h[0])) << 32) | __float_as_uint(h[0]);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a[0]) : "l"(hh), "l"(uint64_t(q.x)));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a[1]) : "l"(hh), "l"(uint64_t(q.y)));
  }
};
template <>
struct SlotAcc<double, 1> {  // two rows
  double a[2];
  __device__ __forceinline__ void set(const double* x) { a[0] = x[0], a[1] = x[1]; }
  __device__ __forceinline__ double get(int i) const { return a[i]; }
  __device__ __forceinline__ void fma(const double* h, ulonglong2 q) {
    a[0] = __fma_rn(h[0], __longlong_as_double(q.x), a[0]);
    a[1] = __fma_rn(h[0], __longlong_as_double(q.y), a[1]);
  }
};

template <>
struct SlotAcc<double, 2> {  // one complex element
  double a[2];
  __device__ __forceinline__ void set(const double* x) { a[0] = x[0], a[1] = x[1]; }
  __device__ __forceinline__ double get(int i) const { return a[i]; }
  __device__ __forceinline__ void fma(const double* h, ulonglong2 q) {
    const double x[2] = {__longlong_as_double(q.x), __longlong_as_double(q.y)};
    cmad(h[0], h[1], x, a);
  }
};
template <>
struct SlotAcc<float, 2> {  // two rows of one complex element
  float a[4];
  __device__ __forceinline__ void set(const float* x) {
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = x[i];
  }
  __device__ __forceinline__ float get(int i) const { return a[i]; }
  __device__ __forceinline__ void fma(const float* h, ulonglong2 q) {
    const float x[4] = {__uint_as_float(uint32_t(q.x)), __uint_as_float(uint32_t(q.x >> 32)),
                        __uint_as_float(uint32_t(q.y)), __uint_as_float(uint32_t(q.y >> 32))};
    cmad(h[0], h[1], x, a);
    cmad(h[0], h[1], x + 2, a + 2);
  }
};

// acc += h * x of one element
template <typename T, int W>
__device__ __forceinline__ void elem_fma(const T* h, const T* x, T* acc) {
  if constexpr (W == 1) acc[0] = fmaT<T>(h[0], x[0], acc[0]);
  else cmad(h[0], h[1], x, acc);
}

// A down hop of a row: the value and the first element of the source row. The plain product over
// tables of one |value| keeps the element with the value's sign in bit 31 instead (PACK): four
// hops per shared-memory load (8 % of the product on 3x4 (6,6), FP64). The Lanczos-fused one, short of
// registers, is slower with it (12 columns of 731,808: 202 -> 217 us).
template <typename T, int W>
struct alignas(8) Hop {
  T val[W];
  uint32_t src;
};

template <typename T, int W, TileForm FORM, bool LZ, bool PAL>
__global__ void __launch_bounds__(1024, 1) k_tile(HxvArgs<T> a, TileArgs<T, W> q) {
  if (!select_column(a)) return;
  constexpr int RT = 16 / int(sizeof(T) * W);  // rows per tile
  constexpr int N = RT * W;                    // reals per slot
  constexpr int KU = 8 / W;                    // down hops in flight
  constexpr bool DIAG = FORM != TileForm::kUpAdd;                            // starts from diag*v, not hv
  constexpr bool DOWN = FORM == TileForm::kDwUp || FORM == TileForm::kUpDw;  // down hops here
  // uprev is subtracted here, after all hops, unless the down pass began from -c * uprev
  constexpr bool SUB = LZ && (DOWN || !lz_sub_in_dw<T>());
  using E = Elem<T, W>;
  constexpr bool PACK = !PAL && !LZ;  // packed down hops
  using H = std::conditional_t<PACK, uint32_t, Hop<T, W>>;
  extern __shared__ __align__(16) unsigned char smem_tile[];
  const int dimup = int(a.dimup);
  ulonglong2* S = reinterpret_cast<ulonglong2*>(smem_tile);
  H* l_hop = reinterpret_cast<H*>(S + dimup + kT16Zero);  // [RT][cap]
  T* s_pal = reinterpret_cast<T*>(l_hop + RT * q.cap);
  uint32_t* s_off = reinterpret_cast<uint32_t*>(s_pal + q.npal * W);  // [nsl]
  __shared__ double s_lz[2];
  __shared__ T s_edw[RT];
  __shared__ uint32_t s_mdw[RT];
  __shared__ int s_cnt[RT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // <v, w>: slices 0, nw, 2 nw, ... of the warp, or (q.two) every other one of them into each
  double pa[2] = {0.0, 0.0}, sc = 1.0;
  if (LZ) {
    sc = 1.0 / a.bn[a.jstep];
    if (threadIdx.x == 0) {
      s_lz[0] = sc;
      s_lz[1] = a.jstep > 0 ? a.bn[a.jstep] / a.bn[a.jstep - 1] : 0.0;
    }
  }
  const T hs = LZ ? T(double(q.h) * sc) : q.h;
  if (PAL)
    for (int i = threadIdx.x; i < q.npal * W; i += blockDim.x) s_pal[i] = T(LZ ? q.pal[i] * sc : q.pal[i]);
  for (int i = threadIdx.x; i < q.nsl; i += blockDim.x) s_off[i] = q.off[i];
  if (threadIdx.x < kT16Zero) S[dimup + threadIdx.x] = make_ulonglong2(0, 0);
  const uint32_t sbase = uint32_t(__cvta_generic_to_shared(S));
  const int nitem = q.ntile * q.csplit;
  for (int item = blockIdx.x; item < nitem; item += gridDim.x) {
    const int tile = q.csplit == 1 ? item : item / q.csplit;
    const int part = item - tile * q.csplit;
    const int s0 = q.nsl * part / q.csplit, s1 = q.nsl * (part + 1) / q.csplit;
    const int64_t r0 = int64_t(tile) * RT;
    const int rows = int(a.dimdw - r0 < RT ? a.dimdw - r0 : RT);
    const E* __restrict__ vt = reinterpret_cast<const E*>(a.v) + r0 * dimup;
    E* __restrict__ ht = reinterpret_cast<E*>(a.hv) + r0 * dimup;
    // The first entries, (rows-in form) sums and (down form) diagonal terms of each slice are
    // loaded while the slice before it runs, the first one's while the tile is staged.
    int sl = s0 + warp;
    bool odd = false;
    uint32_t o = 0;  // next batch
    int np = 0;      // slot pairs left
    uint4 b0 = make_uint4(0u, 0u, 0u, 0u);
    uint2 c0 = make_uint2(0u, 0u);
    E hn[RT] = {};
    T eun = T(0);
    uint32_t mun = 0;
    if (sl < s1) {
      const uint32_t w = q.off[sl];
      o = w >> 9;
      np = int(w & 511u);
      b0 = __ldg(q.ent + o * 32u + lane);
      if (PAL) c0 = __ldg(q.code + o * 32u + lane);
      const int c = min(sl * 32 + lane, dimup - 1);
      if (DIAG) {
        eun = a.e_up[c];
        mun = a.map_up[c];
      } else {
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (r < rows) hn[r] = ht[r * dimup + c];
      }
    }
#pragma unroll 7
    for (int j = threadIdx.x; j < dimup; j += blockDim.x) {
      ulonglong2 slot = make_ulonglong2(0, 0);
      E* xs = reinterpret_cast<E*>(&slot);
#pragma unroll
      for (int r = 0; r < RT; ++r)
        if (r < rows) xs[r] = vt[r * dimup + j];
      S[j] = slot;
    }
    if (DIAG) {
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        if (r >= rows) break;
        const uint32_t k0 = a.off_dw[r0 + r], n = a.off_dw[r0 + r + 1] - k0;
        for (uint32_t k = threadIdx.x; DOWN && k < n; k += blockDim.x) {
          const uint32_t src = a.src_dw[k0 + k] * uint32_t(dimup);
          if constexpr (!PACK) {
            H h;
            h.val[0] = LZ ? T(double(a.val_dw[k0 + k]) * sc) : a.val_dw[k0 + k];
            if (W == 2) h.val[W - 1] = q.vi_dw[k0 + k];
            h.src = src;
            l_hop[r * q.cap + k] = h;
          } else {
            l_hop[r * q.cap + k] = src | (a.val_dw[k0 + k] == q.h_dw ? 0u : 0x80000000u);
          }
        }
        if (threadIdx.x == 0) {
          s_edw[r] = a.e_dw[r0 + r];
          s_mdw[r] = a.map_dw[r0 + r];
          s_cnt[r] = int(n);
        }
      }
    }
    __syncthreads();
    while (sl < s1) {
      const int iup = sl * 32 + lane;
      const bool act = iup < dimup;
      const int c = act ? iup : dimup - 1;  // inactive lanes work on a valid column, store nothing
      const int nsl = sl + nw;
      const bool more = nsl < s1;
      const int cn = min(nsl * 32 + lane, dimup - 1);
      uint32_t on = o;
      int npn = np;
      if (more) {
        const uint32_t w = s_off[nsl];
        on = w >> 9;
        npn = int(w & 511u);
      }
      if (!DOWN) {
        // The next tile's rows into L2 during the second half of this one: with one CTA per SM
        // nothing else covers the staging, which took 9.3 us per 206 KB tile from HBM. Four
        // 128-byte lines per slice; the first half's slices are fetched along with the second's.
        const int64_t nr0 = r0 + int64_t(gridDim.x / q.csplit) * RT;
        const int half = (s1 - s0) >> 1;
        const int ps = lane < 4 ? sl : sl - half;
        constexpr int kLine = 128 / int(sizeof(E));  // columns per line
        const int pr = (lane & 3) / (32 / kLine), pc = ps * 32 + (lane & 3) % (32 / kLine) * kLine;
        if (lane < 8 && sl - s0 >= half && nr0 + pr < a.dimdw && pc < dimup)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const E*>(a.v) + (nr0 + pr) * dimup + pc));
      }
      // uprev: read here next to the down hops; in the up pass fetched into L2 here and read at
      // the end (4x4 (6,6) 818 -> 794 us; the other way round each is slower)
      T up[RT];
      if (SUB && DOWN) {
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (r < rows) up[r] = a.uprev[(r0 + r) * dimup + c];
      }
      if (SUB && !DOWN) {
        constexpr int kLine = 128 / int(sizeof(T)), kPer = 32 / kLine;  // columns per line, lines per row
        const int pr = lane / kPer, pc = sl * 32 + lane % kPer * kLine;
        if (pr < rows && pc < dimup)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a.uprev + (r0 + pr) * dimup + pc));
      }
      // acc += the down hops of the tile's rows
      auto down_hops = [&](T* acc) {
        const E* __restrict__ vc = reinterpret_cast<const E*>(a.v) + c;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          if (r >= rows) break;
          const int n = s_cnt[r];
          const H* lh = l_hop + r * q.cap;
          int k = 0;
          if constexpr (PACK) {
            // K independent source reads, then their terms in order
            auto batch = [&](auto num, const uint32_t* e, int left) {
              constexpr int K = decltype(num)::value;
              E x[K];
#pragma unroll
              for (int u = 0; u < K; ++u)
                if (K > 3 || u < left) x[u] = vc[e[u] & 0x7fffffffu];
#pragma unroll
              for (int u = 0; u < K; ++u)
                if (K > 3 || u < left) acc[r] = fmaT<T>(flip_sign(q.h_dw, e[u]), x[u].x[0], acc[r]);
            };
            const uint4* l4 = reinterpret_cast<const uint4*>(lh);
            for (; k + 8 <= n; k += 8) {
              const uint4 e0 = l4[k >> 2], e1 = l4[(k >> 2) + 1];
              const uint32_t e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
              batch(std::integral_constant<int, 8>{}, e, 8);
            }
            if (k + 4 <= n) {
              const uint4 e0 = l4[k >> 2];
              const uint32_t e[4] = {e0.x, e0.y, e0.z, e0.w};
              batch(std::integral_constant<int, 4>{}, e, 4);
              k += 4;
            }
            if (k < n) {
              const uint4 e0 = l4[k >> 2];
              const uint32_t e[3] = {e0.x, e0.y, e0.z};
              batch(std::integral_constant<int, 3>{}, e, n - k);
            }
          } else {
            for (; k + KU <= n; k += KU) {  // KU independent source reads, then their terms in order
              E x[KU];
#pragma unroll
              for (int u = 0; u < KU; ++u) x[u] = vc[lh[k + u].src];
#pragma unroll
              for (int u = 0; u < KU; ++u) elem_fma<T, W>(lh[k + u].val, x[u].x, acc + r * W);
            }
            if (k < n) {  // the rest: reads past the list repeat its last source
              E x[KU];
#pragma unroll
              for (int u = 0; u < KU - 1; ++u) x[u] = vc[lh[min(k + u, n - 1)].src];
#pragma unroll
              for (int u = 0; u < KU - 1; ++u)
                if (k + u < n) elem_fma<T, W>(lh[k + u].val, x[u].x, acc + r * W);
            }
          }
        }
      };
      T acc0[N];
      if (DIAG) {
        const ulonglong2 xc = S[c];
        const T* xs = reinterpret_cast<const T*>(&xc);
        const T eu = eun;
        const uint32_t mu = mun;
        eun = a.e_up[cn];
        mun = a.map_up[cn];
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          if (r >= rows) {
#pragma unroll
            for (int w = 0; w < W; ++w) acc0[r * W + w] = T(0);
            continue;
          }
          const T d0 = eu + s_edw[r] + a.U * T(__popc(mu & s_mdw[r]));
          const T d = LZ ? T(double(d0) * sc) : d0;
#pragma unroll
          for (int w = 0; w < W; ++w) acc0[r * W + w] = d * xs[r * W + w];
        }
        if (FORM == TileForm::kDwUp) down_hops(acc0);
      } else {
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int w = 0; w < W; ++w) acc0[r * W + w] = hn[r].x[w];
        if (more) {
#pragma unroll
          for (int r = 0; r < RT; ++r)
            if (r < rows) hn[r] = ht[r * dimup + cn];
        }
      }
      SlotAcc<T, W> acc;
      acc.set(acc0);
      // one slot: bits 0..14 its 16 bytes, bit 15 the sign
      auto slot = [&](uint32_t ww, bool odd, uint32_t cd) {
        const uint32_t at = sbase + (odd ? (ww >> 12) & 0x7fff0u : (ww << 4) & 0x7fff0u);
        ulonglong2 x;
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x.x), "=l"(x.y) : "r"(at));
        T h[W];
        if (PAL) {
          const T* pv = s_pal + (cd & 0xffu) * W;
#pragma unroll
          for (int w = 0; w < W; ++w) h[w] = pv[w];
        } else {
          h[0] = flip_sign(hs, odd ? ww : ww << 16);
        }
        acc.fma(h, x);
      };
      for (; np > 0; np -= 4) {
        const uint4 wq = b0;
        const uint2 cq = c0;
        const uint32_t nx = (np > 4 ? ++o : on) * 32u + lane;
        b0 = __ldg(q.ent + nx);
        if (PAL) c0 = __ldg(q.code + nx);
        const uint32_t ws[4] = {wq.x, wq.y, wq.z, wq.w};
        if (np >= 4) {
#pragma unroll
          for (int u = 0; u < 8; ++u) slot(ws[u >> 1], u & 1, (u < 4 ? cq.x : cq.y) >> (8 * (u & 3)));
        } else {  // the slice's last pairs
#pragma unroll
          for (int u = 0; u < 6; ++u) {
            if (u >= 2 * np) break;
            slot(ws[u >> 1], u & 1, (u < 4 ? cq.x : cq.y) >> (8 * (u & 3)));
          }
        }
      }
      if (SUB && !DOWN) {
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (r < rows) up[r] = a.uprev[(r0 + r) * dimup + c];
      }
      T res[N];
#pragma unroll
      for (int i = 0; i < N; ++i) res[i] = acc.get(i);
      if (FORM == TileForm::kUpDw) down_hops(res);
      if (LZ) {
        // w = Hv - c * uprev; partial <v, w>
        const double scl = s_lz[0], cc = s_lz[1];
        const ulonglong2 xc = S[c];
        const T* xs = reinterpret_cast<const T*>(&xc);
        double p1 = DOWN && odd ? pa[1] : pa[0];
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (act && r < rows) {
            const T wt = SUB ? T(double(res[r]) - cc * double(up[r])) : res[r];
            p1 = __fma_rn(double(xs[r]) * scl, double(wt), p1);
            T* p = a.hv + (r0 + r) * dimup + c;
            if (DOWN) *p = wt;
            else __stcs(p, wt);
          }
        if (DOWN && odd) pa[1] = p1;
        else pa[0] = p1;
        if (DOWN) odd = q.two && !odd;
      } else {
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (act && r < rows) {
            E out;
#pragma unroll
            for (int w = 0; w < W; ++w) out.x[w] = res[r * W + w];
            if constexpr (W == 1) {
              if (DOWN) ht[r * dimup + c] = out;
              else __stcs(&ht[r * dimup + c].x[0], out.x[0]);
            } else {
              ht[r * dimup + c] = out;
            }
          }
      }
      sl = nsl;
      o = on;
      np = npn;
    }
    __syncthreads();
  }
  if (LZ) {  // block partial of <v, w>, fixed order
    __shared__ double s_red[32];
    const int ng = DOWN && q.two ? 2 * nw : nw;
#pragma unroll
    for (int g = 0; g < (DOWN ? 2 : 1); ++g) {
      if (g * nw >= ng) break;
      for (int d = 16; d > 0; d >>= 1) pa[g] += __shfl_down_sync(0xffffffffu, pa[g], d);
      if (lane == 0) s_red[warp + g * nw] = pa[g];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < ng; ++w) t += s_red[w];
      a.partial[blockIdx.x] = t;
    }
    finish_in_last_block(a.partial, gridDim.x, a.red_out, 0);
  }
}

template <typename T, int W, TileForm FORM, bool LZ, bool PAL>
int launch(const HxvArgs<T>& a, TileArgs<T, W>& q, cudaStream_t st, int sms) {
  constexpr int RT = 16 / int(sizeof(T) * W);
  constexpr bool DOWN = FORM == TileForm::kDwUp || FORM == TileForm::kUpDw;
  const size_t smem = tile_smem(a.dimup, q.npal, RT * q.cap, sizeof(T) * W);
  auto kern = k_tile<T, W, FORM, LZ, PAL>;
  EDG_CHECK(allow_smem(kern, smem));
  // 64 registers a thread: 1024 threads per SM, in as many CTAs as the tiles leave room for
  const int per_sm = smem <= 54 * 1024 ? 4 : smem <= 111 * 1024 ? 2 : 1;
  q.nsl = int((a.dimup + 31) / 32);
  q.ntile = int((a.dimdw + RT - 1) / RT);
  int warps = 32 / per_sm;
  q.csplit = 1;
  if (DOWN) {
    // Whole product of a sector with few tiles: column parts of a tile, each staging the whole
    // rows again. With fewer slices than resident warps each warp gets one; else parts until
    // three quarters of the resident CTAs have one (3x4 lattice, D = 853,776, one part against
    // two: FP32, 231 tiles, 20.8 against 17.6 us; FP64, 462 tiles, 24.1 against 23.1, with four
    // 26). The CTA then takes no more warps than its rounds of slices fill.
    if (int64_t(q.ntile) * q.nsl <= int64_t(sms) * 32)
      q.csplit = (q.nsl + warps - 1) / warps;
    else
      q.csplit = std::max(1, std::min((3 * sms * per_sm / 4 + q.ntile - 1) / q.ntile, q.nsl / warps));
    const int most = (q.nsl + q.csplit - 1) / q.csplit, rounds = (most + warps - 1) / warps;
    // Two waves or more of CTAs of four warps, eight per SM: their staging and their last rounds
    // overlap better than those of four CTAs of eight (12 Lanczos columns, FP64: 731,808 states
    // 208 -> 187 us, 4x3 (4,4) 133 -> 115; 4x4 (3,8) 147 -> 134; with fewer tiles, 7x2 (4,7),
    // 51 -> 57). The sum <v, w> is the one that eight warps form, so it does not change with the
    // number of columns.
    const bool small = per_sm == 4 && most > 4 && 8 * (smem + 2048) <= 227 * 1024 &&
                       int64_t(q.ntile) * q.csplit * a.ncols >= int64_t(sms) * 16;
    if (small) warps = 4;
    else if (!LZ || per_sm < 4 || most <= warps) warps = (most + rounds - 1) / rounds;
    q.two = small;
  }
  const int threads = 32 * warps;
  int64_t g = int64_t(q.ntile) * q.csplit;
  if (!DOWN || g > kRedMaxBlocks) g = std::min<int64_t>(g, DOWN ? kRedMaxBlocks : int64_t(sms) * per_sm);
  kern<<<dim3(unsigned(g), a.ncols), threads, smem, st>>>(a, q);
  EDG_CUDA(cudaGetLastError());
  return EDG_OK;
}

template <typename T, int W, TileForm FORM, bool LZ>
int launch_pal(const HxvArgs<T>& a, TileArgs<T, W>& q, cudaStream_t st, int sms) {
  if constexpr (W == 1) {
    if (q.npal == 0) return launch<T, W, FORM, LZ, false>(a, q, st, sms);
  }
  return launch<T, W, FORM, LZ, true>(a, q, st, sms);
}

template <typename T, int W>
int tile_pass(const HxvArgs<T>& a, const SpinBasis& up, const SpinBasis& dw, const T* vi_dw, TileForm form, bool lz,
              cudaStream_t st, int sms) {
  const int ord = sizeof(T) == 4 && W == 1 && up.t16_npal == 0 ? 1 : 0;  // FP32: the order-free schedule
  TileArgs<T, W> q;
  q.ent = reinterpret_cast<const uint4*>(up.t16_ent[ord].p);
  q.code = reinterpret_cast<const uint2*>(up.t16_code.p);
  q.off = up.t16_off[ord].p;
  q.pal = up.t16_pal.p;
  q.h = T(up.sell_h);
  q.npal = up.t16_npal;
  q.h_dw = T(dw.sell_h);
  q.cap = form == TileForm::kDwUp || form == TileForm::kUpDw ? (dw.max_row + 3) / 4 * 4 : 0;
  q.vi_dw = vi_dw;
  if constexpr (W == 1) {
    if (lz)
      return form == TileForm::kDwUp ? launch_pal<T, W, TileForm::kDwUp, true>(a, q, st, sms)
                                     : launch_pal<T, W, TileForm::kUpAdd, true>(a, q, st, sms);
  }
  switch (form) {
    case TileForm::kUpAdd: return launch_pal<T, W, TileForm::kUpAdd, false>(a, q, st, sms);
    case TileForm::kDwUp: return launch_pal<T, W, TileForm::kDwUp, false>(a, q, st, sms);
    case TileForm::kUpDw: return launch_pal<T, W, TileForm::kUpDw, false>(a, q, st, sms);
    default: return launch_pal<T, W, TileForm::kUp, false>(a, q, st, sms);
  }
}

}  // namespace

bool tile_available(const edg_sector_s* s, size_t elem, bool down) {
  const SpinBasis& up = s->up;
  if (!up.t16 || (down && !tile_down_index(s->dim))) return false;
  const int rt = int(16 / elem);  // elem: bytes per vector element (a complex one counts whole)
  // the single-value form of the whole product needs one |value| on either side
  if (down && up.t16_npal == 0 && !s->dw.sell_uniform) return false;
  return tile_smem(up.dim, up.t16_npal, down ? rt * ((s->dw.max_row + 3) / 4 * 4) : 0, elem) <= kTileSmemMax;
}

template <typename T>
int tile_real(const HxvArgs<T>& a, const SpinBasis& up, const SpinBasis& dw, TileForm form, bool lz, cudaStream_t st,
              int sms) {
  return tile_pass<T, 1>(a, up, dw, nullptr, form, lz, st, sms);
}
template int tile_real<float>(const HxvArgs<float>&, const SpinBasis&, const SpinBasis&, TileForm, bool, cudaStream_t,
                              int);
template int tile_real<double>(const HxvArgs<double>&, const SpinBasis&, const SpinBasis&, TileForm, bool, cudaStream_t,
                               int);

template <typename T>
int tile_cplx(const HxvArgs<T>& a, const SpinBasis& up, const SpinBasis& dw, const T* vi_dw, TileForm form,
              cudaStream_t st, int sms) {
  return tile_pass<T, 2>(a, up, dw, vi_dw, form, false, st, sms);
}
template int tile_cplx<float>(const HxvArgs<float>&, const SpinBasis&, const SpinBasis&, const float*, TileForm,
                              cudaStream_t, int);
template int tile_cplx<double>(const HxvArgs<double>&, const SpinBasis&, const SpinBasis&, const double*, TileForm,
                               cudaStream_t, int);

}  // namespace edg
