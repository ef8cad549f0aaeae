// hxv.cuh -- arguments and arithmetic shared by the H x v kernels (hxv.cu, tile.cu).
#pragma once

#include "common.cuh"

namespace edg {

template <typename T>
struct HxvArgs {
  const T* __restrict__ v;
  T* __restrict__ hv;
  int64_t dimup, dimdw;
  const uint32_t* __restrict__ off_up;
  const uint32_t* __restrict__ src_up;
  const T* __restrict__ val_up;
  const uint32_t* __restrict__ off_dw;
  const uint32_t* __restrict__ src_dw;
  const T* __restrict__ val_dw;
  const T* __restrict__ e_up;
  const T* __restrict__ e_dw;
  const uint32_t* __restrict__ map_up;
  const uint32_t* __restrict__ map_dw;
  T U;
  // Lanczos-fused mode (v = u / bn[jstep] is applied with the scale folded into the matrix
  // elements; the step forms w = Hv - (bn[j]/bn[j-1]) uprev and the up pass the partial
  // <v, w>; lz_sub_in_dw says which pass subtracts uprev)
  const double* __restrict__ bn = nullptr;
  int jstep = 0;
  const T* __restrict__ uprev = nullptr;
  double* __restrict__ partial = nullptr;  // reduction scratch [kRedSlots]
  double* __restrict__ red_out = nullptr;  // receives <v, w>
  // Block mode (several vectors of the sector in one launch, blockIdx.y = column c): column c
  // reads v + c*vstride, writes hv + c*vstride, uses uprev + c*vstride, bn + c*sstride,
  // red_out + c*sstride and the scratch partial + c*kRedSlots; a column whose active[c] is 0
  // is skipped. ncols is the launch's gridDim.y (1 for a single vector).
  int64_t vstride = 0, sstride = 0;
  const int* __restrict__ active = nullptr;
  int ncols = 1;
  int dwv = 0, upv = 0;  // kernel choice (edg_sector_s::hxv_dw / hxv_up)
};

// Which pass of the Lanczos-fused step subtracts c * uprev. FP32: the down pass, as the start
// of its diagonal term (it runs at a fraction of HBM bandwidth, and the up pass, short of
// registers, then reads no third vector). FP64: the up pass, after all hops, which is the
// reference's order (w = Hv - b u_prev), so FP64 coefficients stay bit-exact.
template <typename T>
constexpr bool lz_sub_in_dw() { return sizeof(T) == 4; }

// Points a block-mode launch's arguments at this CTA's column; false when the column has
// stopped. A single-vector launch (gridDim.y == 1, active == nullptr) is left as it is.
template <typename T>
__device__ __forceinline__ bool select_column(HxvArgs<T>& a) {
  const int64_t c = blockIdx.y;
  if (a.active && !a.active[c]) return false;
  if (c) {
    a.v += c * a.vstride;
    a.hv += c * a.vstride;
    if (a.uprev) a.uprev += c * a.vstride;
    if (a.bn) a.bn += c * a.sstride;
    if (a.partial) a.partial += c * kRedSlots;
    if (a.red_out) a.red_out += c * a.sstride;
  }
  return true;
}

template <typename T>
__device__ __forceinline__ T fmaT(T a, T b, T c);
template <>
__device__ __forceinline__ float fmaT<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }
template <>
__device__ __forceinline__ double fmaT<double>(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename T, int RT>
struct VecT;
template <> struct VecT<float, 1> { using type = float; };
template <> struct VecT<float, 2> { using type = float2; };
template <> struct VecT<float, 4> { using type = float4; };
template <> struct VecT<double, 1> { using type = double; };
template <> struct VecT<double, 2> { using type = double2; };

// acc[0..RT) += h * x[0..RT): packed FP32x2 FMAs where the pair shares h (Blackwell
// fma.rn.f32x2; each lane is an IEEE fma, identical to two scalar ones).
template <typename T, int RT>
struct Fma {
  static __device__ __forceinline__ void run(T h, const T* x, T* acc) {
#pragma unroll
    for (int r = 0; r < RT; ++r) acc[r] = fmaT<T>(h, x[r], acc[r]);
  }
};
__device__ __forceinline__ void ffma2(float h, const float* x, float* acc) {
  uint64_t d;
  const uint64_t uh = (uint64_t(__float_as_uint(h)) << 32) | __float_as_uint(h);
  const uint64_t ux = (uint64_t(__float_as_uint(x[1])) << 32) | __float_as_uint(x[0]);
  const uint64_t ua = (uint64_t(__float_as_uint(acc[1])) << 32) | __float_as_uint(acc[0]);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(uh), "l"(ux), "l"(ua));
  acc[0] = __uint_as_float(uint32_t(d));
  acc[1] = __uint_as_float(uint32_t(d >> 32));
}
template <>
struct Fma<float, 2> {
  static __device__ __forceinline__ void run(float h, const float* x, float* acc) { ffma2(h, x, acc); }
};
template <>
struct Fma<float, 4> {
  static __device__ __forceinline__ void run(float h, const float* x, float* acc) {
    ffma2(h, x, acc);
    ffma2(h, x + 2, acc + 2);
  }
};

// acc += h * x on one complex element (re, im)
template <typename T>
__device__ __forceinline__ void cmad(T hr, T hi, const T* x, T* acc) {
  acc[0] = fmaT<T>(hr, x[0], acc[0]);
  acc[0] = fmaT<T>(-hi, x[1], acc[0]);
  acc[1] = fmaT<T>(hr, x[1], acc[1]);
  acc[1] = fmaT<T>(hi, x[0], acc[1]);
}

__device__ __forceinline__ float flip_sign(float h, uint32_t e) {
  return __uint_as_float(__float_as_uint(h) ^ (e & 0x80000000u));
}
__device__ __forceinline__ double flip_sign(double h, uint32_t e) {
  return __longlong_as_double(__double_as_longlong(h) ^ (static_cast<long long>(e & 0x80000000u) << 32));
}

// ---- tile.cu: the parts of H x v that a row-tile launch computes (see there), for the rows of
// `a`, plain or (lz: kUpAdd and kDwUp) as the Lanczos-fused step
enum class TileForm { kUpAdd, kDwUp, kUpDw, kUp };
template <typename T>
int tile_real(const HxvArgs<T>& a, const SpinBasis& up, const SpinBasis& dw, TileForm form, bool lz, cudaStream_t st,
              int sms);
// The same for a complex sector (vi_dw: imaginary parts of the down values).
template <typename T>
int tile_cplx(const HxvArgs<T>& a, const SpinBasis& up, const SpinBasis& dw, const T* vi_dw, TileForm form,
              cudaStream_t st, int sms);

}  // namespace edg
