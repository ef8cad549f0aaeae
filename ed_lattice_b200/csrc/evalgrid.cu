// evalgrid.cu -- pole sums on frequency grids.
//
// The evaluation loops of lanc_eval_gf_electrons (src/GF/GF_ELECTRONS.f90:503-508):
// G(z_m) = sum_k w_k / (z_m - p_k) over every pole of every state, channel and chain that
// contributes to one Green's function entry, for the Matsubara axis (z = i w_n) and the real
// axis (z = w + i eps). With a few hundred thousand poles and ~10^4 frequencies this is 10^9
// terms w (d - i y) / (d^2 + y^2), d = x - p. A grid of (frequency block, pole chunk) CTAs writes
// per-chunk partial sums, and a second pass adds the chunks in fixed order (deterministic).
// Bound by FP64 arithmetic, most of it in the division, so eight poles share one: with the
// products of pairs, fours and all eight denominators, each reciprocal is a product of the
// others and of 1/all (2.6 products and an eighth of a division per term instead of a division).
// Such a reciprocal carries a few roundings more, the sums fewer: groups are summed apart, chunks
// by pairs. rms error in 1e-16 of the sum of magnitudes, against 64-bit mantissas, with a division
// per term and 64 chunks one after the other / now: 8 poles 0.83 / 0.77, 16 0.92 / 0.89, 64
// 1.41 / 0.69, 150 1.21 / 0.64, 1,200 1.25 / 0.49, 120,000 1.48 / 0.46. Up to 64 poles, where the
// rounding of the quotients counts, each term has its own division (8 poles 1.15 without).
// 120,000 poles x 9,096 frequencies: a division per term 1176 us, per four terms 852, per eight
// 740 with the range tested per group, 662 with it tested per tile of poles.
#include <algorithm>

#include "common.cuh"

namespace edg {
namespace {

constexpr int kEvalThreads = 256;
constexpr int kEvalChunks = 128;  // most pole chunks (second grid dimension)
constexpr int kEvalTile = 1024;   // poles staged in shared memory at a time
constexpr int kEvalOwn = 64;      // most poles whose terms have a division each

__device__ __forceinline__ void add_term(double w, double d, double a, double y, double& re, double& im) {
  const double s = w / a;
  re = __fma_rn(s, d, re);
  im = __fma_rn(-s, y, im);
}

// the terms of eight poles with one division; every denominator within 1e-35..1e35
__device__ __forceinline__ void add_eight(const double* p, const double* w, double x, double y, double yy, double& re,
                                          double& im) {
  double d[8], a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    d[i] = x - p[i];
    a[i] = __fma_rn(d[i], d[i], yy);
  }
  const double a01 = a[0] * a[1], a23 = a[2] * a[3], a45 = a[4] * a[5], a67 = a[6] * a[7];
  const double lo = a01 * a23, hi = a45 * a67;
  const double r = 1.0 / (lo * hi), rlo = r * hi, rhi = r * lo;  // 1/lo, 1/hi
  const double pr[4] = {rlo * a23, rlo * a01, rhi * a67, rhi * a45};  // 1/a01, ...
  double tr = 0.0, ti = 0.0;  // summed apart: fewer roundings at the size of the whole sum
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double s = w[i] * (pr[i >> 1] * a[i ^ 1]);
    tr = __fma_rn(s, d[i], tr);
    ti += s;
  }
  re += tr;
  im = __fma_rn(-ti, y, im);
}

__global__ void __launch_bounds__(kEvalThreads) k_eval_poles(const double* __restrict__ poles,
                                                             const double* __restrict__ weights, int64_t npoles,
                                                             const double* __restrict__ zr,
                                                             const double* __restrict__ zi, int64_t nz,
                                                             double* __restrict__ part) {
  __shared__ __align__(16) double sp[kEvalTile], sw[kEvalTile];
  __shared__ double s_max[kEvalThreads / 32];
  const int64_t m = blockIdx.x * int64_t(kEvalThreads) + threadIdx.x;
  const int64_t per = (npoles + gridDim.y - 1) / gridDim.y;
  const int64_t k0 = blockIdx.y * per, k1 = k0 + per < npoles ? k0 + per : npoles;
  const double x = m < nz ? zr[m] : 0.0, y = m < nz ? zi[m] : 1.0, yy = y * y;
  double re = 0.0, im = 0.0;
  for (int64_t t0 = k0; t0 < k1; t0 += kEvalTile) {
    const int cnt = int(k1 - t0 < kEvalTile ? k1 - t0 : kEvalTile);
    __syncthreads();
    double pm = 0.0;
    for (int q = threadIdx.x; q < cnt; q += kEvalThreads) {
      sp[q] = poles[t0 + q];
      sw[q] = weights[t0 + q];
      pm = fmax(pm, fabs(sp[q]));
    }
    for (int o = 16; o > 0; o >>= 1) pm = fmax(pm, __shfl_xor_sync(0xffffffffu, pm, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = pm;
    __syncthreads();
    for (int w = 0; w < kEvalThreads / 32; ++w) pm = fmax(pm, s_max[w]);
    // y^2 <= a <= (|x| + max |p|)^2 + y^2 for every pole of the tile
    const double far = fabs(x) + pm;
    int q = 0;
    if (npoles > kEvalOwn && yy >= 1e-35 && far * far + yy <= 1e35)
      for (; q + 8 <= cnt; q += 8) add_eight(sp + q, sw + q, x, y, yy, re, im);
    for (; q < cnt; ++q) {
      const double d = x - sp[q];
      add_term(sw[q], d, __fma_rn(d, d, yy), y, re, im);
    }
  }
  if (m < nz) {
    part[(int64_t(blockIdx.y) * nz + m) * 2] = re;
    part[(int64_t(blockIdx.y) * nz + m) * 2 + 1] = im;
  }
}

__global__ void k_eval_sum(const double* __restrict__ part, int nchunks, int64_t nz, double* __restrict__ out) {
  const int64_t m = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (m >= nz) return;
  double re[8], im[8];  // every eighth chunk, then by pairs
#pragma unroll
  for (int i = 0; i < 8; ++i) re[i] = im[i] = 0.0;
  for (int c = 0; c < nchunks; c += 8)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c + i < nchunks) {
        re[i] += part[(int64_t(c + i) * nz + m) * 2];
        im[i] += part[(int64_t(c + i) * nz + m) * 2 + 1];
      }
#pragma unroll
  for (int h = 4; h > 0; h >>= 1)
#pragma unroll
    for (int i = 0; i < h; ++i) {
      re[i] += re[i + h];
      im[i] += im[i + h];
    }
  out[2 * m] = re[0];
  out[2 * m + 1] = im[0];
}

}  // namespace

int eval_poles(int64_t npoles, const double* poles, const double* weights, int64_t nz, const double* z_re,
               const double* z_im, double* out_re, double* out_im) {
  if (npoles == 0 || nz == 0) return EDG_OK;
  int dev = 0;
  EDG_CUDA(cudaGetDevice(&dev));
  cudaStream_t st = nullptr;
  EDG_CUDA(pooled_stream(dev, &st));
  // one buffer: poles, weights, frequencies, sums, per-chunk partial sums
  const int64_t gx = (nz + kEvalThreads - 1) / kEvalThreads;
  const int chunks = int(std::min<int64_t>(kEvalChunks, (npoles + 15) / 16));
  DevBuf<double> buf;
  EDG_CHECK(buf.alloc(size_t(2 * npoles + 4 * nz) + size_t(chunks) * nz * 2, st, "pole sums"));
  double* dp = buf.p;
  double* dw = dp + npoles;
  double* dzr = dw + npoles;
  double* dzi = dzr + nz;
  double* out = dzi + nz;
  double* part = out + 2 * nz;
  EDG_CUDA(cudaMemcpyAsync(dp, poles, npoles * sizeof(double), cudaMemcpyHostToDevice, st));
  EDG_CUDA(cudaMemcpyAsync(dw, weights, npoles * sizeof(double), cudaMemcpyHostToDevice, st));
  EDG_CUDA(cudaMemcpyAsync(dzr, z_re, nz * sizeof(double), cudaMemcpyHostToDevice, st));
  EDG_CUDA(cudaMemcpyAsync(dzi, z_im, nz * sizeof(double), cudaMemcpyHostToDevice, st));
  k_eval_poles<<<dim3(unsigned(gx), unsigned(chunks)), kEvalThreads, 0, st>>>(dp, dw, npoles, dzr, dzi, nz, part);
  k_eval_sum<<<unsigned((nz + 255) / 256), 256, 0, st>>>(part, chunks, nz, out);
  EDG_CUDA(cudaGetLastError());
  std::vector<double> h(size_t(nz) * 2);
  EDG_CUDA(cudaMemcpyAsync(h.data(), out, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  EDG_CUDA(cudaStreamSynchronize(st));
  for (int64_t m = 0; m < nz; ++m) {
    out_re[m] += h[2 * m];
    out_im[m] += h[2 * m + 1];
  }
  return EDG_OK;
}

}  // namespace edg
