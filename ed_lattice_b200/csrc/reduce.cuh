// reduce.cuh -- device helper shared by the kernels that end in a scalar reduction.
#pragma once

#include "common.cuh"

namespace edg {

// Fused reduction tail. Thread 0 of every block has written partial[blockIdx.x]; the last
// block to arrive (counter at partial[kRedMaxBlocks]) sums partial[0..nblk) as kRedThreads
// strided sums, warp by warp, then the warp-shuffle tree, writes *out and resets the counter.
// The order is that of kRedThreads threads whatever the block's size (a multiple of 32). One
// launch per reduction instead of two, with bit-identical results. Every thread of the block
// must call it.
__device__ __forceinline__ void finish_in_last_block(double* __restrict__ partial, int nblk, double* __restrict__ out,
                                                     int do_sqrt) {
  __shared__ int s_last;
  __shared__ double s_fin[kRedThreads / 32];
  unsigned int* ctr = reinterpret_cast<unsigned int*>(partial + kRedMaxBlocks);
  if (threadIdx.x == 0) {
    __threadfence();  // this block's partial is visible before it is counted
    s_last = atomicAdd(ctr, 1u) == unsigned(nblk) - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int vw = wid; vw < kRedThreads / 32; vw += blockDim.x >> 5) {
    double v = 0.0;
    for (int i = vw * 32 + lane; i < nblk; i += kRedThreads) v += __ldcg(partial + i);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) s_fin[vw] = v;
  }
  __syncthreads();
  if (wid == 0) {
    double r = lane < kRedThreads / 32 ? s_fin[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    if (lane == 0) {
      out[0] = do_sqrt ? sqrt(r) : r;
      *ctr = 0u;
    }
  }
}

}  // namespace edg
