// reduce.cuh -- the deterministic pair of sums that ends the correction kernels
// (engine.cu, multi.cu).
#pragma once

namespace ccfv {

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sums (a, b) over the block of THREADS threads; thread 0 has the result.
template <int THREADS>
__device__ __forceinline__ void block_sum(double &a, double &b, double (*red)[THREADS / 32]) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = a;
    red[1][w] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = 0.0;
    for (int k = 0; k < THREADS / 32; ++k) {
      a += red[0][k];
      b += red[1][k];
    }
  }
}

// Sums (a, b) over `blocks` blocks in a fixed order: each block leaves its pair
// in partial[2 block], the last one to finish (counter, left at zero) adds
// them, a fixed set per thread, into out[0], out[1].
template <int THREADS>
__device__ void reduce_pair(double a, double b, double *partial, unsigned *counter, int blocks,
                            double *out) {
  __shared__ double red[2][THREADS / 32];
  __shared__ bool last;
  block_sum<THREADS>(a, b, red);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = a;
    partial[2 * blockIdx.x + 1] = b;
    __threadfence();
    last = atomicAdd(counter, 1u) == (unsigned)blocks - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  a = b = 0.0;
  for (int k = threadIdx.x; k < blocks; k += THREADS) {
    a += __ldcg(partial + 2 * k);
    b += __ldcg(partial + 2 * k + 1);
  }
  block_sum<THREADS>(a, b, red);
  if (threadIdx.x == 0) {
    out[0] = a;
    out[1] = b;
    *counter = 0;
  }
}

}  // namespace ccfv
