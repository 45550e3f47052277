// Deterministic FP64 sums over a grid: block trees, one partial per block, and
// the last block to finish adds the partials in block order.
#pragma once
#include "common.cuh"

namespace ddb {

constexpr int RED_THREADS = 256;
constexpr int RED_MAXK = 8;

__device__ __forceinline__ double2 warp_sum(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  return v;
}

struct NoPost {
  __device__ void operator()(const double2*) const {}
};

// Sums acc[0..k) (k <= KM) over all threads of the grid of RED_THREADS-thread
// blocks into out[0..k); `count` is a zeroed counter that wraps back to 0.  One
// thread of the grid calls post(out) once the sums are there, so a scalar step
// that needs them costs no launch of its own.  Every thread of the grid must
// reach it.
template <int KM, typename Post>
__device__ __forceinline__ void reduce_tail(double2 (&acc)[KM], int k, double2* partials, double2* out, unsigned* count,
                                            Post post) {
  __shared__ double2 wsum[KM][RED_THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < KM; ++q) {  // compile-time indices: acc stays in registers
    if (q >= k) break;
    double2 v = warp_sum(acc[q]);
    if (lane == 0) wsum[q][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    for (int q = 0; q < k; ++q) {
      double2 v = (lane < RED_THREADS / 32) ? wsum[q][lane] : make_double2(0.0, 0.0);
      v = warp_sum(v);
      if (lane == 0) partials[(size_t)q * gridDim.x + blockIdx.x] = v;
    }
  }
  __threadfence();
  if (threadIdx.x == 0) last = (atomicInc(count, gridDim.x - 1) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the last block sums the partials in block order (deterministic)
  for (int q = 0; q < k; ++q) {
    double2 v = make_double2(0.0, 0.0);
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
      const volatile double* pp = reinterpret_cast<volatile double*>(partials + (size_t)q * gridDim.x + b);
      v.x += pp[0];
      v.y += pp[1];
    }
    v = warp_sum(v);
    if (lane == 0) wsum[q][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    for (int q = 0; q < k; ++q) {
      double2 v = (lane < RED_THREADS / 32) ? wsum[q][lane] : make_double2(0.0, 0.0);
      v = warp_sum(v);
      if (lane == 0) out[q] = v;
    }
    if (lane == 0) post(out);
  }
}

}  // namespace ddb
