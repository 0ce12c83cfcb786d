// Deterministic grid-wide reduction used by the stencil and PCG kernels:
// warp shuffles, then per-block partials in global memory; the last block to
// finish (atomic ticket) combines the partials with a fixed assignment and a
// fixed tree, so results do not depend on block scheduling.
#pragma once

#include <cfloat>

#include "kernels.cuh"

namespace ins2d {


enum RedOp { R_SUM = 0, R_MAX = 1, R_MIN = 2 };

static __device__ __forceinline__ double red_combine(double a, double b, int op) {
  return op == R_SUM ? a + b : (op == R_MAX ? fmax(a, b) : fmin(a, b));
}
static __host__ __device__ __forceinline__ double red_identity(int op) {
  return op == R_SUM ? 0.0 : (op == R_MAX ? -DBL_MAX : DBL_MAX);
}

// Block-level reduction of NQ values followed by the grid-level finish: the
// last block to arrive combines all partials in block order.  Every thread
// of every block must call it.  bid, nb: this block's number and their count
// (a part of the grid may reduce on its own scratch).
template <int NQ>
__device__ bool grid_reduce_at(double (&v)[NQ], const int (&ops)[NQ], const RedScratch &red, double (&out)[NQ], int bid,
                               int nb) {
  __shared__ double sh[32][NQ];
  __shared__ bool last;
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int lane = tid & 31, warp = tid >> 5, nw = (blockDim.x * blockDim.y) >> 5;
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = red_combine(v[q], __shfl_down_sync(0xffffffffu, v[q], off), ops[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) sh[warp][q] = v[q];
  __syncthreads();
  // the values' chains side by side, here and below: one after another they
  // were most of a small kernel's time (four values over 256 blocks, k_update_f
  // at 512^2: 11.3 -> 9.1 us)
  double a[NQ];
  auto warps = [&] {
#pragma unroll
    for (int q = 0; q < NQ; ++q) a[q] = sh[0][q];
#pragma unroll 4
    for (int w = 1; w < nw; ++w)
#pragma unroll
      for (int q = 0; q < NQ; ++q) a[q] = red_combine(a[q], sh[w][q], ops[q]);
  };
  if (tid == 0) {
    warps();
#pragma unroll
    for (int q = 0; q < NQ; ++q) red.partials[(size_t)bid * NQ + q] = a[q];
    __threadfence();
    unsigned int ticket = atomicAdd(red.counter, 1u);
    last = (ticket == (unsigned)nb - 1);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  // the last block: each thread combines a fixed strided subset of the
  // partials in order, then a fixed-shape tree -> deterministic result
  const int nthr = blockDim.x * blockDim.y;
#pragma unroll
  for (int q = 0; q < NQ; ++q) a[q] = red_identity(ops[q]);
  // partials read through L2 (ld.global.cg: written by other blocks before
  // their fence), four loads per value in flight, combined in block order
  int b = tid;
  for (; b + 3 * nthr < nb; b += 4 * nthr) {
    double v[4][NQ];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[k][q] = __ldcg(red.partials + (size_t)(b + k * nthr) * NQ + q);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < NQ; ++q) a[q] = red_combine(a[q], v[k][q], ops[q]);
  }
  for (; b < nb; b += nthr)
#pragma unroll
    for (int q = 0; q < NQ; ++q) a[q] = red_combine(a[q], __ldcg(red.partials + (size_t)b * NQ + q), ops[q]);
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < NQ; ++q) a[q] = red_combine(a[q], __shfl_down_sync(0xffffffffu, a[q], off), ops[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) sh[warp][q] = a[q];
  __syncthreads();
  if (tid == 0) {
    warps();
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      red.result[q] = a[q];
      out[q] = a[q];
    }
    *red.counter = 0u;
  }
  return tid == 0;
}

template <int NQ>
__device__ __forceinline__ bool grid_reduce(double (&v)[NQ], const int (&ops)[NQ], const RedScratch &red,
                                            double (&out)[NQ]) {
  return grid_reduce_at<NQ>(v, ops, red, out, blockIdx.x + gridDim.x * blockIdx.y, gridDim.x * gridDim.y);
}

// Variant for callers that only need red.result.
template <int NQ>
__device__ __forceinline__ void grid_reduce(double (&v)[NQ], const int (&ops)[NQ], const RedScratch &red) {
  double out[NQ];
  grid_reduce<NQ>(v, ops, red, out);
}


}  // namespace ins2d
