// The tridiagonal systems of the fast-diagonalization preconditioner
// (fdm_host.hpp, FdmTri): for every mode b of the diagonalized direction
//   (T_s + lam_b diag(h_s)) zh_b = -w_b,
// solved in place on the rows of the nm x n array w.  With the reciprocal
// pivots tabulated, elimination and back substitution are first-order linear
// recurrences y_k = a_k y_{k-1} + b_k with |a_k| < 1; W warps share a row,
// each lane holds C consecutive unknowns, composes their affine maps,
// and the maps' prefix is scanned over the lanes (and the warps).  So a row
// takes two serial chains of C steps and five shuffle rounds each
// instead of two chains of n steps.
#pragma once

#include "kernels.cuh"

namespace ins2d {

constexpr int kTriChunk = 8;

__device__ __forceinline__ double tri_warp_sum(double v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// one lane's part of a system's tables: C unknowns from s0 (zero outside)
template <int C>
struct TriTab {
  double m[C], e[C], ep;  // reciprocal pivots, off-diagonals, the one before s0
};
template <int C>
__device__ __forceinline__ void tri_tables(const FdmD &F, int b, int s0, TriTab<C> &T) {
  const bool row = b < F.nm;
  const double *__restrict__ pv = F.piv + (size_t)(row ? b : 0) * F.n;
  T.ep = (row && s0 > 0 && s0 <= F.n) ? __ldg(F.e + s0 - 1) : 0.0;
#pragma unroll
  for (int k = 0; k < C; ++k) {
    const bool in = row && s0 + k < F.n;
    T.m[k] = in ? __ldg(pv + s0 + k) : 0.0;
    T.e[k] = in ? __ldg(F.e + s0 + k) : 0.0;
  }
}

// Solves system b (b >= F.nm: none, the threads only take part in the
// barriers) by W warps; wr: this warp's place among them.  y: the lane's C
// values of w_b from unknown s0 = (32 wr + lane) C (zero outside), replaced by
// those of zh_b.  sh: 4 doubles per warp of the block, unused (may be null)
// for W == 1, which has no block-level synchronisation.  on_sum(the warp's sum
// over w_b) is called for the null mode.
struct TriNoSum {
  __device__ void operator()(double) const {}
};
template <int W, int C, class OnSum = TriNoSum>
__device__ __forceinline__ void tri_solve(const FdmD &F, int b, int wr, const TriTab<C> &T, double (&y)[C],
                                          double (*sh)[4], OnSum on_sum = OnSum()) {
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w0 = warp - wr;  // w0: the row's first warp
  const int n = F.n, s0 = (wr * 32 + lane) * C;
  const bool row = b < F.nm;
  const bool null = row && b == F.null_mode;
  const double ep = T.ep;
  const double(&m)[C] = T.m;
  const double(&e)[C] = T.e;
  // the null mode's two sums over w (fdm_host.hpp): independent of the scans
  // below, so their shuffles overlap
  double sum = 0.0, part = 0.0;
  if (null) {
#pragma unroll
    for (int k = 0; k < C; ++k) {
      sum += y[k];
      if (s0 + k < n) part += __ldg(F.nmu + s0 + k) * y[k];
    }
    sum = tri_warp_sum(sum);
    part = tri_warp_sum(part);
    on_sum(sum);
  }
  if constexpr (W > 1) {
    if (lane == 0) {
      sh[warp][0] = sum;
      sh[warp][3] = part;
    }
  }
  // elimination: y_k = -(w_k + e_{k-1} y_{k-1}) m_k
  double A = 1.0, B = 0.0;
#pragma unroll
  for (int k = 0; k < C; ++k) {
    const double a = -(k ? e[k - 1] : ep) * m[k];
    y[k] = -y[k] * m[k];
    B = fma(a, B, y[k]);
    A *= a;
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double a2 = __shfl_up_sync(ALL, A, d), b2 = __shfl_up_sync(ALL, B, d);
    if (lane >= d) {
      B = fma(A, b2, B);
      A *= a2;
    }
  }
  double y0 = 0.0;  // value just before this warp's part
  if constexpr (W > 1) {
    if (lane == 31) {
      sh[warp][1] = A;
      sh[warp][2] = B;
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < W - 1; ++v)
      if (v < wr) y0 = fma(sh[w0 + v][1], y0, sh[w0 + v][2]);
  }
  double yi;
  {
    const double a2 = __shfl_up_sync(ALL, A, 1), b2 = __shfl_up_sync(ALL, B, 1);
    yi = lane ? fma(a2, y0, b2) : y0;
  }
#pragma unroll
  for (int k = 0; k < C; ++k) {
    y[k] = fma(-(k ? e[k - 1] : ep) * m[k], yi, y[k]);
    yi = y[k];
  }
  // back substitution: z_k = y_k - e_k m_k z_{k+1}
  A = 1.0;
  B = 0.0;
#pragma unroll
  for (int k = C - 1; k >= 0; --k) {
    const double a = -e[k] * m[k];
    B = fma(a, B, y[k]);
    A *= a;
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double a2 = __shfl_down_sync(ALL, A, d), b2 = __shfl_down_sync(ALL, B, d);
    if (lane + d < 32) {
      B = fma(A, b2, B);
      A *= a2;
    }
  }
  y0 = 0.0;
  if constexpr (W > 1) {
    __syncthreads();
    if (lane == 0) {
      sh[warp][1] = A;
      sh[warp][2] = B;
    }
    __syncthreads();
#pragma unroll
    for (int v = W - 1; v > 0; --v)
      if (v > wr) y0 = fma(sh[w0 + v][1], y0, sh[w0 + v][2]);
  }
  {
    const double a2 = __shfl_down_sync(ALL, A, 1), b2 = __shfl_down_sync(ALL, B, 1);
    yi = lane < 31 ? fma(a2, y0, b2) : y0;
  }
#pragma unroll
  for (int k = C - 1; k >= 0; --k) {
    y[k] = fma(-e[k] * m[k], yi, y[k]);
    yi = y[k];
  }
  if (null) {
    if constexpr (W > 1) {  // written before the scans' barriers
      sum = part = 0.0;
#pragma unroll
      for (int v = 0; v < W; ++v) {
        sum += sh[w0 + v][0];
        part += sh[w0 + v][3];
      }
    }
#pragma unroll
    for (int k = 0; k < C; ++k)
      if (s0 + k < n) y[k] -= fma(sum, __ldg(F.ng + s0 + k), part);
  }
  // cyclic systems: zh = y - (y_0 + cr y_{n-1}) g
  if (F.g) {
    double first = __shfl_sync(ALL, y[0], 0), last = 0.0;
#pragma unroll
    for (int k = 0; k < C; ++k) {
      const double v = __shfl_sync(ALL, y[k], ((n - 1) / C) & 31);
      if (k == (n - 1) % C) last = v;
    }
    if constexpr (W > 1) {
      __syncthreads();  // the null row's sums were read
      if (lane == 0) {
        sh[warp][0] = first;
        sh[warp][3] = last;
      }
      __syncthreads();
      first = sh[w0][0];
      last = sh[w0 + (n - 1) / (32 * C)][3];
    }
    if (row && !null) {
      const double *__restrict__ g = F.g + (size_t)b * n;
      const double c = first + __ldg(F.cr + b) * last;
#pragma unroll
      for (int k = 0; k < C; ++k)
        if (s0 + k < n) y[k] -= c * __ldg(g + s0 + k);
    }
  }
}

// Row b of the nm x n array F.t in place, by W warps of a block of 4
template <int W>
__device__ __forceinline__ void tri_row(const FdmD &F, int b, int wr, double (*sh)[4]) {
  constexpr int C = kTriChunk;
  const int n = F.n, s0 = (wr * 32 + (threadIdx.x & 31)) * C;
  const bool row = b < F.nm;
  double *__restrict__ w = F.t + (size_t)(row ? b : 0) * n;
  TriTab<C> T;
  double y[C];
#pragma unroll
  for (int k = 0; k < C; ++k) y[k] = (row && s0 + k < n) ? w[s0 + k] : 0.0;
  tri_tables<C>(F, b, s0, T);
  tri_solve<W, C>(F, b, wr, T, y, sh);
#pragma unroll
  for (int k = 0; k < C; ++k)
    if (row && s0 + k < n) w[s0 + k] = y[k];
}

}  // namespace ins2d
