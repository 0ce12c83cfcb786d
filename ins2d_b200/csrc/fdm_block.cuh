// Fast-diagonalization preconditioner applied by ONE thread block (the
// single-block PCG of small grids): the two products of fdm_apply, each split
// into 8 x 8 output fragments that the block's warps take in turn, every
// fragment a chain of FP64 MMAs (mma.sync m8n8k4 .f64) whose operands are
// read straight from memory, and the tridiagonal systems, a warp per system.
// Small grids only (kFdmBlockMaxN cells per direction): the operands stay in
// L1/L2.  The intermediates are written by the same kernel, so they are read
// with plain loads; the basis is read-only.
#pragma once

#include "fdm_tri.cuh"
#include "kernels.cuh"

namespace ins2d {

constexpr int kFdmBlockMaxN = 128;

__device__ __forceinline__ void fdm_block_mma(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// C (M x N) = op(A) op(B) (layouts as fdm.cu's gemm_tile).  AC / BC: A / B
// are read-only bases (read through the non-coherent cache).
template <bool TA, bool TB, bool AC, bool BC>
__device__ __forceinline__ void fdm_block_gemm(int M, int N, int K, const double *A, int lda, const double *B, int ldb,
                                               double *C, int ldc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int fm = (M + 7) / 8, fn = (N + 7) / 8;
  for (int f = warp; f < fm * fn; f += nw) {
    const int bm = (f / fn) * 8, bn = (f - (f / fn) * fn) * 8;
    const int m = bm + g, n = bn + g;
    double d0 = 0.0, d1 = 0.0;
    for (int k = 0; k < K; k += 4) {
      const int kk = k + t;
      double a = 0.0, b = 0.0;
      if (m < M && kk < K) {
        const double *pa = TA ? A + (size_t)kk * lda + m : A + (size_t)m * lda + kk;
        a = AC ? __ldg(pa) : *pa;
      }
      if (n < N && kk < K) {
        const double *pb = TB ? B + (size_t)n * ldb + kk : B + (size_t)kk * ldb + n;
        b = BC ? __ldg(pb) : *pb;
      }
      fdm_block_mma(d0, d1, a, b);
    }
    const int row = bm + g;
    if (row < M) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = bn + 2 * t + h;
        if (col < N) C[(size_t)row * ldc + col] = h ? d1 : d0;
      }
    }
  }
}

// z = A^+ r by the whole block; r must be complete (the caller synchronised
// after writing it); z is complete for every thread on return
__device__ __forceinline__ void fdm_apply_block(const FdmD &F, const double *r, double *z) {
  const int nm = F.nm, n = F.n, nw = blockDim.x >> 5, warp = threadIdx.x >> 5;
  if (F.xmodes)
    fdm_block_gemm<true, true, true, false>(nm, n, nm, F.Q, nm, r, nm, F.t, n);
  else
    fdm_block_gemm<true, false, true, false>(nm, n, nm, F.Q, nm, r, n, F.t, n);
  __syncthreads();
  for (int b = warp; b < nm; b += nw) tri_row<1>(F, b, 0, nullptr);
  __syncthreads();
  if (F.xmodes)
    fdm_block_gemm<true, true, false, true>(n, nm, nm, F.t, n, F.Q, nm, z, nm);
  else
    fdm_block_gemm<false, false, true, false>(nm, n, nm, F.Q, nm, F.t, n, z, n);
  __syncthreads();
}

}  // namespace ins2d
