// Fast-diagonalization preconditioner of the device PCG.
//
// The pressure matrix is separable, A = M Om^-1 G = -(diag(hy) (x) TX + TY (x)
// diag(hx)) (operator_divergence.m:208 with the 1D factors of setup.cpp).
// With the generalized eigenbasis of ONE direction, T_m Q = diag(h_m) Q Lam
// (Q' diag(h_m) Q = I, fdm_host.cpp), an application is
//   w = Q' r,   (T_s + lam_b diag(h_s)) zh_b = -w_b for every mode b,   z = Q zh
// (the null mode of a singular A left out): two dense FP64 products and a
// batch of tridiagonal solves.  Applied exactly this is the inverse on the
// range of A, so the PCG -- which keeps cg.F's control flow and stopping rule
// -- converges in one or two iterations.  Diagonalizing both directions
// instead costs four products.
//
// What bounds it: the FP64 tensor-core rate (mma.sync m8n8k4 .f64; FP64 has
// no tcgen05 kind) on grids of more than 512 cells per direction, and on
// smaller ones the number of output tiles and their serial K loop.  Hence
// 32 x 32 output tiles (257 x 301 cells: 90 tiles, 512^2: 256, for 148 SMs)
// and operand slabs copied to shared memory by cp.async, kStages - 1 ahead.
// One solve of one pass on B200, tiles of 64 x 64 / 64 x 32 / 32 x 32 with
// four warps / 32 x 32 with eight: 301 x 257 cells 128 / 114 / 99.0 / 98.6 us,
// 512^2 150 / 127 / 120 / 118 us, 1024^2 276 / 334 / 281 / 285 us; 2 slabs
// instead of 4: 512^2 129 us; slabs of depth 32: 121 us.
#include <algorithm>

#include "fdm_tri.cuh"
#include "ins2d.h"
#include "kernels.cuh"
#include "reduce.cuh"

namespace ins2d {

namespace {

constexpr int kBM = 32, kBN = 32, kBK = 16, kStages = 4;  // output tile, depth and number of operand slabs
constexpr int kWarpsM = 2, kWarpsN = 4, kThreads = 32 * kWarpsM * kWarpsN;
// a slab in shared memory is padded to rows of 4 mod 16 doubles, so that a
// warp's fragment loads (four consecutive rows by four consecutive columns
// per half warp) hit distinct banks, whichever of its two indices is the row
constexpr int kSlab = kBM * (kBK + 4) > kBK * (kBM + 4) ? kBM * (kBK + 4) : kBK * (kBM + 4);
static_assert(kBM == kBN, "one slab size for both operands");

__device__ __forceinline__ void dmma_884(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
// asynchronous copy of BYTES (8 or 16); the last BYTES - valid are zero-filled
template <int BYTES>
__device__ __forceinline__ void cp_async_fill(double *dst, const double *src, int valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(valid) : "memory");
}

// Copies one operand slab, V elements per copy: rows r0.. (NR) and columns
// l0.. (NL) of the R x L row-major operand A (ld), to S with pitch NL + 4;
// zero outside A.
template <int NR, int NL, int V>
__device__ __forceinline__ void load_slab(double *S, const double *__restrict__ A, int ld, int r0, int R, int l0,
                                          int L) {
  constexpr int PER = NL / V;
#pragma unroll
  for (int q = 0; q < (NR * PER) / kThreads; ++q) {
    const int e = threadIdx.x + kThreads * q;
    const int r = e / PER, l = (e % PER) * V;
    const int gr = r0 + r, gl = l0 + l;
    const int left = gr < R ? L - gl : 0;
    const int valid = left >= V ? V : (left > 0 ? left : 0);
    const double *src = valid > 0 ? A + (size_t)gr * ld + gl : A;
    cp_async_fill<8 * V>(S + r * (NL + 4) + l, src, 8 * valid);
  }
}
template <int NR, int NL>
__device__ __forceinline__ void load_slab(double *S, const double *__restrict__ A, int ld, int r0, int R, int l0,
                                          int L, bool v16) {
  if (v16)
    load_slab<NR, NL, 2>(S, A, ld, r0, R, l0, L);
  else
    load_slab<NR, NL, 1>(S, A, ld, r0, R, l0, L);
}

// One kBM x kBN tile (rows m0.., columns n0..) of C = op(A) op(B), op(A) M x K,
// op(B) K x N.  TA: A stored K x M (element (m,k) at A[k*lda + m]); else
// A[m*lda + k].  TB: B stored N x K; else K x N.  epi(row, column, value) for
// every element of C in range; sm: both operands' slabs.  Fragment layout of m8n8k4 .f64 (group
// g = lane / 4, t = lane % 4): A holds (row g, col t), B (row t, col g), C/D
// (row g, cols 2t, 2t+1).
template <bool TA, bool TB, class Epi>
__device__ __forceinline__ void gemm_tile(int M, int N, int K, const double *__restrict__ A, int lda,
                                          const double *__restrict__ B, int ldb, int m0, int n0, double *sm, Epi epi) {
  double *As = sm, *Bs = sm + kStages * kSlab;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  constexpr int WM = kBM / kWarpsM, WN = kBN / kWarpsN, NI = WM / 8, NJ = WN / 8;
  const int wm = (warp % kWarpsM) * WM, wn = (warp / kWarpsM) * WN;
  // 16-byte copies where every row starts on a 16-byte boundary
  const bool va = (lda & 1) == 0 && ((uintptr_t)A & 15) == 0, vb = (ldb & 1) == 0 && ((uintptr_t)B & 15) == 0;
  const int nk = (K + kBK - 1) / kBK;
  auto load = [&](int kt) {
    double *as = As + (kt % kStages) * kSlab, *bs = Bs + (kt % kStages) * kSlab;
    if (TA)
      load_slab<kBK, kBM>(as, A, lda, kt * kBK, K, m0, M, va);
    else
      load_slab<kBM, kBK>(as, A, lda, m0, M, kt * kBK, K, va);
    if (TB)
      load_slab<kBN, kBK>(bs, B, ldb, n0, N, kt * kBK, K, vb);
    else
      load_slab<kBK, kBN>(bs, B, ldb, kt * kBK, K, n0, N, vb);
  };
  double acc[NI][NJ][2] = {};
#pragma unroll
  for (int q = 0; q < kStages - 1; ++q) {
    if (q < nk) load(q);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // slab kt complete for every thread; slab kt - 1 read by every thread
    if (kt + kStages - 1 < nk) load(kt + kStages - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const double *as = As + (kt % kStages) * kSlab, *bs = Bs + (kt % kStages) * kSlab;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double a[NI], b[NJ];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int m = wm + 8 * i + g;
        a[i] = TA ? as[(kk + t) * (kBM + 4) + m] : as[m * (kBK + 4) + kk + t];
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int n = wn + 8 * j + g;
        b[j] = TB ? bs[n * (kBK + 4) + kk + t] : bs[(kk + t) * (kBN + 4) + n];
      }
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma_884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gm = m0 + wm + 8 * i + g, gn = n0 + wn + 8 * j + 2 * t + h;
        if (gm < M && gn < N) epi(gm, gn, acc[i][j][h]);
      }
}

// w = Q' r: rows = modes, columns = the unknowns of the systems
__device__ __forceinline__ void fdm_forward(const FdmD &F, const double *__restrict__ r, int m0, int n0, double *sm) {
  const int nm = F.nm, n = F.n;
  auto store = [&](int b, int i, double v) { F.t[(size_t)b * n + i] = v; };
  if (F.xmodes)  // r is n x nm (rows j = unknowns)
    gemm_tile<true, true>(nm, n, nm, F.Q, nm, r, nm, m0, n0, sm, store);
  else  // r is nm x n
    gemm_tile<true, false>(nm, n, nm, F.Q, nm, r, n, m0, n0, sm, store);
}
// z = Q zh, element (j, i) handed to epi(index, value)
template <class Epi>
__device__ __forceinline__ void fdm_backward(const FdmD &F, int m0, int n0, double *sm, Epi epi) {
  const int nm = F.nm, n = F.n, nx = F.nx;
  auto out = [&](int j, int i, double v) { epi((size_t)j * nx + i, v); };
  if (F.xmodes)
    gemm_tile<true, true>(n, nm, nm, F.t, n, F.Q, nm, m0, n0, sm, out);
  else
    gemm_tile<false, false>(nm, n, nm, F.Q, nm, F.t, n, m0, n0, sm, out);
}

__global__ void __launch_bounds__(kThreads) k_fdm_fwd(const __grid_constant__ FdmD F, const PcgWork W,
                                                      const double *__restrict__ f) {
  __shared__ __align__(16) double sm[2 * kStages * kSlab];
  if (*(volatile const int *)&W.sc->done) return;
  fdm_forward(F, W.sc->it == 0 ? f : W.r, blockIdx.y * kBM, blockIdx.x * kBN, sm);
}

// z = Q zh with r'z reduced in the same pass (deterministic, reduce.cuh)
__global__ void __launch_bounds__(kThreads) k_fdm_bwd(const __grid_constant__ FdmD F, const PcgWork W,
                                                      const double *__restrict__ f) {
  __shared__ __align__(16) double sm[2 * kStages * kSlab];
  if (*(volatile int *)&W.sc->done) return;
  const double *__restrict__ r = W.sc->it == 0 ? f : W.r;
  double q[1] = {0.0};
  const int ops[1] = {R_SUM};
  fdm_backward(F, blockIdx.y * kBM, blockIdx.x * kBN, sm, [&](size_t k, double v) {
    F.z[k] = v;
    q[0] += __ldg(r + k) * v;
  });
  RedScratch red;
  red.partials = W.partials;
  red.counter = &W.sc->counter;
  red.result = W.partials + (size_t)W.blocks * 8;
  red.max_blocks = W.blocks;
  double out[1];
  if (grid_reduce<1>(q, ops, red, out)) pcg_new_rz(W.sc, out[0]);
}

template <int W>
__global__ void __launch_bounds__(128) k_fdm_tri(const __grid_constant__ FdmD F, const int *__restrict__ done) {
  __shared__ double sh[4][4];
  if (*(volatile const int *)done) return;
  const int warp = threadIdx.x >> 5;
  tri_row<W>(F, blockIdx.x * (4 / W) + warp / W, warp % W, sh);
}

// the same for the members of an ensemble that still iterate
__global__ void __launch_bounds__(kThreads) k_fdm_fwd_ens(const FdmD *__restrict__ Fs, const int4 *__restrict__ tiles,
                                                          const EnsCg *__restrict__ cg) {
  __shared__ __align__(16) double sm[2 * kStages * kSlab];
  const int4 t = tiles[blockIdx.x];
  if (*(volatile const int *)&cg[t.x].done) return;
  const FdmD &F = Fs[t.x];
  const int m0 = t.y * kBM, n0 = t.z * kBN;
  if (m0 < F.nm && n0 < F.n) fdm_forward(F, cg[t.x].it == 0 ? F.f : F.r, m0, n0, sm);
}
__global__ void __launch_bounds__(kThreads) k_fdm_bwd_ens(const FdmD *__restrict__ Fs, const int4 *__restrict__ tiles,
                                                          EnsCg *__restrict__ cg) {
  __shared__ __align__(16) double sm[2 * kStages * kSlab];
  const int4 t = tiles[blockIdx.x];
  EnsCg &C = cg[t.x];
  if (*(volatile const int *)&C.done) return;
  const FdmD &F = Fs[t.x];
  const int m0 = t.y * kBM, n0 = t.z * kBN;
  if (m0 >= F.ny || n0 >= F.nx) return;
  const double *__restrict__ r = C.it == 0 ? F.f : F.r;
  double q[1] = {0.0};
  const int ops[1] = {R_SUM};
  fdm_backward(F, m0, n0, sm, [&](size_t k, double v) {
    F.z[k] = v;
    q[0] += __ldg(r + k) * v;
  });
  const int tx = (F.nx + kBN - 1) / kBN, nb = tx * ((F.ny + kBM - 1) / kBM);
  RedScratch red;
  red.partials = C.part;
  red.counter = &C.ticket;
  red.result = C.part + nb;
  double out[1];
  if (grid_reduce_at<1>(q, ops, red, out, t.y * tx + t.z, nb)) {
    if (!isfinite(out[0])) {
      C.status = INS2D_ENONFINITE;  // the member's update ends its solve
      C.beta = 0.0;
    } else {
      C.beta = C.it == 0 ? 0.0 : out[0] / C.rz;
      C.rz = out[0];
    }
  }
}
template <int W>
__global__ void __launch_bounds__(128) k_fdm_tri_ens(const FdmD *__restrict__ Fs, const int2 *__restrict__ rows,
                                                     const EnsCg *__restrict__ cg) {
  __shared__ double sh[4][4];
  const int2 t = rows[blockIdx.x];
  if (*(volatile const int *)&cg[t.x].done) return;
  const int warp = threadIdx.x >> 5;
  tri_row<W>(Fs[t.x], t.y + warp / W, warp % W, sh);
}

int row_warps(int n) { return n <= 32 * kTriChunk ? 1 : (n <= 64 * kTriChunk ? 2 : 4); }
static_assert(4 * 32 * kTriChunk >= 1024, "four warps hold the longest row (kFdmMaxN)");

template <int W>
void launch_tri(const FdmD &F, const int *done, cudaStream_t s) {
  k_fdm_tri<W><<<(F.nm + 4 / W - 1) / (4 / W), 128, 0, s>>>(F, done);
}

}  // namespace

void fdm_apply(const FdmD &F, const PcgWork &W, const double *f, cudaStream_t s) {
  const int *done = &W.sc->done;
  k_fdm_fwd<<<dim3((F.n + kBN - 1) / kBN, (F.nm + kBM - 1) / kBM), kThreads, 0, s>>>(F, W, f);
  const int w = row_warps(F.n);
  if (w == 1)
    launch_tri<1>(F, done, s);
  else if (w == 2)
    launch_tri<2>(F, done, s);
  else
    launch_tri<4>(F, done, s);
  k_fdm_bwd<<<dim3((F.nx + kBN - 1) / kBN, (F.ny + kBM - 1) / kBM), kThreads, 0, s>>>(F, W, f);
}

void fdm_ens_lists(const std::vector<FdmD> &F, const std::vector<int> &order, EnsFdmPlan &pl, std::vector<int4> &tiles,
                   std::vector<int2> &rows) {
  int nmax = 0;
  for (const FdmD &f : F) nmax = std::max(nmax, f.n);
  pl.warps = row_warps(nmax);
  // one list for both products: the forward one's nm x n and the backward
  // one's ny x nx tiles (a tile outside a product's range returns)
  for (int m : order) {
    const int M = std::max(F[m].nm, F[m].ny), N = std::max(F[m].n, F[m].nx);
    for (int bi = 0; bi < (M + kBM - 1) / kBM; ++bi)
      for (int bj = 0; bj < (N + kBN - 1) / kBN; ++bj) tiles.push_back(make_int4(m, bi, bj, 0));
    for (int b = 0; b < F[m].nm; b += 4 / pl.warps) rows.push_back(make_int2(m, b));
  }
  pl.ntiles = (int)tiles.size();
  pl.nrows = (int)rows.size();
}

void fdm_apply_ens(const EnsFdmPlan &pl, EnsCg *cg, cudaStream_t s) {
  if (pl.ntiles <= 0) return;
  k_fdm_fwd_ens<<<pl.ntiles, kThreads, 0, s>>>(pl.F, pl.tiles, cg);
  if (pl.warps == 1)
    k_fdm_tri_ens<1><<<pl.nrows, 128, 0, s>>>(pl.F, pl.rows, cg);
  else if (pl.warps == 2)
    k_fdm_tri_ens<2><<<pl.nrows, 128, 0, s>>>(pl.F, pl.rows, cg);
  else
    k_fdm_tri_ens<4><<<pl.nrows, 128, 0, s>>>(pl.F, pl.rows, cg);
  k_fdm_bwd_ens<<<pl.ntiles, kThreads, 0, s>>>(pl.F, pl.tiles, cg);
}

}  // namespace ins2d
