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
// no tcgen05 kind) on grids of 512 cells per direction and more, and on
// smaller ones the number of output tiles (fewer than SMs) and their serial
// K loop.  So the tile shape follows the grid (tile_config), and operand
// slabs are copied to shared memory by cp.async, kStages - 1 slabs ahead.
#include <algorithm>

#include "fdm_tri.cuh"
#include "ins2d.h"
#include "kernels.cuh"
#include "reduce.cuh"

namespace ins2d {

namespace {

constexpr int kBK = 16;       // depth of an operand slab
constexpr int kThreads = 128;  // 2 x 2 warps per output tile

// tile shapes; their shared memory: kStages slabs of both operands, each
// padded to rows of 4 mod 16 doubles, so that a warp's fragment loads (four
// consecutive rows by four consecutive columns per half warp) hit distinct banks
template <int CFG>
struct Tile;
template <>
struct Tile<0> {
  static constexpr int BM = 64, BN = 64, STAGES = 3;
};
template <>
struct Tile<1> {
  static constexpr int BM = 64, BN = 32, STAGES = 4;
};
template <>
struct Tile<2> {
  static constexpr int BM = 32, BN = 32, STAGES = 4;
};
__host__ __device__ constexpr int slab(int bmn) {
  const int kmajor = kBK * (bmn + 4), mmajor = bmn * (kBK + 4);
  return kmajor > mmajor ? kmajor : mmajor;
}
template <int CFG>
constexpr int tile_smem() {
  return Tile<CFG>::STAGES * (slab(Tile<CFG>::BM) + slab(Tile<CFG>::BN)) * (int)sizeof(double);
}

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

// Copies one operand slab: rows of `len` contiguous elements.  The operand is
// stored R x L row-major (ld); the slab takes R0.. (NR of them) by L0.. (NL),
// to S with pitch NL + 4.  V elements per copy.
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

// One BM x BN tile (rows m0.., columns n0..) of C = op(A) op(B), op(A) M x K,
// op(B) K x N.  TA: A stored K x M (element (m,k) at A[k*lda + m]); else
// A[m*lda + k].  TB: B stored N x K; else K x N.  epi(row, column, value) for
// every element of C in range.  Fragment layout of m8n8k4 .f64 (group
// g = lane / 4, t = lane % 4): A holds (row g, col t), B (row t, col g), C/D
// (row g, cols 2t, 2t+1).
template <int CFG, bool TA, bool TB, class Epi>
__device__ __forceinline__ void gemm_tile(int M, int N, int K, const double *__restrict__ A, int lda,
                                          const double *__restrict__ B, int ldb, int m0, int n0, Epi epi) {
  constexpr int BM = Tile<CFG>::BM, BN = Tile<CFG>::BN, ST = Tile<CFG>::STAGES;
  constexpr int SA = slab(BM), SB = slab(BN);
  extern __shared__ __align__(16) double smem[];
  double *As = smem, *Bs = smem + ST * SA;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  constexpr int WM = BM / 2, WN = BN / 2, NI = WM / 8, NJ = WN / 8;
  const int wm = (warp & 1) * WM, wn = (warp >> 1) * WN;
  // 16-byte copies where every row starts on a 16-byte boundary
  const bool va = (lda & 1) == 0 && ((uintptr_t)A & 15) == 0, vb = (ldb & 1) == 0 && ((uintptr_t)B & 15) == 0;
  const int nk = (K + kBK - 1) / kBK;
  auto load = [&](int kt) {
    double *as = As + (kt % ST) * SA, *bs = Bs + (kt % ST) * SB;
    if (TA)
      load_slab<kBK, BM>(as, A, lda, kt * kBK, K, m0, M, va);
    else
      load_slab<BM, kBK>(as, A, lda, m0, M, kt * kBK, K, va);
    if (TB)
      load_slab<BN, kBK>(bs, B, ldb, n0, N, kt * kBK, K, vb);
    else
      load_slab<kBK, BN>(bs, B, ldb, kt * kBK, K, n0, N, vb);
  };
  double acc[NI][NJ][2] = {};
#pragma unroll
  for (int q = 0; q < ST - 1; ++q) {
    if (q < nk) load(q);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");
    __syncthreads();  // slab kt complete for every thread; slab kt - 1 read by every thread
    if (kt + ST - 1 < nk) load(kt + ST - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const double *as = As + (kt % ST) * SA, *bs = Bs + (kt % ST) * SB;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double a[NI], b[NJ];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int m = wm + 8 * i + g;
        a[i] = TA ? as[(kk + t) * (BM + 4) + m] : as[m * (kBK + 4) + kk + t];
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int n = wn + 8 * j + g;
        b[j] = TB ? bs[n * (kBK + 4) + kk + t] : bs[(kk + t) * (BN + 4) + n];
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
template <int CFG>
__device__ __forceinline__ void fdm_forward(const FdmD &F, const double *__restrict__ r, int m0, int n0) {
  const int nm = F.nm, n = F.n;
  auto store = [&](int b, int i, double v) { F.t[(size_t)b * n + i] = v; };
  if (F.xmodes)  // r is n x nm (rows j = unknowns)
    gemm_tile<CFG, true, true>(nm, n, nm, F.Q, nm, r, nm, m0, n0, store);
  else  // r is nm x n
    gemm_tile<CFG, true, false>(nm, n, nm, F.Q, nm, r, n, m0, n0, store);
}
// z = Q zh, element (j, i) handed to epi(index, value)
template <int CFG, class Epi>
__device__ __forceinline__ void fdm_backward(const FdmD &F, int m0, int n0, Epi epi) {
  const int nm = F.nm, n = F.n, nx = F.nx;
  auto out = [&](int j, int i, double v) { epi((size_t)j * nx + i, v); };
  if (F.xmodes)
    gemm_tile<CFG, true, true>(n, nm, nm, F.t, n, F.Q, nm, m0, n0, out);
  else
    gemm_tile<CFG, false, false>(nm, n, nm, F.Q, nm, F.t, n, m0, n0, out);
}

template <int CFG>
__global__ void __launch_bounds__(kThreads) k_fdm_fwd(const __grid_constant__ FdmD F, const PcgWork W,
                                                      const double *__restrict__ f) {
  if (*(volatile const int *)&W.sc->done) return;
  fdm_forward<CFG>(F, W.sc->it == 0 ? f : W.r, blockIdx.y * Tile<CFG>::BM, blockIdx.x * Tile<CFG>::BN);
}

// z = Q zh with r'z reduced in the same pass (deterministic, reduce.cuh)
template <int CFG>
__global__ void __launch_bounds__(kThreads) k_fdm_bwd(const __grid_constant__ FdmD F, const PcgWork W,
                                                      const double *__restrict__ f) {
  if (*(volatile int *)&W.sc->done) return;
  const double *__restrict__ r = W.sc->it == 0 ? f : W.r;
  double q[1] = {0.0};
  const int ops[1] = {R_SUM};
  fdm_backward<CFG>(F, blockIdx.y * Tile<CFG>::BM, blockIdx.x * Tile<CFG>::BN, [&](size_t k, double v) {
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
template <int CFG>
__global__ void __launch_bounds__(kThreads) k_fdm_fwd_ens(const FdmD *__restrict__ Fs, const int4 *__restrict__ tiles,
                                                          const EnsCg *__restrict__ cg) {
  const int4 t = tiles[blockIdx.x];
  if (*(volatile const int *)&cg[t.x].done) return;
  const FdmD &F = Fs[t.x];
  const int m0 = t.y * Tile<CFG>::BM, n0 = t.z * Tile<CFG>::BN;
  if (m0 < F.nm && n0 < F.n) fdm_forward<CFG>(F, F.r, m0, n0);
}
template <int CFG>
__global__ void __launch_bounds__(kThreads) k_fdm_bwd_ens(const FdmD *__restrict__ Fs, const int4 *__restrict__ tiles,
                                                          const EnsCg *__restrict__ cg) {
  const int4 t = tiles[blockIdx.x];
  if (*(volatile const int *)&cg[t.x].done) return;
  const FdmD &F = Fs[t.x];
  const int m0 = t.y * Tile<CFG>::BM, n0 = t.z * Tile<CFG>::BN;
  if (m0 < F.ny && n0 < F.nx) fdm_backward<CFG>(F, m0, n0, [&](size_t k, double v) { F.z[k] = v; });
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

// Tile shape: the one with the least work on the busiest SM, tiles of one
// launch spread evenly; the larger one on a tie (it reads its operands fewer
// times).
int tile_config(long long t64, long long t6432, long long t32, int nsm) {
  const long long w0 = ((t64 + nsm - 1) / nsm) * 4, w1 = ((t6432 + nsm - 1) / nsm) * 2, w2 = (t32 + nsm - 1) / nsm;
  return w0 <= w1 && w0 <= w2 ? 0 : (w1 <= w2 ? 1 : 2);
}
long long tiles_of(long long M, long long N, int bm, int bn) { return ((M + bm - 1) / bm) * ((N + bn - 1) / bn); }
int row_warps(int n) { return n <= 32 * kTriChunk ? 1 : (n <= 64 * kTriChunk ? 2 : 4); }
static_assert(4 * 32 * kTriChunk >= 1024, "four warps hold the longest row (kFdmMaxN)");

template <int CFG>
void launch_fwd(const FdmD &F, const PcgWork &W, const double *f, cudaStream_t s) {
  const dim3 g((F.n + Tile<CFG>::BN - 1) / Tile<CFG>::BN, (F.nm + Tile<CFG>::BM - 1) / Tile<CFG>::BM);
  k_fdm_fwd<CFG><<<g, kThreads, tile_smem<CFG>(), s>>>(F, W, f);
}
template <int CFG>
void launch_bwd(const FdmD &F, const PcgWork &W, const double *f, cudaStream_t s) {
  const dim3 g((F.nx + Tile<CFG>::BN - 1) / Tile<CFG>::BN, (F.ny + Tile<CFG>::BM - 1) / Tile<CFG>::BM);
  k_fdm_bwd<CFG><<<g, kThreads, tile_smem<CFG>(), s>>>(F, W, f);
}
template <int W>
void launch_tri(const FdmD &F, const int *done, cudaStream_t s) {
  k_fdm_tri<W><<<(F.nm + 4 / W - 1) / (4 / W), 128, 0, s>>>(F, done);
}

}  // namespace

cudaError_t fdm_prepare() {
  cudaError_t first = cudaSuccess;
  auto opt_in = [&](const void *k, int bytes) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (first == cudaSuccess) first = e;
  };
#define INS2D_FDM_OPT_IN(C)                                   \
  opt_in((const void *)k_fdm_fwd<C>, tile_smem<C>());         \
  opt_in((const void *)k_fdm_bwd<C>, tile_smem<C>());         \
  opt_in((const void *)k_fdm_fwd_ens<C>, tile_smem<C>());     \
  opt_in((const void *)k_fdm_bwd_ens<C>, tile_smem<C>());
  INS2D_FDM_OPT_IN(0)
  INS2D_FDM_OPT_IN(1)
  INS2D_FDM_OPT_IN(2)
#undef INS2D_FDM_OPT_IN
  return first;
}

void fdm_apply(const FdmD &F, const PcgWork &W, const double *f, cudaStream_t s) {
  const int *done = &W.sc->done;
  const int cfg = tile_config(tiles_of(F.ny, F.nx, 64, 64),
                              std::min(tiles_of(F.ny, F.nx, 64, 32), tiles_of(F.nx, F.ny, 64, 32)),
                              tiles_of(F.ny, F.nx, 32, 32), F.nsm);
  if (cfg == 0)
    launch_fwd<0>(F, W, f, s);
  else if (cfg == 1)
    launch_fwd<1>(F, W, f, s);
  else
    launch_fwd<2>(F, W, f, s);
  const int w = row_warps(F.n);
  if (w == 1)
    launch_tri<1>(F, done, s);
  else if (w == 2)
    launch_tri<2>(F, done, s);
  else
    launch_tri<4>(F, done, s);
  if (cfg == 0)
    launch_bwd<0>(F, W, f, s);
  else if (cfg == 1)
    launch_bwd<1>(F, W, f, s);
  else
    launch_bwd<2>(F, W, f, s);
}

void fdm_ens_lists(const std::vector<FdmD> &F, const std::vector<int> &order, int nsm, EnsFdmPlan &pl,
                   std::vector<int4> &tiles, std::vector<int2> &rows) {
  long long t0 = 0, t1 = 0, t2 = 0;
  int nmax = 0;
  for (const FdmD &f : F) {
    t0 += tiles_of(f.nm, f.n, 64, 64);
    t1 += tiles_of(f.nm, f.n, 64, 32);
    t2 += tiles_of(f.nm, f.n, 32, 32);
    nmax = std::max(nmax, f.n);
  }
  pl.cfg = tile_config(t0, t1, t2, nsm);
  pl.warps = row_warps(nmax);
  const int bm = pl.cfg == 2 ? 32 : 64, bn = pl.cfg == 0 ? 64 : 32;
  // one list for both products: the forward one's nm x n and the backward
  // one's ny x nx tiles (a tile outside a product's range returns)
  for (int m : order) {
    const int M = std::max(F[m].nm, F[m].ny), N = std::max(F[m].n, F[m].nx);
    for (int bi = 0; bi < (M + bm - 1) / bm; ++bi)
      for (int bj = 0; bj < (N + bn - 1) / bn; ++bj) tiles.push_back(make_int4(m, bi, bj, 0));
    for (int b = 0; b < F[m].nm; b += 4 / pl.warps) rows.push_back(make_int2(m, b));
  }
  pl.ntiles = (int)tiles.size();
  pl.nrows = (int)rows.size();
}

void fdm_apply_ens(const EnsFdmPlan &pl, const EnsCg *cg, cudaStream_t s) {
  if (pl.ntiles <= 0) return;
  if (pl.cfg == 0)
    k_fdm_fwd_ens<0><<<pl.ntiles, kThreads, tile_smem<0>(), s>>>(pl.F, pl.tiles, cg);
  else if (pl.cfg == 1)
    k_fdm_fwd_ens<1><<<pl.ntiles, kThreads, tile_smem<1>(), s>>>(pl.F, pl.tiles, cg);
  else
    k_fdm_fwd_ens<2><<<pl.ntiles, kThreads, tile_smem<2>(), s>>>(pl.F, pl.tiles, cg);
  if (pl.warps == 1)
    k_fdm_tri_ens<1><<<pl.nrows, 128, 0, s>>>(pl.F, pl.rows, cg);
  else if (pl.warps == 2)
    k_fdm_tri_ens<2><<<pl.nrows, 128, 0, s>>>(pl.F, pl.rows, cg);
  else
    k_fdm_tri_ens<4><<<pl.nrows, 128, 0, s>>>(pl.F, pl.rows, cg);
  if (pl.cfg == 0)
    k_fdm_bwd_ens<0><<<pl.ntiles, kThreads, tile_smem<0>(), s>>>(pl.F, pl.tiles, cg);
  else if (pl.cfg == 1)
    k_fdm_bwd_ens<1><<<pl.ntiles, kThreads, tile_smem<1>(), s>>>(pl.F, pl.tiles, cg);
  else
    k_fdm_bwd_ens<2><<<pl.ntiles, kThreads, tile_smem<2>(), s>>>(pl.F, pl.tiles, cg);
}

}  // namespace ins2d
