// The whole fast-diagonalization PCG solve of a small grid (at most
// kFdmClusterMaxN cells per direction) in one launch of one thread-block
// cluster, optionally with the divergence that gives its right-hand side.
//
// Such a solve is bound by latency: two products of at most 128^3 operations,
// nm scans, one stencil and four reductions, each waiting for the one before.
// So every array lives in shared memory.  The eight blocks split the systems'
// direction s: block c holds r, p, x, q, z of the cells (m, s), all m and its
// slice of s, and computes its columns of both products from a shared-memory
// copy of the basis (read through L1 where it does not fit).  The tridiagonal
// systems run along s, so the blocks exchange the transformed residual and
// the solution through distributed shared memory (block c solves its slice of
// the modes b, a warp per system).  A pass takes five cluster barriers.
// Measured on B200 against one thread block working from L1/L2 and a separate
// divergence launch: RK44 step of the 64^2 cavity (four solves) 0.228 ->
// 0.117 ms.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>

#include "fdm_tri.cuh"
#include "ins2d.h"
#include "kernels.cuh"
#include "reduce.cuh"

namespace cg = cooperative_groups;

namespace ins2d {

namespace {

constexpr int kC = 8;             // blocks of the cluster
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTriC = kFdmClusterMaxN / 32;  // unknowns per lane of a system
constexpr int kSmemMax = 226 * 1024;  // dynamic; the reductions' slots are static

// sizes of one solve
struct Geo {
  int nm, n;      // modes, unknowns per system
  int ns, nb;     // systems' unknowns and modes per block (the last blocks may hold fewer or none)
  int ld;         // pitch of the cell arrays: ns rounded up to 8, plus 4 (4 or 12 mod 16: conflict-free fragments)
  int ldt;        // pitch of the rows of systems
  int mp;         // modes rounded up to 8
  int qp;         // pitch of the basis (4 mod 16), 0: not in shared memory
};
__host__ __device__ inline size_t cells(const Geo &g) { return (size_t)g.mp * g.ld; }
__host__ __device__ inline size_t smem_doubles(const Geo &g) {
  return 6 * cells(g) + (size_t)g.nb * g.ldt + 2 * (size_t)g.mp + (size_t)g.mp * g.qp;
}
Geo make_geo(const FdmD &F) {
  Geo g;
  g.nm = F.nm;
  g.n = F.n;
  g.ns = (F.n + kC - 1) / kC;
  g.nb = (F.nm + kC - 1) / kC;
  g.ld = ((g.ns + 7) / 8) * 8 + 4;
  g.ldt = F.n + 1;
  g.mp = ((F.nm + 7) / 8) * 8;
  g.qp = ((F.nm + 15) / 16) * 16 + 4;
  if (smem_doubles(g) * sizeof(double) > kSmemMax) g.qp = 0;
  return g;
}

__device__ __forceinline__ void mma884(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// C = op(Q) B on 8 x 8 fragments taken by the block's warps in turn; B: cell
// array (rows k, pitch ld), zero-padded rows and columns; TRANS: op(Q)(i, k) =
// Q(k, i), else Q(i, k); epi(row, column, value) for every fragment element.
// Two accumulator pairs halve the chain of dependent MMAs.
template <bool TRANS, class QF, class Epi>
__device__ __forceinline__ void product(const Geo &g, const QF &q, const double *B, Epi epi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gr = lane >> 2, t = lane & 3;
  const int tn = g.ld >> 3, tiles = (g.mp >> 3) * tn;  // ld = 8 tn + 4
  for (int f = warp; f < tiles; f += kWarps) {
    const int bm = (f / tn) * 8, bn = (f % tn) * 8;
    double c0 = 0.0, c1 = 0.0, d0 = 0.0, d1 = 0.0;
    const double *b = B + (size_t)t * g.ld + bn + gr;
#pragma unroll 4
    for (int k = 0; k < g.mp; k += 8) {
      const double a0 = TRANS ? q(k + t, bm + gr) : q(bm + gr, k + t);
      const double a1 = TRANS ? q(k + 4 + t, bm + gr) : q(bm + gr, k + 4 + t);
      mma884(c0, c1, a0, b[(size_t)k * g.ld]);
      mma884(d0, d1, a1, b[(size_t)(k + 4) * g.ld]);
    }
    epi(bm + gr, bn + 2 * t, c0 + d0);
    epi(bm + gr, bn + 2 * t + 1, c1 + d1);
  }
}

// Sum / max / min of NQ values over the cluster: every block's partial to
// every block, a cluster barrier, and the same ordered combination in every
// thread.  slot alternates between two buffers.
template <int NQ>
__device__ __forceinline__ void cluster_reduce(cg::cluster_group &cl, double (&v)[NQ], const int (&ops)[NQ],
                                               double (*warp_part)[4], double (*part)[kC][4], int &slot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[q] = red_combine(v[q], __shfl_xor_sync(0xffffffffu, v[q], off), ops[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) warp_part[warp][q] = v[q];
  __syncthreads();
  if (threadIdx.x < kC) {
    double *dst = cl.map_shared_rank(&part[slot][cl.block_rank()][0], threadIdx.x);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double a = warp_part[0][q];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) a = red_combine(a, warp_part[w][q], ops[q]);
      dst[q] = a;
    }
  }
  cl.sync();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double a = part[slot][0][q];
#pragma unroll
    for (int c = 1; c < kC; ++c) a = red_combine(a, part[slot][c][q], ops[q]);
    v[q] = a;
  }
  slot ^= 1;
}

// QS: the basis in shared memory
template <bool QS>
__global__ void __cluster_dims__(kC, 1, 1) __launch_bounds__(kThreads, 1)
    k_pcg_cluster(const __grid_constant__ DevOps P, const __grid_constant__ FdmD F, const PcgWork W, const Geo g,
                  const __grid_constant__ SolveSrc src, double *__restrict__ dp, double tol2, long long maxit,
                  int accumulate, SolveAccum *acc) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double warp_part[kWarps][4];
  __shared__ double part[2][kC][4];
  cg::cluster_group cl = cg::this_cluster();
  const int c = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nm = g.nm, n = g.n, ld = g.ld;
  const int s0 = c * g.ns, s1 = min(s0 + g.ns, n), nl = max(s1 - s0, 0);  // this block's slice
  const size_t nc = cells(g);
  double *r = sm, *p = r + nc, *x = p + nc, *q = x + nc, *z = q + nc, *zh = z + nc;
  double *rows = zh + nc, *pl = rows + (size_t)g.nb * g.ldt, *pr = pl + g.mp, *Qs = pr + g.mp;
  int slot = 0;
  cl.sync();  // every block runs before any other writes to its shared memory
  // zero padding of the products' right operands
  for (size_t k = tid; k < nc; k += kThreads) {
    r[k] = 0.0;
    zh[k] = 0.0;
  }
  if (QS)
    for (int k = tid; k < g.mp * g.mp; k += kThreads) {
      const int i = k / g.mp, b = k - i * g.mp;
      Qs[(size_t)i * g.qp + b] = (i < nm && b < nm) ? __ldg(F.Q + (size_t)i * nm + b) : 0.0;
    }
  auto basis = [&](int i, int b) -> double {
    if constexpr (QS)
      return Qs[(size_t)i * g.qp + b];
    else
      return (i < nm && b < nm) ? __ldg(F.Q + (size_t)i * nm + b) : 0.0;
  };
  // this warp's systems: rows warp, warp + 8 of the block's slice of modes
  constexpr int RW = (kFdmClusterMaxN / kC + kWarps - 1) / kWarps;
  TriTab<kTriC> tab[RW];
#pragma unroll
  for (int u = 0; u < RW; ++u) {
    const int lb = warp + u * kWarps, b = c * g.nb + lb;
    tri_tables<kTriC>(F, lb < g.nb ? b : F.nm, lane * kTriC, tab[u]);
  }
  __syncthreads();
  // cell l of the slice: (m, s), x fastest in memory
  auto cell = [&](int l, int &m, int &sl) {
    if (F.xmodes) {
      sl = l / nm;
      m = l - sl * nm;
    } else {
      m = l / nl;
      sl = l - m * nl;
    }
  };
  const int ncell = nm * nl;
  // right-hand side (cg.F:207-229 with x_in = 0)
  double a2[2] = {0.0, 0.0};
  const int op2[2] = {R_SUM, R_MAX};
  for (int l = tid; l < ncell; l += kThreads) {
    int m, sl;
    cell(l, m, sl);
    const int i = F.xmodes ? m : s0 + sl, j = F.xmodes ? s0 + sl : m;
    const double f = src.mode == 0   ? src.f[(size_t)j * P.Npx + i]
                     : src.mode == 1 ? div_cell_f(P, WPlain{src.f}, src.alpha, src.beta, src.gamma, i, j)
                                     : div_cell_f(P, src.ws, src.alpha, src.beta, src.gamma, i, j);
    r[m * ld + sl] = f;
    a2[0] += f * f;
    a2[1] = fmax(a2[1], fabs(f));
  }
  cluster_reduce<2>(cl, a2, op2, warp_part, part, slot);
  const double rr0 = a2[0];
  double rz = 0.0, rr = 0.0, maxx = 0.0, minx = 0.0, maxres = 0.0;
  long long it = 0;
  int status = 0;
  bool done = (a2[1] < 1e-14 || rr0 <= tol2);  // pressure_poisson.m:33-38, cg.F:222-227
  if (!isfinite(rr0)) {
    status = INS2D_ENONFINITE;
    done = true;
  }
  const Tab &Tm = F.xmodes ? P.TX : P.TY, &Ts = F.xmodes ? P.TY : P.TX;
  const double *hm = F.xmodes ? P.hx : P.hy, *hs = F.xmodes ? P.hy : P.hx;
  const int op1[1] = {R_SUM};
  // the loop's exits are taken by all blocks alike: every condition comes
  // from a cluster-wide reduction
  while (!done) {
    // w = Q' r, each row to the block that solves it
    product<true>(g, basis, r, [&](int b, int sl, double v) {
      if (b < nm && sl < nl) {
        const int o = b / g.nb;
        cl.map_shared_rank(rows, o)[(size_t)(b - o * g.nb) * g.ldt + s0 + sl] = v;
      }
    });
    cl.sync();
#pragma unroll
    for (int u = 0; u < RW; ++u) {
      const int lb = warp + u * kWarps, b = lb < g.nb ? c * g.nb + lb : F.nm;
      if (b >= nm) continue;
      const double *w = rows + (size_t)lb * g.ldt;
      double y[kTriC];
#pragma unroll
      for (int k = 0; k < kTriC; ++k) y[k] = lane * kTriC + k < n ? w[lane * kTriC + k] : 0.0;
      tri_solve<1, kTriC>(F, b, 0, tab[u], y, nullptr);
#pragma unroll
      for (int k = 0; k < kTriC; ++k) {
        const int s = lane * kTriC + k;
        if (s < n) {
          const int o = s / g.ns;
          cl.map_shared_rank(zh, o)[(size_t)b * ld + s - o * g.ns] = y[k];
        }
      }
    }
    cl.sync();
    double a1[1] = {0.0};
    product<false>(g, basis, zh, [&](int m, int sl, double v) {
      if (m < nm && sl < nl) {
        z[m * ld + sl] = v;
        a1[0] += r[m * ld + sl] * v;
      }
    });
    cluster_reduce<1>(cl, a1, op1, warp_part, part, slot);
    if (!isfinite(a1[0])) {
      status = INS2D_ENONFINITE;
      break;
    }
    const bool first = it == 0;
    const double beta = first ? 0.0 : a1[0] / rz;
    rz = a1[0];
    // p = z + beta p, with the neighbouring columns' (kept in pl, pr)
    for (int l = tid; l < ncell; l += kThreads) {
      int m, sl;
      cell(l, m, sl);
      const int k = m * ld + sl;
      p[k] = first ? z[k] : z[k] + beta * p[k];
    }
    const int sL = s0 > 0 ? s0 - 1 : n - 1, sR = s1 < n ? s1 : 0;  // wrapped: used by cyclic rows only
    for (int l = tid; l < 2 * nm && nl > 0; l += kThreads) {
      const int m = l % nm;
      const bool left = l < nm;
      const int s = left ? sL : sR, o = s / g.ns;
      const double zv = cl.map_shared_rank(z, o)[(size_t)m * ld + s - o * g.ns];
      double &h = (left ? pl : pr)[m];
      h = first ? zv : zv + beta * h;
    }
    __syncthreads();
    // q = A p, p'q
    a1[0] = 0.0;
    for (int l = tid; l < ncell; l += kThreads) {
      int m, sl;
      cell(l, m, sl);
      const int s = s0 + sl;
      const int32_t *cm = Tm.c + kT * m, *cs = Ts.c + kT * s;
      const double *wm = Tm.w + kT * m, *ws = Ts.w + kT * s;
      double tm = 0.0, ts = 0.0;
#pragma unroll
      for (int k = 0; k < kT; ++k) {
        tm += __ldg(wm + k) * p[__ldg(cm + k) * ld + sl];
        const int sc = __ldg(cs + k);
        const double wv = __ldg(ws + k);
        const double pv = sc >= s0 && sc < s1 ? p[m * ld + sc - s0] : (sc == sL ? pl[m] : pr[m]);
        if (wv != 0.0) ts += wv * pv;
      }
      const double aq = -(__ldg(hs + s) * tm + __ldg(hm + m) * ts);
      q[m * ld + sl] = aq;
      a1[0] += p[m * ld + sl] * aq;
    }
    cluster_reduce<1>(cl, a1, op1, warp_part, part, slot);
    const double pq = a1[0];
    if (!isfinite(pq)) {
      status = INS2D_ENONFINITE;
      break;
    }
    if (pq == 0.0) {
      status = INS2D_EBREAKDOWN;
      break;
    }
    const double alpha = rz / pq;
    double a4[4] = {0.0, -DBL_MAX, DBL_MAX, 0.0};
    const int op4[4] = {R_SUM, R_MAX, R_MIN, R_MAX};
    for (int l = tid; l < ncell; l += kThreads) {
      int m, sl;
      cell(l, m, sl);
      const int k = m * ld + sl;
      const double xv = (first ? 0.0 : x[k]) + alpha * p[k];
      const double rv = r[k] - alpha * q[k];
      x[k] = xv;
      r[k] = rv;
      a4[0] += rv * rv;
      a4[1] = fmax(a4[1], xv);
      a4[2] = fmin(a4[2], xv);
      a4[3] = fmax(a4[3], fabs(rv));
    }
    cluster_reduce<4>(cl, a4, op4, warp_part, part, slot);
    ++it;
    rr = a4[0] / rr0;
    maxx = a4[1];
    minx = a4[2];
    maxres = a4[3];
    if (!isfinite(rr)) {
      status = INS2D_ENONFINITE;
      break;
    }
    if (rr <= tol2) break;
    if (it >= maxit) {
      status = INS2D_ENOTCONV;
      break;
    }
  }
  if (status == 0)
    for (int l = tid; l < ncell; l += kThreads) {
      int m, sl;
      cell(l, m, sl);
      const int i = F.xmodes ? m : s0 + sl, j = F.xmodes ? s0 + sl : m;
      const size_t k = (size_t)j * P.Npx + i;
      const double xv = it ? x[m * ld + sl] : 0.0;
      W.x[k] = xv;  // the recorded solution (ins2d_record_pairs)
      dp[k] = accumulate ? dp[k] + xv : xv;
    }
  if (c == 0 && tid == 0) {
    PcgScalars *out = W.sc;
    out->rr0 = rr0;
    out->rr = rr;
    out->it = it;
    out->maxx = maxx;
    out->minx = minx;
    out->maxres = maxres;
    out->status = status;
    out->done = 1;
    out->tol2 = tol2;
    out->maxit = maxit;
    if (acc) solve_accum(out, acc);
  }
  cl.sync();  // no block leaves while another may still write to its shared memory
}

}  // namespace

bool pcg_use_cluster(const FdmD &F) { return !F.spectral && std::max(F.nm, F.n) <= kFdmClusterMaxN; }

cudaError_t pcg_cluster_prepare() {
  const cudaError_t e = cudaFuncSetAttribute((const void *)k_pcg_cluster<true>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute((const void *)k_pcg_cluster<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kSmemMax);
}

void pcg_solve_cluster(const DevOps &P, const FdmD &F, const PcgWork &W, const SolveSrc &src, double *dp, double tol,
                       long long maxit, bool accumulate, SolveAccum *acc, cudaStream_t s) {
  const Geo g = make_geo(F);
  const size_t bytes = smem_doubles(g) * sizeof(double);
  if (g.qp)
    k_pcg_cluster<true><<<kC, kThreads, bytes, s>>>(P, F, W, g, src, dp, tol * tol, maxit, accumulate ? 1 : 0, acc);
  else
    k_pcg_cluster<false><<<kC, kThreads, bytes, s>>>(P, F, W, g, src, dp, tol * tol, maxit, accumulate ? 1 : 0, acc);
}

}  // namespace ins2d
