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
// Beside the barriers (about 1000 cycles each) a launch pays for the first
// touch of its parameters, tables and instructions; what depends on the
// context and the boundary values alone is loaded before the wait for the previous
// kernel (programmatic dependent launch, DevOps::pdl).  Measured on B200, RK44 step
// of the 64^2 cavity (four solves): one thread block working from L1/L2 and a
// separate divergence launch 0.228 ms; eight blocks of 256 threads with
// scattered 8-byte exchanges 0.117 ms; 512 threads, 16-byte exchanges and
// staged operator rows 0.104 ms (two or four blocks: 0.131, 0.112 ms); with
// programmatic launches 0.096 ms.
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

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kN = kFdmClusterMaxN;
constexpr int kTriC = kN / 32;        // unknowns per lane of a system
constexpr int kSmemMax = 197 * 1024;  // dynamic; 29.5 KB of tables are static
constexpr int kC = 8;                // blocks of the cluster

// sizes of one solve
struct Geo {
  int nm, n;      // modes, unknowns per system
  int ns, nb;     // systems' unknowns (even) and modes per block (the last blocks may hold fewer or none)
  int ld;         // pitch of the cell arrays: ns rounded up to 8, plus 4 (4 or 12 mod 16: conflict-free fragments)
  int ldt;        // pitch of the rows of systems
  int mp;         // modes rounded up to 8
  int qp;         // pitch of the basis (4 mod 16), 0: not in shared memory
  int lg;         // cells of a slice are numbered with a power-of-two pitch 2^lg of the fast index
};
__host__ __device__ inline size_t cells(const Geo &g) { return (size_t)g.mp * g.ld; }
__host__ __device__ inline size_t smem_doubles(const Geo &g) {
  return 6 * cells(g) + (size_t)g.nb * g.ldt + 4 * (size_t)g.mp + (size_t)g.mp * g.qp;
}
Geo make_geo(const FdmD &F) {
  Geo g;
  g.nm = F.nm;
  g.n = F.n;
  g.ns = 2 * ((F.n + 2 * kC - 1) / (2 * kC));
  g.nb = (F.nm + kC - 1) / kC;
  g.ld = ((g.ns + 7) / 8) * 8 + 4;
  g.ldt = (F.n + 3) & ~1;
  g.mp = ((F.nm + 7) / 8) * 8;
  g.qp = ((F.nm + 15) / 16) * 16 + 4;
  if (smem_doubles(g) * sizeof(double) > kSmemMax) g.qp = 0;
  const int fast = F.xmodes ? F.nm : g.ns;
  g.lg = 0;
  while ((1 << g.lg) < fast) ++g.lg;
  return g;
}

__device__ __forceinline__ void mma884(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// C = op(Q) B on 8 x 8 fragments taken by the block's warps in turn; B: cell
// array (rows k, pitch ld), zero-padded rows and columns; TRANS: op(Q)(i, k) =
// Q(k, i), else Q(i, k); epi(row, column, value, next column's value), columns
// even.  Two accumulator pairs halve the chain of dependent MMAs.
template <bool TRANS, class QF, class Epi>
__device__ __forceinline__ void product(const Geo &g, const QF &q, const double *B, Epi epi) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gr = lane >> 2, t = lane & 3;
  const int tm = g.mp >> 3, tiles = tm * (g.ld >> 3);  // ld = 8 x column tiles + 4
  for (int f = warp; f < tiles; f += kWarps) {
    int bn = 0, bm = f;
    while (bm >= tm) {
      bm -= tm;
      bn += 8;
    }
    bm *= 8;
    double c0 = 0.0, c1 = 0.0, d0 = 0.0, d1 = 0.0;
    const double *b = B + (size_t)t * g.ld + bn + gr;
#pragma unroll 4
    for (int k = 0; k < g.mp; k += 8) {
      const double a0 = TRANS ? q(k + t, bm + gr) : q(bm + gr, k + t);
      const double a1 = TRANS ? q(k + 4 + t, bm + gr) : q(bm + gr, k + 4 + t);
      mma884(c0, c1, a0, b[(size_t)k * g.ld]);
      mma884(d0, d1, a1, b[(size_t)(k + 4) * g.ld]);
    }
    epi(bm + gr, bn + 2 * t, c0 + d0, c1 + d1);
  }
}

__device__ __forceinline__ double combine(double a, double b, int op) {
  return op == R_SUM ? a + b : (op == R_MAX ? (a > b ? a : b) : (a < b ? a : b));
}
// Sum / max / min of NQ values over the cluster: the block's value (warp
// shuffles, then warp 0), one packet to every block, a cluster barrier, and
// the same ordered combination in every thread.  slot alternates between two
// buffers.  Remote stores are few and wide throughout this kernel: an SM
// sends one packet in several cycles (a packet per warp instead of per block
// made the four-value reduction 4300 cycles, against about 1700).
template <int NQ>
__device__ __forceinline__ void cluster_reduce(cg::cluster_group &cl, double (&v)[NQ], const int (&ops)[NQ],
                                               double (*warp_part)[kWarps], double (*part)[kC][4], int &slot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = combine(v[q], __shfl_xor_sync(0xffffffffu, v[q], off), ops[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) warp_part[q][warp] = v[q];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = warp_part[q][lane & (kWarps - 1)];
#pragma unroll
    for (int off = kWarps / 2; off > 0; off >>= 1)
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] = combine(v[q], __shfl_xor_sync(0xffffffffu, v[q], off), ops[q]);
    if (lane < kC) {
      double2 *dst = reinterpret_cast<double2 *>(cl.map_shared_rank(&part[slot][cl.block_rank()][0], lane));
      dst[0] = make_double2(v[0], NQ > 1 ? v[NQ > 1 ? 1 : 0] : 0.0);
      if (NQ > 2) dst[1] = make_double2(v[NQ > 2 ? 2 : 0], v[NQ > 3 ? 3 : 0]);
    }
  }
  cl.sync();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double a = part[slot][0][q];
#pragma unroll
    for (int c = 1; c < kC; ++c) a = combine(a, part[slot][c][q], ops[q]);
    v[q] = a;
  }
  slot ^= 1;
}
static_assert(kWarps == 16, "two lanes per warp partial");

// one direction's rows of the operators in shared memory: the factor of A, the
// divergence (W is read at their columns), boundary coefficients and values
struct DirRows {
  int ac[kT][kN], mc[kT][kN];
  double aw[kT][kN], mw[kT][kN], h[kN], b1[kN], b2[kN], v1[kN], v2[kN];
};
__device__ __forceinline__ void load_dir(DirRows &D, int k, const Tab &A, const Tab &M, const double *h, int r,
                                         bool div, const double *v1, const double *v2) {
  D.h[k] = __ldg(h + r);
#pragma unroll
  for (int q = 0; q < kT; ++q) {
    const double w = __ldg(A.w + kT * r + q);
    const int c = __ldg(A.c + kT * r + q);
    D.aw[q][k] = w;
    D.ac[q][k] = w != 0.0 ? c : r;
  }
  if (!div) return;
#pragma unroll
  for (int q = 0; q < kT; ++q) {
    D.mw[q][k] = __ldg(M.w + kT * r + q);
    D.mc[q][k] = __ldg(M.c + kT * r + q);
  }
  D.b1[k] = __ldg(M.b1 + r);
  D.b2[k] = __ldg(M.b2 + r);
  D.v1[k] = __ldg(v1 + r);
  D.v2[k] = __ldg(v2 + r);
}

// QS: the basis in shared memory
template <bool QS>
__global__ void __launch_bounds__(kThreads, 1)
    k_pcg_cluster(const __grid_constant__ DevOps P, const __grid_constant__ FdmD F, const PcgWork W, const Geo g,
                  const __grid_constant__ SolveSrc src, double *__restrict__ dp, double tol2, long long maxit,
                  int accumulate, SolveAccum *acc) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double warp_part[4][kWarps];
  __shared__ __align__(16) double part2[2][kC][4], part4[2][kC][4];
  // the sum over the null mode's w, as its block sends it, and what follows from the
  // first pass's (tests of it made here once spilled 24 bytes: ten steps 28 us longer)
  __shared__ double wsum;
  __shared__ RhsRange range;
  __shared__ DirRows dm, ds;  // along the modes' and the systems' direction
  cg::cluster_group cl = cg::this_cluster();
  cl.barrier_arrive();  // every block runs before any other writes to its shared memory (waited for below)
  const int c = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nm = g.nm, n = g.n, ld = g.ld;
  const int s0 = c * g.ns, s1 = min(s0 + g.ns, n), nl = max(s1 - s0, 0);  // this block's slice
  const size_t nc = cells(g);
  double *r = sm, *p = r + nc, *x = p + nc, *q = x + nc, *z = q + nc, *zh = z + nc;
  // halo columns of p on the left and right, of z as the neighbours send them
  double *rows = zh + nc, *ph = rows + (size_t)g.nb * g.ldt, *zhalo = ph + 2 * g.mp, *Qs = zhalo + 2 * g.mp;
  int slot2 = 0, slot4 = 0;
  if (QS) {  // asynchronous: complete before the first product
    for (int i = warp; i < g.mp; i += kWarps)
      for (int b = lane; b < g.mp; b += 32) {
        const bool in = i < nm && b < nm;
        const unsigned d = (unsigned)__cvta_generic_to_shared(Qs + (size_t)i * g.qp + b);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d),
                     "l"(F.Q + (in ? (size_t)i * nm + b : 0)), "r"(in ? 8 : 0)
                     : "memory");
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  auto basis = [&](int i, int b) -> double {
    if constexpr (QS)
      return Qs[(size_t)i * g.qp + b];
    else
      return (i < nm && b < nm) ? __ldg(F.Q + (size_t)i * nm + b) : 0.0;
  };
  // the operators' rows
  const bool xm = F.xmodes;
  const bool div = src.mode != 0 && src.beta == 0.0;
  if (tid < nm)
    load_dir(dm, tid, xm ? P.TX : P.TY, xm ? P.MX : P.MY, xm ? P.hx : P.hy, tid, div, xm ? P.bc.vLo_i : P.bc.uLe_i,
             xm ? P.bc.vUp_i : P.bc.uRi_i);
  else if (tid >= kThreads / 2 && tid - kThreads / 2 < nl)
    load_dir(ds, tid - kThreads / 2, xm ? P.TY : P.TX, xm ? P.MY : P.MX, xm ? P.hy : P.hx, s0 + tid - kThreads / 2,
             div, xm ? P.bc.uLe_i : P.bc.vLo_i, xm ? P.bc.uRi_i : P.bc.vUp_i);
  if (tid == 0) range = RhsRange::none();
  // zero padding of the products' right operands
  for (int k = tid; k < (int)nc; k += kThreads) {
    r[k] = 0.0;
    zh[k] = 0.0;
  }
  __syncthreads();
  // cell l of the slice: (m, sl), the index of x fastest; false: padding
  const int nslots = (xm ? nl : nm) << g.lg;
  auto cell = [&](int l, int &m, int &sl) {
    const int a = l & ((1 << g.lg) - 1), b = l >> g.lg;
    m = xm ? a : b;
    sl = xm ? b : a;
    return m < nm && sl < nl;
  };
  // f = (M W + alpha yM) gamma from the rows above
  auto div_at = [&](const auto &Wf, int m, int sl, int i, int j) {
    const DirRows &dx = xm ? dm : ds, &dy = xm ? ds : dm;
    const int a = xm ? m : sl, b = xm ? sl : m;
    double u = 0.0, v = 0.0;
#pragma unroll
    for (int k = 0; k < kT; ++k) {
      u += dx.mw[k][a] * Wf((long long)j * P.Nux + dx.mc[k][a]);
      v += dy.mw[k][b] * Wf(P.Nu + (long long)dy.mc[k][b] * P.Nvx + i);
    }
    double d = dy.h[b] * u + dx.h[a] * v;
    if (src.alpha != 0.0)
      d += src.alpha * (dy.h[b] * (dx.b1[a] * dy.v1[b] + dx.b2[a] * dy.v2[b]) +
                        dx.h[a] * (dy.b1[b] * dx.v1[a] + dy.b2[b] * dx.v2[a]));
    return d * src.gamma;
  };
  // this warp's first system (tables of the others are read when they are solved)
  const int b0 = c * g.nb, b1 = min(b0 + g.nb, nm);
  TriTab<kTriC> tab;
  tri_tables<kTriC>(F, b0 + warp < b1 ? b0 + warp : nm, lane * kTriC, tab);
  // everything above reads tables of the context and boundary values, complete
  // before the previous kernel started (pdl_wait); the right-hand side is its work
  pdl_wait();
  pdl_trigger();
  // right-hand side (cg.F:207-229 with x_in = 0)
  double a2[2] = {0.0, 0.0};
  const int op2[2] = {R_SUM, R_MAX};
#pragma unroll 2
  for (int l = tid; l < nslots; l += kThreads) {
    int m, sl;
    if (!cell(l, m, sl)) continue;
    const int s = s0 + sl, i = xm ? m : s, j = xm ? s : m;
    double f;
    if (src.mode == 0)
      f = src.f[(size_t)j * P.Npx + i];
    else if (src.mode == 1)
      f = div ? div_at(WPlain{src.f}, m, sl, i, j)
              : div_cell_f(P, WPlain{src.f}, src.alpha, src.beta, src.gamma, i, j);
    else
      f = div ? div_at(src.ws, m, sl, i, j) : div_cell_f(P, src.ws, src.alpha, src.beta, src.gamma, i, j);
    r[m * ld + sl] = f;
    a2[0] += f * f;
    a2[1] = fabs(f) > a2[1] ? fabs(f) : a2[1];
  }
  // the halo columns (wrapped ones serve cyclic rows only) and the blocks whose
  // left / right halo column is this block's last / first one
  const int sL = s0 > 0 ? s0 - 1 : n - 1, sR = s1 < n ? s1 : 0;
  const int bl = sR / g.ns, br = sL / g.ns;
  cl.barrier_wait();
  cluster_reduce<2>(cl, a2, op2, warp_part, part2, slot2);
  const double rr0 = a2[0];
  double rz = 0.0, rr = 0.0, maxx = 0.0, minx = 0.0, maxres = 0.0;
  long long it = 0;
  int status = 0;
  bool done = (a2[1] < 1e-14 || rr0 <= tol2);  // pressure_poisson.m:33-38, cg.F:222-227
  if (!isfinite(rr0)) {
    status = INS2D_ENONFINITE;
    done = true;
  }
  const int op1[1] = {R_SUM};
  if (QS) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
  }
  // the loop's exits are taken by all blocks alike: every condition comes
  // from a cluster-wide reduction
  while (!done) {
    // w = Q' r, each row to the block that solves it
    product<true>(g, basis, r, [&](int b, int sl, double v0, double v1) {
      if (b < nm && sl < nl) {
        const int o = b / g.nb;
        double *d = cl.map_shared_rank(rows, o) + (size_t)(b - o * g.nb) * g.ldt + s0 + sl;
        *reinterpret_cast<double2 *>(d) = make_double2(v0, v1);  // rows hold n + 1 values or more
      }
    });
    cl.sync();
    for (int b = b0 + warp; b < b1; b += kWarps) {
      double *w = rows + (size_t)(b - b0) * g.ldt;
      double y[kTriC];
#pragma unroll
      for (int k = 0; k < kTriC; ++k) y[k] = lane * kTriC + k < n ? w[lane * kTriC + k] : 0.0;
      if (b != b0 + warp) {
        TriTab<kTriC> t2;
        tri_tables<kTriC>(F, b, lane * kTriC, t2);
        tri_solve<1, kTriC>(F, b, 0, t2, y, nullptr);
      } else {
        tri_solve<1, kTriC>(F, b, 0, tab, y, nullptr, [&](double s) {
          if (lane < kC) *cl.map_shared_rank(&wsum, lane) = s;  // the first pass's is read
        });
      }
      // back through the row, so that consecutive lanes send consecutive values
#pragma unroll
      for (int k = 0; k < kTriC; ++k)
        if (lane * kTriC + k < n) w[lane * kTriC + k] = y[k];
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kN / 64; ++k) {
        const int s = 2 * (lane + 32 * k);
        if (s < n) {
          const int o = s / g.ns;
          double *d = cl.map_shared_rank(zh, o) + (size_t)b * ld + s - o * g.ns;
          *reinterpret_cast<double2 *>(d) =
              make_double2(w[s], s + 1 < n ? w[s + 1] : 0.0);  // a padding column stays zero
        }
      }
    }
    cl.sync();
    // by a warp that has no fragment of the product on small grids
    if (it == 0 && F.null_mode >= 0 && tid == kThreads - 1)
      range = RhsRange::of(wsum * F.mean_w, (double)nm * n, rr0, tol2);
    double a1[1] = {0.0};
    product<false>(g, basis, zh, [&](int m, int sl, double v0, double v1) {
      if (m >= nm || sl >= nl) return;
      const int k = m * ld + sl;
      z[k] = v0;
      a1[0] += r[k] * v0;
      if (sl == 0) cl.map_shared_rank(zhalo, br)[g.mp + m] = v0;
      if (sl + 1 < nl) {
        z[k + 1] = v1;
        a1[0] += r[k + 1] * v1;
      }
      if (sl + 2 >= nl) cl.map_shared_rank(zhalo, bl)[m] = sl + 1 < nl ? v1 : v0;
    });
    cluster_reduce<1>(cl, a1, op1, warp_part, part2, slot2);
    if (!isfinite(a1[0])) {
      status = INS2D_ENONFINITE;
      break;
    }
    const bool first = it == 0;
    if (first && range.refused(rr0, tol2)) {
      status = INS2D_ENOTCONV;
      break;
    }
    const double beta = first ? 0.0 : a1[0] / rz;
    rz = a1[0];
    // p = z + beta p, with the neighbouring columns'
    for (int k = tid; k < (int)nc; k += kThreads) p[k] = first ? z[k] : z[k] + beta * p[k];
    for (int k = tid; k < 2 * g.mp; k += kThreads) ph[k] = first ? zhalo[k] : zhalo[k] + beta * ph[k];
    __syncthreads();
    // q = A p, p'q
    a1[0] = 0.0;
#pragma unroll 2
    for (int l = tid; l < nslots; l += kThreads) {
      int m, sl;
      if (!cell(l, m, sl)) continue;
      double tm = 0.0, ts = 0.0;
#pragma unroll
      for (int k = 0; k < kT; ++k) {
        tm += dm.aw[k][m] * p[dm.ac[k][m] * ld + sl];
        const int sc = ds.ac[k][sl];
        const double *at = sc >= s0 && sc < s1 ? p + m * ld + sc - s0 : (sc == sL ? ph + m : ph + g.mp + m);
        ts += ds.aw[k][sl] * *at;
      }
      const double aq = -(ds.h[sl] * tm + dm.h[m] * ts);
      q[m * ld + sl] = aq;
      a1[0] += p[m * ld + sl] * aq;
    }
    cluster_reduce<1>(cl, a1, op1, warp_part, part2, slot2);
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
#pragma unroll 2
    for (int l = tid; l < nslots; l += kThreads) {
      int m, sl;
      if (!cell(l, m, sl)) continue;
      const int k = m * ld + sl;
      const double xv = (first ? 0.0 : x[k]) + alpha * p[k];
      const double rv = (r[k] - (first ? range.mean : 0.0)) - alpha * q[k];
      x[k] = xv;
      r[k] = rv;
      a4[0] += rv * rv;
      a4[1] = combine(a4[1], xv, R_MAX);
      a4[2] = combine(a4[2], xv, R_MIN);
      a4[3] = combine(a4[3], fabs(rv), R_MAX);
    }
    cluster_reduce<4>(cl, a4, op4, warp_part, part4, slot4);
    ++it;
    rr = (a4[0] + range.add(rr0, tol2)) / rr0;
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
#pragma unroll 2
    for (int l = tid; l < nslots; l += kThreads) {
      int m, sl;
      if (!cell(l, m, sl)) continue;
      const int s = s0 + sl, i = xm ? m : s, j = xm ? s : m;
      const size_t k = (size_t)j * P.Npx + i;
      const double xv = it ? x[m * ld + sl] : 0.0;
      W.x[k] = xv;  // the recorded solution (ins2d_record_pairs)
      dp[k] = accumulate ? dp[k] + xv : xv;
    }
  if (c == 0 && tid == 0) {
    PcgScalars *out = W.sc;
    out->rr0 = rr0;
    out->rr = it == 0 && status == INS2D_ENOTCONV ? range.miss / rr0 : rr;
    out->it = it;
    out->maxx = maxx;
    out->minx = minx;
    out->maxres = maxres;
    out->status = status;
    out->done = 1;
    out->tol2 = tol2;
    out->maxit = maxit;
    if (acc) solve_accum(out, acc);
    if (W.hsc) *W.hsc = *out;
  }
  cl.sync();  // no block leaves while another may still write to its shared memory
}

template <bool QS>
cudaError_t launch_cluster(const DevOps &P, const FdmD &F, const PcgWork &W, const Geo &g, const SolveSrc &src,
                           double *dp, double tol2, long long maxit, int accumulate, SolveAccum *acc, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kC);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_doubles(g) * sizeof(double);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kC;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = P.pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, k_pcg_cluster<QS>, P, F, W, g, src, dp, tol2, maxit, accumulate, acc);
}

}  // namespace

bool pcg_use_cluster(const FdmD &F) { return !F.spectral && std::max(F.nm, F.n) <= kFdmClusterMaxN; }

cudaError_t pcg_cluster_prepare() {
  cudaError_t first = cudaSuccess;
  auto opt_in = [&](const void *k) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (first == cudaSuccess) first = e;
  };
  opt_in((const void *)k_pcg_cluster<true>);
  opt_in((const void *)k_pcg_cluster<false>);
  return first;
}

cudaError_t pcg_solve_cluster(const DevOps &P, const FdmD &F, const PcgWork &W, const SolveSrc &src, double *dp,
                              double tol, long long maxit, bool accumulate, SolveAccum *acc, cudaStream_t s) {
  const Geo g = make_geo(F);
  const int ac = accumulate ? 1 : 0;
  return g.qp ? launch_cluster<true>(P, F, W, g, src, dp, tol * tol, maxit, ac, acc, s)
              : launch_cluster<false>(P, F, W, g, src, dp, tol * tol, maxit, ac, acc, s);
}

}  // namespace ins2d
