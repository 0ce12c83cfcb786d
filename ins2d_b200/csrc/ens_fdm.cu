// Poisson solves of an ensemble with the fast-diagonalization preconditioner,
// batched across members: the passes of pcg.cu's single-grid path, every
// kernel one launch over the work of all members that still iterate.
//
// A solve of members of 64 to 256 cells per direction is bound by its
// launches.  So a member's scalars are advanced by its last block in each
// reduction (no one-block kernels between), its statistics and the loop
// condition by the update, the divergence is formed by the initialisation and
// the solution is read by the projection.  24 members, RK44 step on B200:
// eleven launches and eleven more per pass before, 0.881 ms; six launches and
// five more per pass, 0.787 ms; with the members' ends below, 0.748 ms.
#include <cfloat>

#include "ins2d.h"
#include "kernels.cuh"
#include "reduce.cuh"

namespace ins2d {

namespace {

constexpr int kThreads = 256;
constexpr int kPer = kEnsCells / kThreads;  // cells per thread

__device__ __forceinline__ RedScratch member_red(EnsCg &C, int nq) {
  RedScratch r;
  r.partials = C.part;
  r.counter = &C.ticket;
  r.result = C.part + (size_t)C.ntiles * nq;
  r.max_blocks = C.ntiles;
  return r;
}

__device__ __forceinline__ void add_stats(const EnsCg &C, EnsStats &st) {
  st.n_solves += 1;
  st.iters_total += C.it;
  st.iters_max = C.it > st.iters_max ? C.it : st.iters_max;
  const double n1 = sqrt(C.rr);
  st.norm1_max = n1 > st.norm1_max ? n1 : st.norm1_max;
  if (C.status != 0 && st.status == 0) st.status = C.status;
}

// One thread per member and launch, when the member's scalars are final; the
// last member's sets the loop condition (first: before any pass).  The ticket
// counts members in its low and those still iterating in its high half: a
// ticket per block and a scan of the members' flags were 511 atomics on one
// word and another round of loads for 24 members (k_ef_update 11.9 -> 9.4 us, ten steps 7.75 ->
// 7.48 ms).
__device__ __forceinline__ void end_member(const EnsFdmRun &R, const LoopCond &cond, bool active, bool first) {
  const unsigned long long t = atomicAdd(R.ticket, 1ull + (active ? 1ull << 32 : 0ull)) + 1ull + (active ? 1ull << 32 : 0ull);
  if ((unsigned)t != (unsigned)R.n) return;
  const int act = (int)(t >> 32), loops = first ? 0 : *R.loops + 1;
  *R.ticket = 0ull;
  *R.loops = loops;
  set_cond(cond, act > 0 && loops < cond.limit);
}

__device__ __forceinline__ void copy_ops(DevOps *dst, const DevOps *src) {
  for (int k = threadIdx.x; k < (int)(sizeof(DevOps) / 8); k += blockDim.x)
    ((long long *)dst)[k] = ((const long long *)src)[k];
}

// f = (M Wt + yM/dt) gamma (mode 0) or M wres (mode 1); f'f, max|f|, sum
__global__ void __launch_bounds__(kThreads) k_ef_init(const EnsFdmRun R, int mode, double gamma, const LoopCond cond) {
  __shared__ __align__(16) DevOps sP;
  const int4 t = R.tiles[blockIdx.x];
  const EnsMemberD &M = R.mem[t.x];
  EnsCg &C = R.cg[t.x];
  copy_ops(&sP, &M.P);
  __syncthreads();
  const double *W = mode == 0 ? M.Wt : M.wres;
  const double alpha = mode == 0 ? 1.0 / M.dt : 0.0, g = mode == 0 ? gamma : 1.0;
  double q[3] = {0.0, 0.0, 0.0};
  const int ops[3] = {R_SUM, R_MAX, R_SUM};
  // loads of all the thread's cells before the first store, here and below: a
  // store in between orders the next cell's loads behind it
  const int Np = (int)sP.Np, Npx = sP.Npx;
  double *__restrict__ f = M.f;
  double fv[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x, j = k / Npx;
    fv[u] = k < Np ? div_cell(sP, W, alpha, 0.0, g, k - j * Npx, j) : 0.0;
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x;
    if (k < Np) f[k] = fv[u];
    q[0] += fv[u] * fv[u];
    q[1] = fmax(q[1], fabs(fv[u]));
    q[2] += fv[u];
  }
  double out[3];
  if (grid_reduce_at<3>(q, ops, member_red(C, 3), out, t.z, C.ntiles)) {
    const RhsRange range = C.singular ? RhsRange::of(out[2] / Np, Np, out[0], C.tol2) : RhsRange::none();
    C.mean = range.mean;
    C.add = range.add(out[0], C.tol2);
    C.rr0 = out[0];
    C.rr = 0.0;
    C.rz = 0.0;
    C.it = 0;
    C.status = 0;
    // pressure_poisson.m:33-38, cg.F:222-227
    int done = (out[1] < 1e-14 || C.rr0 <= C.tol2) ? 1 : 0;
    if (!isfinite(C.rr0)) {
      C.status = INS2D_ENONFINITE;
      done = 1;
    }
    if (!done && range.refused(out[0], C.tol2)) {
      C.status = INS2D_ENOTCONV;
      C.rr = range.miss / C.rr0;
      done = 1;
    }
    if (done) add_stats(C, R.stats[t.x]);
    C.done = done;
    C.stage = mode == 0;
    if (done && C.stage && C.status == 0) C.zero = 1;
    end_member(R, cond, !done, true);
  }
}

// p = z + beta p (directions alternate between two buffers), q = A p, p'q
__global__ void __launch_bounds__(kThreads) k_ef_step(const EnsFdmRun R) {
  const int4 t = R.tiles[blockIdx.x];
  EnsCg &C = R.cg[t.x];
  const EnsMemberD &M = R.mem[t.x];
  const int stop = *(volatile int *)&C.done;  // with the other scalars: one latency
  const long long it = C.it;
  const double beta = C.beta;
  const PcgWork W = M.W;
  const auto TX = M.P.TX, TY = M.P.TY;
  const double *__restrict__ hx = M.P.hx, *__restrict__ hy = M.P.hy;
  const int Npx = M.P.Npx, Np = (int)M.P.Np;
  if (stop) return;
  const bool first = it == 0, odd = it & 1;
  const double *__restrict__ z = M.zf, *__restrict__ po = odd ? W.p : W.p2;
  double *__restrict__ pn = odd ? W.p2 : W.p;
  auto pv = [&](long long k) {
    double v = __ldg(z + k);
    if (!first) v += beta * __ldg(po + k);
    return v;
  };
  double q[1] = {0.0};
  const int ops[1] = {R_SUM};
  double aq[kPer], pc[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x, j = k / Npx, i = k - j * Npx;
    aq[u] = pc[u] = 0.0;
    if (k < Np) {
      aq[u] = -(__ldg(hy + j) * tab_x_f(TX, i, pv, (long long)j * Npx) +
                __ldg(hx + i) * tab_y_f(TY, j, pv, 0, Npx, i));
      pc[u] = pv(k);
    }
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x;
    if (k < Np) {
      W.q[k] = aq[u];
      pn[k] = pc[u];
      q[0] += pc[u] * aq[u];
    }
  }
  double out[1];
  if (grid_reduce_at<1>(q, ops, member_red(C, 1), out, t.z, C.ntiles)) {
    if (!isfinite(out[0]))
      C.status = INS2D_ENONFINITE;
    else if (out[0] == 0.0 && C.status == 0)
      C.status = INS2D_EBREAKDOWN;
    C.alpha = C.status ? 0.0 : C.rz / out[0];
  }
}

// x += alpha p, r -= alpha q (x = 0, r = f before the first pass), the stopping
// rule, statistics and loop condition; a stage's solution becomes the member's
// when it has converged (a failed solve leaves the one before)
__global__ void __launch_bounds__(kThreads) k_ef_update(const EnsFdmRun R, const LoopCond cond) {
  const int4 t = R.tiles[blockIdx.x];
  EnsCg &C = R.cg[t.x];
  const EnsMemberD &M = R.mem[t.x];
  const int stop = *(volatile int *)&C.done;  // with the other scalars: one latency
  const long long it = C.it;
  const double alpha = C.alpha, sub = it == 0 ? C.mean : 0.0;
  const int sol = C.sol;
  const PcgWork W = M.W;
  double *xw = sol == 0 ? M.dp : M.W.x;
  const double *__restrict__ f = M.f;
  const int Np = (int)M.P.Np;
  if (stop) {
    if (t.z == 0 && threadIdx.x == 0) end_member(R, cond, false, false);
    return;
  }
  const bool first = it == 0;
  const double *__restrict__ p = (it & 1) ? W.p2 : W.p;
  double q[1] = {0.0};
  const int ops[1] = {R_SUM};
  double x[kPer], r[kPer];
  const double *ro = first ? f : W.r;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x;
    x[u] = r[u] = 0.0;
    if (k < Np) {
      x[u] = (first ? 0.0 : xw[k]) + alpha * __ldg(p + k);
      r[u] = (ro[k] - sub) - alpha * __ldg(W.q + k);
    }
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x;
    if (k < Np) {
      xw[k] = x[u];
      W.r[k] = r[u];
      q[0] += r[u] * r[u];
    }
  }
  double out[1];
  if (grid_reduce_at<1>(q, ops, member_red(C, 1), out, t.z, C.ntiles)) {
    int done = 0;
    if (C.status != 0) {  // found by this pass's reductions (cg.F:240-262)
      done = 1;
    } else {
      C.it += 1;
      C.rr = (out[0] + C.add) / C.rr0;
      if (!isfinite(C.rr)) {
        C.status = INS2D_ENONFINITE;
        done = 1;
      } else if (C.rr <= C.tol2) {
        done = 1;
      } else if (C.it >= C.maxit) {
        C.status = INS2D_ENOTCONV;
        done = 1;
      }
    }
    if (done) add_stats(C, R.stats[t.x]);
    C.done = done;
    if (done && C.stage && C.status == 0) {
      C.sol = sol ^ 1;
      C.zero = 0;
    }
    end_member(R, cond, !done, false);
  }
}

__global__ void __launch_bounds__(kThreads) k_ef_finish(const EnsFdmRun R) {
  const int4 t = R.tiles[blockIdx.x];
  const EnsCg &C = R.cg[t.x];
  if (C.it == 0 || C.status != 0) return;
  const EnsMemberD &M = R.mem[t.x];
  const double *__restrict__ x = C.sol == 0 ? M.dp : M.W.x;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int k = t.y + u * kThreads + threadIdx.x;
    if (k < M.P.Np) M.p[k] += x[k];
  }
}

}  // namespace

size_t ens_fdm_scratch(int nx, int ny) {
  const size_t cells = ((size_t)nx * ny + kEnsCells - 1) / kEnsCells;
  const size_t tiles = (size_t)((nx + 31) / 32) * ((ny + 31) / 32);  // fdm.cu's output tiles
  return 3 * cells + tiles + 8;
}

void ens_fdm_init(const EnsFdmRun &R, int mode, double gamma, cudaGraphConditionalHandle h, int limit, cudaStream_t s) {
  k_ef_init<<<R.ntiles, kThreads, 0, s>>>(R, mode, gamma, LoopCond{h, limit});
}
void ens_fdm_pass(const EnsFdmRun &R, const EnsFdmPlan &pl, cudaGraphConditionalHandle h, int limit, cudaStream_t s) {
  fdm_apply_ens(pl, R.cg, s);
  k_ef_step<<<R.ntiles, kThreads, 0, s>>>(R);
  k_ef_update<<<R.ntiles, kThreads, 0, s>>>(R, LoopCond{h, limit});
}
void ens_fdm_finish(const EnsFdmRun &R, cudaStream_t s) { k_ef_finish<<<R.ntiles, kThreads, 0, s>>>(R); }

}  // namespace ins2d
