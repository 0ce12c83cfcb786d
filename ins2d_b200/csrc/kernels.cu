// Stencil kernels of the INS2D hot path: RK stage right-hand side, residual,
// F, divergence, projection, Laplacian and conservation diagnostics.
//
// Thread mapping: one thread per (i,j) of the union of the u, v and p index
// spaces, 32x8 thread blocks (x fastest, coalesced along rows).  Stencil
// neighbours are served from L1/L2; each field is read from DRAM once per
// kernel.  Reductions are deterministic: per-block partials reduced in block
// order by the last block to finish.
#include <algorithm>
#include <cfloat>
#include <cstdlib>

#include "kernels.cuh"
#include "reduce.cuh"

namespace ins2d {

bool pdl_enabled() {
  static const bool on = [] {
    const char *v = std::getenv("INS2D_PDL");
    return v && v[0] == '1';
  }();
  return on;
}

namespace {

constexpr int BX = 32, BY = 8;

inline dim3 grid_for(int nx, int ny) { return dim3((nx + BX - 1) / BX, (ny + BY - 1) / BY); }

template <bool SAMEC>
__global__ void __launch_bounds__(256) k_F(const __grid_constant__ DevOps P, const double *__restrict__ V,
                                          const double *__restrict__ C, const double *__restrict__ p,
                                          double *__restrict__ Fo, const RedScratch red) {
  const int i = blockIdx.x * BX + threadIdx.x;
  const int j = blockIdx.y * BY + threadIdx.y;
  const double *u = V, *v = V + P.Nu, *cu = C, *cv = C + P.Nu;
  const double ypfac = p ? 1.0 : 0.0;
  double mx[1] = {0.0};
  const int ops[1] = {R_MAX};
  if (i < P.Nux && j < P.Nuy) {
    const long long idx = (long long)j * P.Nux + i;
    double R = rhs_u<double, SAMEC>(P, u, v, cu, cv, i, j, ypfac);
    if (p) R -= grad_x(P, p, i, j);
    Fo[idx] = R;
    mx[0] = fmax(mx[0], fabs(R));
  }
  if (i < P.Nvx && j < P.Nvy) {
    const long long idx = P.Nu + (long long)j * P.Nvx + i;
    double R = rhs_v<double, SAMEC>(P, u, v, cu, cv, i, j, ypfac);
    if (p) R -= grad_y(P, p, i, j);
    Fo[idx] = R;
    mx[0] = fmax(mx[0], fabs(R));
  }
  grid_reduce<1>(mx, ops, red);
}

template <bool WANTMAX, class F>
__global__ void __launch_bounds__(256) k_div(const __grid_constant__ DevOps P, const F W, double alpha, double beta,
                                            double gamma, double *__restrict__ f, const RedScratch red) {
  const int i = blockIdx.x * BX + threadIdx.x;
  const int j = blockIdx.y * BY + threadIdx.y;
  double mx[1] = {0.0};
  const int ops[1] = {R_MAX};
  if (i < P.Npx && j < P.Npy) {
    const double d = div_cell_f(P, W, alpha, beta, gamma, i, j);
    f[(long long)j * P.Npx + i] = d;
    mx[0] = fabs(d);
  }
  if (WANTMAX) grid_reduce<1>(mx, ops, red);
}

// V_out(i,j) = dt (Wt - c Om^-1 G dp) at the u and v points of (i,j)
__device__ __forceinline__ void project_cell(const DevOps &P, const double *__restrict__ Wt,
                                             const double *__restrict__ dp, double dt, double c,
                                             double *__restrict__ Vo, int i, int j) {
  if (i < P.Nux && j < P.Nuy) {
    const long long idx = (long long)j * P.Nux + i;
    Vo[idx] = dt * (Wt[idx] - c * om_inv_u(P, i, j) * grad_x_fast(P, dp, i, j));
  }
  if (i < P.Nvx && j < P.Nvy) {
    const long long idx = P.Nu + (long long)j * P.Nvx + i;
    Vo[idx] = dt * (Wt[idx] - c * om_inv_v(P, i, j) * grad_y_fast(P, dp, i, j));
  }
}

// Each thread projects kProjRows rows (BY apart) of one column: src.load(idx)
// what it reads at a point, src.store(idx, that, c Om^-1 (G dp)).  A block
// whose every row of both gradients is regular issues the loads of all its
// points before the first store; a store between them, or a branch per point,
// leaves one point's loads in flight at a time.  Ten steps at 512^2 1.052 ->
// 0.953 ms, two at 2048^2 1.752 -> 1.736 ms; two rows a thread 0.972 and 1.738,
// four blocks per SM (spills) 0.974 and 1.754.
#ifndef INS2D_PROJ_ROWS
#define INS2D_PROJ_ROWS 4
#endif
#ifndef INS2D_PROJ_MINB
#define INS2D_PROJ_MINB 3
#endif
constexpr int kProjRows = INS2D_PROJ_ROWS;
template <typename Src>
__device__ __forceinline__ void project_rows(const DevOps &P, const Src &src, const double *__restrict__ dp, double c) {
  const int i0 = blockIdx.x * BX, jb = blockIdx.y * (BY * kProjRows), ie = i0 + BX, je = jb + BY * kProjRows;
  const int i = i0 + threadIdx.x, j0 = jb + threadIdx.y;
  const RegD &X = P.rMXT, &Y = P.rMYT;
  if (ie <= P.Nux && ie <= P.Nvx && je <= P.Nuy && je <= P.Nvy && i0 >= X.lo && ie <= X.hi && jb >= Y.lo &&
      je <= Y.hi) {
    typename Src::Raw u[kProjRows], v[kProjRows];
    double gu[kProjRows], gv[kProjRows];
#pragma unroll
    for (int r = 0; r < kProjRows; ++r) {
      const int j = j0 + r * BY;
      u[r] = src.load((long long)j * P.Nux + i);
      v[r] = src.load(P.Nu + (long long)j * P.Nvx + i);
      gu[r] = c * om_inv_u(P, i, j) * (-__ldg(P.hy + j) * reg_x(X, i, dp, (long long)j * P.Npx));
      gv[r] = c * om_inv_v(P, i, j) * (-__ldg(P.hx + i) * reg_y(Y, j, dp, P.Npx, i));
    }
#pragma unroll
    for (int r = 0; r < kProjRows; ++r) {
      const int j = j0 + r * BY;
      src.store((long long)j * P.Nux + i, u[r], gu[r]);
      src.store(P.Nu + (long long)j * P.Nvx + i, v[r], gv[r]);
    }
    return;
  }
#pragma unroll 1
  for (int r = 0; r < kProjRows; ++r) {
    const int j = j0 + r * BY;
    if (i < P.Nux && j < P.Nuy) {
      const long long k = (long long)j * P.Nux + i;
      src.store(k, src.load(k), c * om_inv_u(P, i, j) * grad_x_fast(P, dp, i, j));
    }
    if (i < P.Nvx && j < P.Nvy) {
      const long long k = P.Nu + (long long)j * P.Nvx + i;
      src.store(k, src.load(k), c * om_inv_v(P, i, j) * grad_y_fast(P, dp, i, j));
    }
  }
}

struct ProjPlain {
  const double *Wt;
  double *Vo;
  double dt;
  using Raw = double;
  __device__ __forceinline__ Raw load(long long k) const { return __ldg(Wt + k); }
  __device__ __forceinline__ void store(long long k, Raw w, double g) const { Vo[k] = dt * (w - g); }
};
__global__ void __launch_bounds__(256, INS2D_PROJ_MINB) k_project(const __grid_constant__ DevOps P,
                                                                  const double *__restrict__ Wt,
                                                                  const double *__restrict__ dp, double dt, double c,
                                                                  double *__restrict__ Vo) {
  pdl_wait();
  pdl_trigger();
  project_rows(P, ProjPlain{Wt, Vo, dt}, dp, c);
}

// the first stage from the cached residual fused into its projection:
// Wt = Vn/dt + aii kV0 (k_stage_cached's expression) formed in registers, so
// Wt is neither written nor read again (the first stage solves no Poisson
// equation when the boundary conditions are steady: dp = p)
struct ProjCached {
  const double *Vn, *kV0;
  double *Vo;
  double aii, inv_dt, dt;
  struct Raw {
    double v, k;
  };
  __device__ __forceinline__ Raw load(long long k) const { return Raw{__ldg(Vn + k), __ldg(kV0 + k)}; }
  __device__ __forceinline__ void store(long long k, Raw w, double g) const {
    Vo[k] = dt * ((w.v * inv_dt + aii * w.k) - g);
  }
};
__global__ void __launch_bounds__(256, INS2D_PROJ_MINB) k_project_cached(
    const __grid_constant__ DevOps P, const double *__restrict__ Vn, const double *__restrict__ kV0, double aii,
    double inv_dt, const double *__restrict__ dp, double dt, double c, double *__restrict__ Vo) {
  pdl_wait();
  pdl_trigger();
  project_rows(P, ProjCached{Vn, kV0, Vo, aii, inv_dt, dt}, dp, c);
}

// FP32-storage stages: V_out = Vn + dt (a T - c Om^-1 G dp) in FP64 (T = the
// stage's Vtemp / a), stored as TO: float for the next stage's stencils, double
// for the new state (then V_out may be Vn itself: each point is read before it
// is written by the same thread)
template <typename TO>
struct Proj32 {
  const double *Vn;
  const float *T;
  TO *Vo;
  double a, dt;
  struct Raw {
    double v;
    float t;
  };
  __device__ __forceinline__ Raw load(long long k) const { return Raw{Vn[k], __ldg(T + k)}; }
  __device__ __forceinline__ void store(long long k, Raw w, double g) const {
    Vo[k] = (TO)(w.v + dt * (a * (double)w.t - g));
  }
};
template <typename TO>
__global__ void __launch_bounds__(256, INS2D_PROJ_MINB) k_project32(const __grid_constant__ DevOps P, const double *Vn,
                                                                    const float *__restrict__ T, double a,
                                                                    const double *__restrict__ dp, double dt, double c,
                                                                    TO *Vo) {
  pdl_wait();
  pdl_trigger();
  project_rows(P, Proj32<TO>{Vn, T, Vo, a, dt}, dp, c);
}

__global__ void __launch_bounds__(256) k_correct(const __grid_constant__ DevOps P, const double *__restrict__ Vi,
                                                const double *__restrict__ dp, double *__restrict__ Vo) {
  const int i = blockIdx.x * BX + threadIdx.x;
  const int j = blockIdx.y * BY + threadIdx.y;
  if (i < P.Nux && j < P.Nuy) {
    const long long idx = (long long)j * P.Nux + i;
    Vo[idx] = Vi[idx] - om_inv_u(P, i, j) * grad_x(P, dp, i, j);
  }
  if (i < P.Nvx && j < P.Nvy) {
    const long long idx = P.Nu + (long long)j * P.Nvx + i;
    Vo[idx] = Vi[idx] - om_inv_v(P, i, j) * grad_y(P, dp, i, j);
  }
}

__global__ void __launch_bounds__(256) k_lap(const __grid_constant__ DevOps P, const double *__restrict__ p,
                                            double *__restrict__ Ap) {
  const int i = blockIdx.x * BX + threadIdx.x;
  const int j = blockIdx.y * BY + threadIdx.y;
  if (i < P.Npx && j < P.Npy) Ap[(long long)j * P.Npx + i] = lap(P, p, i, j);
}

// {max|M V + yM|, sums of Omu u, Omv v, Omu u^2, Omv v^2}; a thread walks
// `rows` consecutive rows of one column.  Blocks whose cells are all regular
// two-point rows of Mx and My (no boundary terms, no wrap in y) take a loop
// with running pointers and weights in registers: three field loads and about
// 35 instructions per cell, several rows' loads in flight; the general loop
// (120 instructions a cell, and dependent loads) was bound by issue and
// latency.  Measured on B200, general loop everywhere with rows 8 apart: 54 us
// at 2048^2, now 38 us; 18.5 us at 64^2, now 9.5 us (16 rows were one
// thread's serial work; fewer while the launch has less than two blocks per SM).
__global__ void __launch_bounds__(256) k_conservation(const __grid_constant__ DevOps P, const double *__restrict__ V,
                                                     int rows, const RedScratch red) {
  const int i0 = blockIdx.x * BX, i = i0 + threadIdx.x;
  const int jb = blockIdx.y * BY * rows, j0 = jb + threadIdx.y * rows;
  const double *u = V, *v = V + P.Nu;
  double q[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int ops[5] = {R_MAX, R_SUM, R_SUM, R_SUM, R_SUM};
  const RegD &X = P.rMX, &Y = P.rMY;
  const int ie = i0 + BX, je = jb + BY * rows;  // end of the block's cells
  if (i0 >= X.lo && ie <= X.hi && jb >= Y.lo && je <= Y.hi && X.two && Y.two && (X.s == 0 || X.s == -1) &&
      (Y.s == 0 || Y.s == -1) && jb + Y.s >= 0 && je + Y.s < Y.n && ie <= P.Nux && ie <= P.Nvx && je <= P.Nuy &&
      je <= P.Nvy) {
    const double w0 = __ldg(X.w0 + i), w1 = __ldg(X.w1 + i), hx = __ldg(P.hx + i), gx = __ldg(P.gxi + i);
    const int c0 = wrapn(i + X.s, X.n), c1 = wrapn(c0 + 1, X.n);
    const double *u0 = u + (long long)j0 * P.Nux + c0, *vp = v + (long long)(j0 + Y.s) * P.Nvx + i;
    const int du = c1 - c0;
    const double *hy = P.hy + j0, *gy = P.gyi + j0, *m0 = Y.w0 + j0, *m1 = Y.w1 + j0;
    double va = __ldg(vp);
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
      vp += P.Nvx;
      const double ua = __ldg(u0), ub = __ldg(u0 + du), vb = __ldg(vp);
      u0 += P.Nux;
      const double h = __ldg(hy + r);
      q[0] = fmax(q[0], fabs(h * (w0 * ua + w1 * ub) + hx * (__ldg(m0 + r) * va + __ldg(m1 + r) * vb)));
      const double x = X.s == 0 ? ua : ub, y = Y.s == 0 ? va : vb;
      const double ou = h * gx, ov = __ldg(gy + r) * hx;
      q[1] += ou * x;
      q[3] += ou * x * x;
      q[2] += ov * y;
      q[4] += ov * y * y;
      va = vb;
    }
  } else {
    for (int r = 0; r < rows; ++r) {
      const int j = j0 + r;
      if (i < P.Npx && j < P.Npy) q[0] = fmax(q[0], fabs(div_cell_f(P, WPlain{V}, 1.0, 0.0, 1.0, i, j)));
      if (i < P.Nux && j < P.Nuy) {
        const double om = __ldg(P.hy + j) * __ldg(P.gxi + i);
        const double x = __ldg(u + (long long)j * P.Nux + i);
        q[1] += om * x;
        q[3] += om * x * x;
      }
      if (i < P.Nvx && j < P.Nvy) {
        const double om = __ldg(P.gyi + j) * __ldg(P.hx + i);
        const double x = __ldg(v + (long long)j * P.Nvx + i);
        q[2] += om * x;
        q[4] += om * x * x;
      }
    }
  }
  grid_reduce<5>(q, ops, red);
}

__global__ void k_stage_cached(const double *__restrict__ kV0, const double *__restrict__ Vn, double aii,
                               double inv_dt, double *__restrict__ Wt, long long n) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    Wt[k] = Vn[k] * inv_dt + aii * kV0[k];
}

__global__ void k_add(const double *__restrict__ x, double *__restrict__ y, long long n) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    y[k] += x[k];
}

// --- ensembles ---------------------------------------------------------------------
__device__ __forceinline__ void copy_ops(DevOps *dst, const DevOps *src) {
  const int tid = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
  for (int k = tid; k < (int)(sizeof(DevOps) / 8); k += nt) ((long long *)dst)[k] = ((const long long *)src)[k];
}

__global__ void __launch_bounds__(256) k_div_ens(const EnsMemberD *__restrict__ mem, const int4 *__restrict__ tiles,
                                                int mode, double gamma) {
  __shared__ __align__(16) DevOps sP;
  const int4 t = tiles[blockIdx.x];
  const EnsMemberD &M = mem[t.x];
  copy_ops(&sP, &M.P);
  __syncthreads();
  const int i = t.y * BX + threadIdx.x, j = t.z * BY + threadIdx.y;
  if (i < sP.Npx && j < sP.Npy)
    M.f[(long long)j * sP.Npx + i] =
        mode == 0 ? div_cell(sP, M.Wt, 1.0 / M.dt, 0.0, gamma, i, j) : div_cell(sP, M.wres, 0.0, 0.0, 1.0, i, j);
}

__global__ void __launch_bounds__(256) k_project_ens(const EnsMemberD *__restrict__ mem,
                                                    const int4 *__restrict__ tiles, double c, int from_p,
                                                    int last, const EnsCg *__restrict__ cg) {
  __shared__ __align__(16) DevOps sP;
  const int4 t = tiles[blockIdx.x];
  const EnsMemberD &M = mem[t.x];
  copy_ops(&sP, &M.P);
  __syncthreads();
  const int i = t.y * BX + threadIdx.x, j = t.z * BY + threadIdx.y;
  double *__restrict__ Vo = last ? M.V : M.Vs;
  if (cg && cg[t.x].zero) {  // dp = 0
    if (i < sP.Nux && j < sP.Nuy) Vo[(long long)j * sP.Nux + i] = M.dt * M.Wt[(long long)j * sP.Nux + i];
    if (i < sP.Nvx && j < sP.Nvy) {
      const long long k = sP.Nu + (long long)j * sP.Nvx + i;
      Vo[k] = M.dt * M.Wt[k];
    }
    return;
  }
  project_cell(sP, M.Wt, from_p ? M.p : (cg && cg[t.x].sol == 0 ? M.W.x : M.dp), M.dt, c, Vo, i, j);
}

__global__ void __launch_bounds__(256) k_stage_cached_ens(const EnsMemberD *__restrict__ mem,
                                                         const int4 *__restrict__ tiles, double aii) {
  const int4 t = tiles[blockIdx.x];
  const EnsMemberD &M = mem[t.x];
  const double inv_dt = 1.0 / M.dt;
  const int i = t.y * BX + threadIdx.x, j = t.z * BY + threadIdx.y;
  const DevOps &P = M.P;
  if (i < P.Nux && j < P.Nuy) {
    const long long idx = (long long)j * P.Nux + i;
    M.Wt[idx] = M.V[idx] * inv_dt + aii * M.kV[0][idx];
  }
  if (i < P.Nvx && j < P.Nvy) {
    const long long idx = P.Nu + (long long)j * P.Nvx + i;
    M.Wt[idx] = M.V[idx] * inv_dt + aii * M.kV[0][idx];
  }
}

}  // namespace

void launch_F(const DevOps &P, const double *V, const double *C, const double *p, double *F_out,
              const RedScratch &red, cudaStream_t s) {
  dim3 g = grid_for(P.Nux > P.Nvx ? P.Nux : P.Nvx, P.Nuy > P.Nvy ? P.Nuy : P.Nvy);
  if (C == nullptr || C == V)
    k_F<true><<<g, dim3(BX, BY), 0, s>>>(P, V, V, p, F_out, red);
  else
    k_F<false><<<g, dim3(BX, BY), 0, s>>>(P, V, C, p, F_out, red);
}

void launch_div(const DevOps &P, const double *W, double alpha, double beta, double gamma, double *f,
                bool want_max, const RedScratch &red, cudaStream_t s) {
  dim3 g = grid_for(P.Npx, P.Npy);
  if (want_max)
    k_div<true><<<g, dim3(BX, BY), 0, s>>>(P, WPlain{W}, alpha, beta, gamma, f, red);
  else
    k_div<false><<<g, dim3(BX, BY), 0, s>>>(P, WPlain{W}, alpha, beta, gamma, f, red);
}

void launch_div_split(const DevOps &P, const double *Vn, const float *T, double sv, double sa, double alpha,
                      double beta, double gamma, double *f, cudaStream_t s) {
  k_div<false><<<grid_for(P.Npx, P.Npy), dim3(BX, BY), 0, s>>>(P, WSplit{Vn, T, sv, sa}, alpha, beta, gamma, f,
                                                                RedScratch{});
}

void launch_project(const DevOps &P, const double *Wt, const double *dp, double dt, double c, double *V_out,
                    cudaStream_t s) {
  const int nx = P.Nux > P.Nvx ? P.Nux : P.Nvx, ny = P.Nuy > P.Nvy ? P.Nuy : P.Nvy;
  const dim3 g((nx + BX - 1) / BX, (ny + BY * kProjRows - 1) / (BY * kProjRows));
  launch_kp(P.pdl, k_project, g, dim3(BX, BY), 0, s, P, Wt, dp, dt, c, V_out);
}

template <typename TO>
void launch_project32_t(const DevOps &P, const double *Vn, const float *T, double a, const double *dp, double dt,
                        double c, TO *V_out, cudaStream_t s) {
  const int nx = P.Nux > P.Nvx ? P.Nux : P.Nvx, ny = P.Nuy > P.Nvy ? P.Nuy : P.Nvy;
  const dim3 g((nx + BX - 1) / BX, (ny + BY * kProjRows - 1) / (BY * kProjRows));
  launch_kp(P.pdl, k_project32<TO>, g, dim3(BX, BY), 0, s, P, Vn, T, a, dp, dt, c, V_out);
}
void launch_project32(const DevOps &P, const double *Vn, const float *T, double a, const double *dp, double dt,
                      double c, float *V_out, cudaStream_t s) {
  launch_project32_t(P, Vn, T, a, dp, dt, c, V_out, s);
}
void launch_project32(const DevOps &P, const double *Vn, const float *T, double a, const double *dp, double dt,
                      double c, double *V_out, cudaStream_t s) {
  launch_project32_t(P, Vn, T, a, dp, dt, c, V_out, s);
}

void launch_project_cached(const DevOps &P, const double *Vn, const double *kV0, double aii, double inv_dt,
                           const double *dp, double dt, double c, double *V_out, cudaStream_t s) {
  const int nx = P.Nux > P.Nvx ? P.Nux : P.Nvx, ny = P.Nuy > P.Nvy ? P.Nuy : P.Nvy;
  const dim3 g((nx + BX - 1) / BX, (ny + BY * kProjRows - 1) / (BY * kProjRows));
  launch_kp(P.pdl, k_project_cached, g, dim3(BX, BY), 0, s, P, Vn, kV0, aii, inv_dt, dp, dt, c, V_out);
}

void launch_correct(const DevOps &P, const double *V_in, const double *dp, double *V_out, cudaStream_t s) {
  dim3 g = grid_for(P.Nux > P.Nvx ? P.Nux : P.Nvx, P.Nuy > P.Nvy ? P.Nuy : P.Nvy);
  k_correct<<<g, dim3(BX, BY), 0, s>>>(P, V_in, dp, V_out);
}

void launch_lap(const DevOps &P, const double *p, double *Ap, cudaStream_t s) {
  k_lap<<<grid_for(P.Npx, P.Npy), dim3(BX, BY), 0, s>>>(P, p, Ap);
}

void launch_conservation(const DevOps &P, const double *V, const RedScratch &red, cudaStream_t s) {
  const int nx = P.Nux > P.Nvx ? P.Nux : P.Nvx, ny = P.Nuy > P.Nvy ? P.Nuy : P.Nvy;
  int rows = 16;
  auto grid = [&](int r) { return dim3((nx + BX - 1) / BX, (ny + BY * r - 1) / (BY * r)); };
  while (rows > 1 && (long long)grid(rows).x * grid(rows).y < 2LL * P.nsm) rows >>= 1;
  k_conservation<<<grid(rows), dim3(BX, BY), 0, s>>>(P, V, rows, red);
}

void launch_stage_cached(const double *kV0, const double *Vn, double aii, double inv_dt, double *Wt, long long n,
                         cudaStream_t s) {
  long long b = (n + 255) / 256;
  if (b > 148 * 32) b = 148 * 32;
  k_stage_cached<<<(unsigned)b, 256, 0, s>>>(kV0, Vn, aii, inv_dt, Wt, n);
}

void launch_add(const double *x, double *y, long long n, cudaStream_t s) {
  long long b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  k_add<<<(unsigned)b, 256, 0, s>>>(x, y, n);
}

}  // namespace ins2d

namespace ins2d {

void cell_tiles(const DevOps &P, int member, std::vector<int4> &out) {
  const int nx = std::max(P.Npx, std::max(P.Nux, P.Nvx)), ny = std::max(P.Npy, std::max(P.Nuy, P.Nvy));
  for (int by = 0; by < (ny + BY - 1) / BY; ++by)
    for (int bx = 0; bx < (nx + BX - 1) / BX; ++bx) out.push_back(make_int4(member, bx, by, 0));
}

void launch_div_ens(const EnsMemberD *mem, const int4 *tiles, int n, int mode, double gamma, cudaStream_t s) {
  if (n > 0) k_div_ens<<<n, dim3(BX, BY), 0, s>>>(mem, tiles, mode, gamma);
}

void launch_project_ens(const EnsMemberD *mem, const int4 *tiles, int n, double c, int from_p, int last,
                        const EnsCg *cg, cudaStream_t s) {
  if (n > 0) k_project_ens<<<n, dim3(BX, BY), 0, s>>>(mem, tiles, c, from_p, last, cg);
}

void launch_stage_cached_ens(const EnsMemberD *mem, const int4 *tiles, int n, double aii, cudaStream_t s) {
  if (n > 0) k_stage_cached_ens<<<n, dim3(BX, BY), 0, s>>>(mem, tiles, aii);
}

}  // namespace ins2d
