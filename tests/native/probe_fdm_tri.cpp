// Test-only: the separable inverse's tables (fdm_host.hpp, FdmTri) applied on
// the host in the order the device kernels use them.
#include <cmath>
#include <vector>

#include "fdm_host.hpp"

using namespace ins2d;

// z = A^+ r for r as ny x nx rows; out = {xmodes, null_mode, cyclic}
extern "C" void probe_fdm_tri_apply(void *h, const double *r, double *z, int *out) {
  const HostOps &H = *(const HostOps *)h;
  const FdmTri F = fdm_tri(H.TX, H.hx, H.TY, H.hy);
  const int nm = F.nm, n = F.n, nx = H.Npx;
  out[0] = F.xmodes;
  out[1] = F.null_mode;
  out[2] = !F.g.empty();
  auto at = [&](int m, int s) { return F.xmodes ? (size_t)s * nx + m : (size_t)m * nx + s; };
  std::vector<double> y(n), Z((size_t)nm * n);
  for (int b = 0; b < nm; ++b) {
    const double *p = &F.piv[(size_t)b * n];
    double sum = 0.0, part = 0.0;
    for (int s = 0; s < n; ++s) {
      double w = 0.0;
      for (int m = 0; m < nm; ++m) w += F.Q[(size_t)m * nm + b] * r[at(m, s)];
      y[s] = w;
      sum += w;
      if (b == F.null_mode) part += F.nmu[s] * w;
    }
    const bool null = b == F.null_mode;
    for (int s = 0; s < n; ++s) y[s] = -(y[s] + (s ? F.e[s - 1] * y[s - 1] : 0.0)) * p[s];
    for (int s = n - 2; s >= 0; --s) y[s] -= F.e[s] * p[s] * y[s + 1];
    if (!null && !F.g.empty()) part = y[0] + F.cr[b] * y[n - 1];
    for (int s = 0; s < n; ++s)
      Z[(size_t)b * n + s] = y[s] - (null ? part + sum * F.ng[s] : (F.g.empty() ? 0.0 : part * F.g[(size_t)b * n + s]));
  }
  for (int m = 0; m < nm; ++m)
    for (int s = 0; s < n; ++s) {
      double v = 0.0;
      for (int b = 0; b < nm; ++b) v += F.Q[(size_t)m * nm + b] * Z[(size_t)b * n + s];
      z[at(m, s)] = v;
    }
}
