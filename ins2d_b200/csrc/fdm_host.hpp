// Host side of the fast-diagonalization preconditioner (fdm.cu): the
// generalized eigen-decompositions of the 1D factors of the pressure matrix.
#pragma once

#include <vector>

#include "setup.hpp"

namespace ins2d {

// T q = lambda diag(h) q for a symmetric positive semidefinite n x n matrix
// T: Q (row-major, Q[i*n + a] = q_a(i)) with Q' diag(h) Q = I, lam ascending.
struct FdmHost1D {
  int n = 0;
  std::vector<double> Q, lam;
};
FdmHost1D fdm_1d(const Table &T, const std::vector<double> &h);

// Data of the separable inverse with ONE diagonalized direction: with the
// eigenbasis Q of the mode direction (T_m Q = diag(h_m) Q diag(lam)),
//   A z = r  <=>  (T_s + lam_b diag(h_s)) zh_b = -(Q' r)_b for every mode b,
//   z = Q zh,
// a tridiagonal system of n unknowns per mode (cyclic in a periodic direction).
// piv holds the reciprocal pivots of its elimination, so the device only
// runs two first-order recurrences per system (fdm_tri.cuh).
struct FdmTri {
  bool xmodes = false;  // modes along x and systems along y, or the other way round
  int nm = 0, n = 0;    // modes, unknowns of a system
  std::vector<double> Q, lam;  // nm x nm (Q[i*nm + b]), ascending
  std::vector<double> h;       // cell widths of the system's direction (n)
  std::vector<double> e;       // T_s(i, i+1), zero from n - 1 on (n rounded up to 8)
  std::vector<double> piv;     // nm x n reciprocal pivots
  // cyclic systems (Sherman-Morrison): zh = y - (y_0 + cr_b y_{n-1}) g_b
  std::vector<double> g, cr;   // nm x n and nm, empty when not cyclic
  // mode whose system is singular (closed and periodic domains; -1: none):
  // its right-hand side is made consistent and the h-weighted mean of its
  // solution removed, i.e. the null mode is left out.  With y the elimination
  // that sets the last unknown to zero, both are rank-one corrections:
  //   zh = y - sum(w) ng - (nmu' w),  ng, nmu of n values
  int null_mode = -1;
  std::vector<double> ng, nmu;
};
// the mode direction is the one with fewer cells (fewer operations)
FdmTri fdm_tri(const Table &TX, const std::vector<double> &hx, const Table &TY, const std::vector<double> &hy);

// Eigen-decomposition of a symmetric n x n matrix A (row-major, destroyed):
// A = V diag(w) V', V row-major (V[i*n + a] = component i of eigenvector a),
// w ascending.  Householder reduction to tridiagonal form, then the implicit
// QL iteration with Wilkinson-type shifts (Bowdler, Martin, Reinsch and
// Wilkinson's algorithm), eigenvectors accumulated.  Throws on no convergence.
void sym_eig(int n, std::vector<double> &A, std::vector<double> &V, std::vector<double> &w);

// largest 1D size for which the context builds the preconditioner (the
// set-up is O(n^3) on the host, the application two dense products and a
// batch of tridiagonal solves)
constexpr int kFdmMaxN = 1024;

}  // namespace ins2d
