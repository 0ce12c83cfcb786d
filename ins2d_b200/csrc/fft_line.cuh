// One-dimensional complex transforms of any length in shared memory, for the
// row and column passes of grids whose sides are no powers of two from 64 up
// (those have compile-time shapes, fft.cu).
//
// Lengths whose prime factors are at most kMaxFactor: mixed-radix Stockham
// passes (natural order in and out, ping-pong between two buffers): radix 8,
// 4, 2, 3, 5, 7 in registers, other primes by direct sums.  Other lengths:
// Bluestein's algorithm, a cyclic convolution with the chirp e^{i pi k^2 / n}
// of power-of-two length m >= 2n - 1.  Either way O(n log n) operations per
// line, where direct sums take n^2.  A pass is bound by its shared-memory
// round trip and barrier, so the passes are few and their reads contiguous.
// A prime of up to 127 is a pass of direct sums: one pass where Bluestein's
// algorithm takes two transforms of twice the length and three products (67 x 67
// solve 38.9 and 48.7 us, 113 x 113 46.3 and 49.1, 127 x 127 the same; with 31 for
// the limit 37 x 37 took 48.6 us instead of 34.4, plain sums over the line 39.1).
// Measured on B200 against direct sums: 1000 x 600 solve 2271 -> 54 us (rows
// 8.6 and 8.5 us, columns 18.6 us), 40 x 40 step on host arrays 225 -> 203 us.
#pragma once

#include "kernels.cuh"

namespace ins2d {

constexpr int kMaxFactor = 127;

// shared-memory slot of value i: eight lanes of 16-byte accesses a power of
// two apart fall on distinct banks
__host__ __device__ __forceinline__ int line_slot(int i) { return i + (i >> 3); }
__host__ __device__ __forceinline__ int line_ld(int m) { return line_slot(m - 1) + 1; }

__device__ __forceinline__ double2 c_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 c_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 c_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 c_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a

__device__ __forceinline__ double line_cos(int R, int q) {  // cos(2 pi q / R), sin below
  if (R == 3) return -0.5;
  if (R == 5) return (q == 1 || q == 4) ? 0.30901699437494742410 : -0.80901699437494742410;
  return (q == 1 || q == 6) ? 0.62348980185873353053
                            : ((q == 2 || q == 5) ? -0.22252093395631440429 : -0.90096886790241912624);
}
__device__ __forceinline__ double line_sin(int R, int q) {
  if (R == 3) return q == 1 ? 0.86602540378443864676 : -0.86602540378443864676;
  if (R == 5) {
    const double v = (q == 1 || q == 4) ? 0.95105651629515357212 : 0.58778525229247312917;
    return q <= 2 ? v : -v;
  }
  const double v = (q == 1 || q == 6) ? 0.78183148246802980871
                                      : ((q == 2 || q == 5) ? 0.97492791218182360702 : 0.43388373911755812048);
  return q <= 3 ? v : -v;
}

// forward DFT of R values in registers
template <int R>
__device__ __forceinline__ void line_dft(double2 (&x)[R]) {
  if constexpr (R == 2) {
    const double2 a = x[0];
    x[0] = c_add(a, x[1]);
    x[1] = c_sub(a, x[1]);
  } else if constexpr (R == 4) {
    const double2 a = c_add(x[0], x[2]), b = c_sub(x[0], x[2]), c = c_add(x[1], x[3]), d = c_mi(c_sub(x[1], x[3]));
    x[0] = c_add(a, c);
    x[1] = c_add(b, d);
    x[2] = c_sub(a, c);
    x[3] = c_sub(b, d);
  } else if constexpr (R == 8) {
    double2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    line_dft<4>(e);
    line_dft<4>(o);
    constexpr double r = 0.70710678118654752440;
    o[1] = make_double2((o[1].x + o[1].y) * r, (o[1].y - o[1].x) * r);
    o[2] = c_mi(o[2]);
    o[3] = make_double2((o[3].y - o[3].x) * r, -(o[3].x + o[3].y) * r);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = c_add(e[k], o[k]);
      x[k + 4] = c_sub(e[k], o[k]);
    }
  } else {  // 3, 5, 7: pairs j, R - j
    constexpr int H = (R - 1) / 2;
    double2 tp[H], tm[H];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      tp[j - 1] = c_add(x[j], x[R - j]);
      tm[j - 1] = c_sub(x[j], x[R - j]);
    }
    const double2 x0 = x[0];
#pragma unroll
    for (int j = 0; j < H; ++j) x[0] = c_add(x[0], tp[j]);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      double2 a = x0, b = make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 1; j <= H; ++j) {
        const double c = line_cos(R, (j * k) % R), s = line_sin(R, (j * k) % R);
        a.x += c * tp[j - 1].x;
        a.y += c * tp[j - 1].y;
        b.x += s * tm[j - 1].x;
        b.y += s * tm[j - 1].y;
      }
      b = c_mi(b);
      x[k] = c_add(a, b);
      x[R - k] = c_sub(a, b);
    }
  }
}

__device__ __forceinline__ unsigned fast_div(unsigned b, unsigned d, unsigned inv) {
  return d == 1 ? b : __umulhi(b, inv);
}

// One Stockham pass of radix R over `lines` lines (pitch ld) from a to b: with
// p = butterfly / s, q = butterfly mod s, values butterfly + k m/R become, times
// W_m^(p s k), values q + s (R p + k).
template <int R>
__device__ __forceinline__ void line_pass(const FftLine &L, int i, const double2 *a, double2 *b, int lines, int ld,
                                          const double2 *__restrict__ tw) {
  const unsigned nb = L.m / R, s = L.s[i], inv_s = L.inv_s[i], inv_b = L.inv_b[i];
  for (unsigned idx = threadIdx.x; idx < lines * nb; idx += blockDim.x) {
    const unsigned line = lines > 1 ? fast_div(idx, nb, inv_b) : 0u, u = idx - line * nb;
    const unsigned p = fast_div(u, s, inv_s), q = u - p * s;
    const double2 *A = a + line * ld;
    double2 *B = b + line * ld;
    double2 x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = A[line_slot(u + k * nb)];
    double2 w[R];
    const unsigned e = p * s;
#pragma unroll
    for (int k = 1; k < R; ++k) w[k] = __ldg(tw + e * k);
    line_dft<R>(x);
    const unsigned o = q + s * R * p;
    B[line_slot(o)] = x[0];
#pragma unroll
    for (int k = 1; k < R; ++k) B[line_slot(o + s * k)] = c_mul(x[k], w[k]);
  }
}
// the same for any odd radix by direct sums.  A thread forms outputs k and R - k
// of a butterfly together (their sums over the pairs j, R - j differ in a sign
// only): a quarter of the loads of one output per thread.
__device__ __forceinline__ void line_pass_any(const FftLine &L, int i, const double2 *a, double2 *b, int lines,
                                              int ld, const double2 *__restrict__ tw) {
  const unsigned R = L.r[i], nb = L.m / R, s = L.s[i], h = R / 2, per = nb * (h + 1);
  for (unsigned idx = threadIdx.x; idx < lines * per; idx += blockDim.x) {
    const unsigned line = lines > 1 ? idx / per : 0u, v = idx - line * per;
    const unsigned k = v / nb, u = v - k * nb;  // outputs k, R - k of butterfly u
    const unsigned p = fast_div(u, s, L.inv_s[i]), q = u - p * s;
    const double2 *A = a + line * ld;
    double2 *B = b + line * ld;
    const unsigned o = q + s * R * p;
    double2 x = A[line_slot(u)], y = make_double2(0.0, 0.0);
    unsigned jk = 0;
#pragma unroll 2
    for (unsigned j = 1; j <= h; ++j) {
      const double2 f = A[line_slot(u + j * nb)], g = A[line_slot(u + (R - j) * nb)];
      jk += k;
      if (jk >= R) jk -= R;
      const double2 w = __ldg(tw + jk * nb);  // cos, -sin
      x.x += w.x * (f.x + g.x);
      x.y += w.x * (f.y + g.y);
      y.x += w.y * (f.x - g.x);
      y.y += w.y * (f.y - g.y);
    }
    // x + i y and x - i y
    if (k == 0) {
      B[line_slot(o)] = x;
    } else {
      const unsigned e = p * s * k, m = R - k;
      B[line_slot(o + s * k)] = c_mul(make_double2(x.x - y.y, x.y + y.x), __ldg(tw + e));
      B[line_slot(o + s * m)] = c_mul(make_double2(x.x + y.y, x.y - y.x), __ldg(tw + p * s * m));
    }
  }
}

// the Stockham passes of `lines` lines in a (b: the other buffer); returns
// the buffer that holds the result.  Synchronised at the end.
__device__ __forceinline__ double2 *line_passes(const FftLine &L, double2 *a, double2 *b, int lines, int ld,
                                                const double2 *__restrict__ tw) {
  for (int i = 0; i < L.np; ++i) {
    switch (L.r[i]) {
      case 2: line_pass<2>(L, i, a, b, lines, ld, tw); break;
      case 3: line_pass<3>(L, i, a, b, lines, ld, tw); break;
      case 4: line_pass<4>(L, i, a, b, lines, ld, tw); break;
      case 5: line_pass<5>(L, i, a, b, lines, ld, tw); break;
      case 7: line_pass<7>(L, i, a, b, lines, ld, tw); break;
      case 8: line_pass<8>(L, i, a, b, lines, ld, tw); break;
      default: line_pass_any(L, i, a, b, lines, ld, tw); break;
    }
    __syncthreads();
    double2 *t = a;
    a = b;
    b = t;
  }
  return a;
}

// Forward DFT of `lines` lines of n values (slots line_slot(k) of a, pitch
// ld = line_ld(m)); the caller synchronised after writing them.  Returns the
// buffer with the result in natural order, synchronised.  An inverse transform
// is the forward one between exchanges of real and imaginary parts.
__device__ __forceinline__ double2 *line_transform(const FftLine &L, double2 *a, double2 *b, int lines, int ld,
                                                   const double2 *__restrict__ tab) {
  if (L.m == L.n) return line_passes(L, a, b, lines, ld, tab);
  // Bluestein: W^(jk) = c_j c_k / c_(k-j), c_k = e^{-i pi k^2/n}; tables: the
  // passes' twiddles (m), the chirp c (n), the transformed filter (m/2 + 1
  // values of a symmetric sequence)
  const double2 *chirp = tab + L.m, *filt = chirp + L.n;
  for (int line = 0; line < lines; ++line) {
    double2 *A = a + line * ld;
    for (int k = threadIdx.x; k < L.m; k += blockDim.x)
      A[line_slot(k)] = k < L.n ? c_mul(A[line_slot(k)], __ldg(chirp + k)) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  double2 *c = line_passes(L, a, b, lines, ld, tab);
  double2 *d = c == a ? b : a;
  for (int line = 0; line < lines; ++line) {
    double2 *A = c + line * ld;
    for (int k = threadIdx.x; k < L.m; k += blockDim.x) {
      const double2 v = c_mul(A[line_slot(k)], __ldg(filt + (2 * k <= L.m ? k : L.m - k)));
      A[line_slot(k)] = make_double2(v.y, v.x);
    }
  }
  __syncthreads();
  double2 *e = line_passes(L, c, d, lines, ld, tab);
  const double sc = 1.0 / L.m;
  for (int line = 0; line < lines; ++line) {
    double2 *A = e + line * ld;
    for (int k = threadIdx.x; k < L.n; k += blockDim.x) {
      const double2 v = A[line_slot(k)];
      A[line_slot(k)] = c_mul(make_double2(v.y * sc, v.x * sc), __ldg(chirp + k));
    }
  }
  __syncthreads();
  return e;
}

}  // namespace ins2d
