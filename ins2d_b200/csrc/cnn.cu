// The learned initial guess of the pressure solve: a six-layer 3x3
// convolutional network trained on the solver's own (right-hand side,
// pressure) pairs.  There is no counterpart in the reference (its solves start
// from zero, pressure_poisson.m:61-70); the network only changes where CG
// starts, never the stopping rule.
//
// Layout: activations NHWC on the pressure grid (pixel (i,j) at j*Npx + i,
// x fastest, then the 32 channels of the pixel: 64 bytes of BF16), a batch of
// B fields one after another.  Master weights are FP32 in one flat vector:
//   W1 [32 co][9 t]            (1 -> 32)
//   W2..W5 [32 co][9 t][32 ci] (32 -> 32, ReLU after each)
//   W6 [9 t][32 ci]            (32 -> 1, scaled by out_scale)
// with t = (dy+1)*3 + (dx+1) and out(p) = sum_t W[t] in(p + (dx,dy)) (zero
// padding).  Rounding points (the oracle emulates them): layer outputs 1..5
// and the gradients dZ1..dZ5 are stored as BF16 (round to nearest even);
// everything else is FP32.
//
// Tensor cores: the 32 -> 32 layers are implicit GEMMs on BF16 tensor cores
// with FP32 accumulators:
//   forward        Z[p][co]   = sum_{t,ci} W[co][t][ci] A[p+t][ci]    M = pixels, N = 32, K = 288
//   backward-data  dA[p][ci]  = sum_{t,co} W[co][8-t][ci] dZ[p+t][co] (the same kernel, transposed weights)
//   weight grad    dW[co][t,ci] = sum_p dZ[p][co] A[p+t][ci]          M = 32, N = 288, K = pixels
// The default path runs on tcgen05.mma with TMEM accumulators: the first two by
// k_conv_row_tc (k_conv_mid_tc on narrow fields), the weight gradient by
// k_wgrad_tc, and the 32 -> 1 layer by k_conv_out_tc, whose FP32 weights are three
// BF16 parts each.  The other path runs on mma.sync m16n8k16 (k_conv_mid,
// k_wgrad_mid).  The 1 -> 32 layer, the edge layers' gradients (2 x 288 MACs per
// pixel), the losses (squared error; the residual loss with the context's operator tables),
// the solver's odd-part application and Adam are FP32 / FP64 CUDA-core kernels.
// Per pixel and 32 -> 32 layer the traffic is one read of the input activations
// and one write of the output (64 bytes each in BF16).
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <stdexcept>
#include <vector>

#include "cnn.cuh"
#include "ins2d.h"
#include "kernels.cuh"

namespace ins2d {
namespace cnn {

namespace {

using bf16 = __nv_bfloat16;

constexpr int TW = 16, TH = 8;             // output tile of the 32 -> 32 kernels
constexpr int HWD = TW + 2, HHT = TH + 2;  // halo tile
constexpr int PSTR = 40;                   // bf16 per halo pixel in shared memory (32 + 8: no bank conflicts)
constexpr int WSTR = kK + 8;               // bf16 per output channel of the shared weights
constexpr int kRedBlocks = 1184;           // capacity of the reduction partials (148 x 8)
constexpr int kWgBlocks = 592;             // weight-gradient blocks (148 x 4)

#define CK(x)                                                                                 \
  do {                                                                                        \
    cudaError_t e_ = (x);                                                                     \
    if (e_ != cudaSuccess) throw CudaError(std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ void unpack8(const uint4 &v, float (&o)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    o[2 * k] = __uint_as_float(w[k] << 16);
    o[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
}

// --- the edge layers (1 -> 32, 32 -> 1 and their gradients) ----------------------
// 288 FP32 multiply-adds per pixel against 64 bytes of its activations: bound
// by memory as long as neither weights nor window values cost a load per
// multiply-add.  So a thread owns one column of a tile and 8 of its 32
// channels, keeps the 72 weights (or weight-gradient sums) of those channels
// in registers, and walks down the column with a sliding 3 x 3 window of the
// one-channel field staged in shared memory: three shared loads and one
// 16-byte access of the activations per 72 multiply-adds.  Measured on B200,
// 4 fields of 512^2, against one thread per pixel (weights read from shared
// memory) and one thread per weight (pixels read one by one): layer 1 53 ->
// 29 us, layer 6 116 -> 42 us, dZ5 95 -> 45 us, weight gradients 1017 and
// 908 -> 36 us each.
constexpr int kEC = 64, kER = 16;    // columns (four threads each) and rows of a tile
constexpr int kEThreads = 4 * kEC;
constexpr int kEP = kEC + 4;         // pitch of the staged field
constexpr int kEBlocksPerSm = 2;

struct EdgeTile {
  int x0, y0;
  long long f;  // first pixel of the field
};
__device__ __forceinline__ EdgeTile edge_tile(long long tile, int tiles_x, int tiles_y, int step_x, int H, int W) {
  EdgeTile t;
  const long long per = (long long)tiles_x * tiles_y;
  const int b = (int)(tile / per), rem = (int)(tile - b * per);
  t.y0 = (rem / tiles_x) * kER;
  t.x0 = (rem % tiles_x) * step_x;
  t.f = (long long)b * H * W;
  return t;
}
// the field's rows y0 - 1 .. y0 + kER, columns x0 - 1 .. x0 + kEC, zero outside
__device__ __forceinline__ void stage_field(const float *__restrict__ s, const EdgeTile &t, int H, int W,
                                            float (*st)[kEP]) {
  for (int i = threadIdx.x; i < (kER + 2) * (kEC + 2); i += kEThreads) {
    const int r = i / (kEC + 2), c = i - r * (kEC + 2);
    const int y = t.y0 - 1 + r, x = t.x0 - 1 + c;
    st[r][c] = (y >= 0 && y < H && x >= 0 && x < W) ? __ldg(s + t.f + (long long)y * W + x) : 0.0f;
  }
}

// out[p][c] = BF16 of sum_t w[c][t] s[p + t] with ReLU (MODE 0: layer 1), or of
// (sum_t W6[t][c] s[p - t]) [mask[p][c] > 0] (MODE 1: dZ5 from dy)
template <int MODE>
__global__ void __launch_bounds__(kEThreads, kEBlocksPerSm)
    k_expand(const float *__restrict__ s, const float *__restrict__ w, const bf16 *__restrict__ mask,
             bf16 *__restrict__ out, int B, int H, int W, int tiles_x, int tiles_y) {
  pdl_wait();
  pdl_trigger();
  __shared__ float st[kER + 2][kEP];
  const int cg = threadIdx.x & 3, col = threadIdx.x >> 2;
  float wr[8][kTaps];  // [channel][tap of s[p + tap]]
#pragma unroll
  for (int e = 0; e < 8; ++e)
#pragma unroll
    for (int t = 0; t < kTaps; ++t)
      wr[e][t] = MODE == 0 ? __ldg(w + (8 * cg + e) * kTaps + t) : __ldg(w + (kTaps - 1 - t) * kC + 8 * cg + e);
  const long long ntiles = (long long)B * tiles_x * tiles_y;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const EdgeTile t = edge_tile(tile, tiles_x, tiles_y, kEC, H, W);
    __syncthreads();
    stage_field(s, t, H, W, st);
    __syncthreads();
    const int x = t.x0 + col;
    if (x >= W) continue;
    float a[kTaps];
#pragma unroll
    for (int k = 0; k < 6; ++k) a[3 + k] = st[k / 3][col + k % 3];
    const int rows = min(kER, H - t.y0);
#pragma unroll 2
    for (int r = 0; r < rows; ++r) {
#pragma unroll
      for (int k = 0; k < 6; ++k) a[k] = a[k + 3];
#pragma unroll
      for (int k = 0; k < 3; ++k) a[6 + k] = st[r + 2][col + k];
      const long long pix = t.f + (long long)(t.y0 + r) * W + x;
      float m[8];
      if (MODE == 1) unpack8(__ldg(reinterpret_cast<const uint4 *>(mask + pix * kC + 8 * cg)), m);
      float z[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        z[e] = 0.0f;
#pragma unroll
        for (int q = 0; q < kTaps; ++q) {
          const int k = MODE == 0 ? q : kTaps - 1 - q;  // the sums' order of the taps
          z[e] = fmaf(wr[e][k], a[k], z[e]);
        }
        if (MODE == 0)
          z[e] = fmaxf(z[e], 0.0f);
        else if (!(m[e] > 0.0f))
          z[e] = 0.0f;
      }
      *reinterpret_cast<uint4 *>(out + pix * kC + 8 * cg) =
          make_uint4(pack2(z[0], z[1]), pack2(z[2], z[3]), pack2(z[4], z[5]), pack2(z[6], z[7]));
    }
  }
}

// layer 6: y[p] = scale sum_t sum_c W6[t][c] a5[p + t][c].  Tiles of kEC - 2
// output columns: a thread walks one input column, forms its 9 tap sums over
// 8 channels and keeps, per dx, the running sums of the rows it contributes
// to; four threads' channels by shuffles, the three columns of an output
// through shared memory (two alternating rows, one barrier per row).
__global__ void __launch_bounds__(kEThreads, kEBlocksPerSm)
    k_conv_out(const bf16 *__restrict__ a5, const float *__restrict__ w6, float scale, float *__restrict__ y, int B,
               int H, int W, int tiles_x, int tiles_y) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sv[2][3][kEC];
  const int cg = threadIdx.x & 3, col = threadIdx.x >> 2;
  float wr[kTaps][8];
#pragma unroll
  for (int t = 0; t < kTaps; ++t)
#pragma unroll
    for (int e = 0; e < 8; ++e) wr[t][e] = __ldg(w6 + t * kC + 8 * cg + e);
  const long long ntiles = (long long)B * tiles_x * tiles_y;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const EdgeTile t = edge_tile(tile, tiles_x, tiles_y, kEC - 2, H, W);
    const int x = t.x0 - 1 + col;  // this thread's input column
    const bool xin = x >= 0 && x < W;
    float up[3] = {0.0f, 0.0f, 0.0f}, mid[3] = {0.0f, 0.0f, 0.0f};  // rows r - 1 and r without their later taps
    const int rows = min(kER, H - t.y0);
#pragma unroll 2
    for (int r = -1; r <= rows; ++r) {
      const int yy = t.y0 + r;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (xin && yy >= 0 && yy < H)
        v = __ldg(reinterpret_cast<const uint4 *>(a5 + (t.f + (long long)yy * W + x) * kC + 8 * cg));
      float a[8], q[kTaps];
      unpack8(v, a);
#pragma unroll
      for (int k = 0; k < kTaps; ++k) {
        q[k] = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) q[k] = fmaf(wr[k][e], a[e], q[k]);
      }
      float o[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        o[k] = up[k] + q[6 + k];  // row r - 1: this row is its dy = +1
        up[k] = mid[k] + q[3 + k];
        mid[k] = q[k];
        o[k] += __shfl_xor_sync(0xffffffffu, o[k], 1);
        o[k] += __shfl_xor_sync(0xffffffffu, o[k], 2);
      }
      if (r < 1) continue;  // row r - 1 >= 0 of the tile
      if (cg == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) sv[r & 1][k][col] = o[k];
      __syncthreads();
      const int oc = threadIdx.x;
      if (oc < kEC - 2 && t.x0 + oc < W)
        y[t.f + (long long)(yy - 1) * W + t.x0 + oc] =
            scale * (sv[r & 1][0][oc] + sv[r & 1][1][oc + 1] + sv[r & 1][2][oc + 2]);
    }
    __syncthreads();
  }
}

// the part of g[c][t] below of the calling block's tiles, tap by tap
__device__ __noinline__ float wgrad_edge_sum(const bf16 *__restrict__ xv, const float *__restrict__ s, int c, int t,
                                             int B, int H, int W, int tiles_x, int tiles_y) {
  const int dx = t % 3 - 1, dy = t / 3 - 1;
  const long long ntiles = (long long)B * tiles_x * tiles_y;
  float v = 0.0f;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const EdgeTile e = edge_tile(tile, tiles_x, tiles_y, kEC, H, W);
    for (int y = max(e.y0, -dy); y < min(e.y0 + kER, H - max(dy, 0)); ++y)
      for (int x = max(e.x0, -dx); x < min(e.x0 + kEC, W - max(dx, 0)); ++x) {
        const long long p = e.f + (long long)y * W + x;
        v = fmaf(__bfloat162float(xv[p * kC + c]), __ldg(s + p + (long long)dy * W + dx), v);
        if (isnan(v)) return v;  // whatever follows
      }
  }
  return v;
}

// Weight gradients of the edge layers: g[c][t] = sum_p x[p][c] s[p + t], one
// partial sum per block at part[t' * 32 + c]; LAYER 1: x = dZ1, s = in, t' = t;
// LAYER 6: x = A5, s = dy, t' = 8 - t (dW6[t][c] = sum_p dy[p] A5[p + t][c]).
// Taps outside the field are staged zeros, which make NaN of an infinite x: a
// sum that is NaN is formed again without them.
template <int LAYER>
__global__ void __launch_bounds__(kEThreads, kEBlocksPerSm)
    k_wgrad_edge(const bf16 *__restrict__ xv, const float *__restrict__ s, float *__restrict__ part, int B, int H,
                 int W, int tiles_x, int tiles_y) {
  pdl_wait();
  pdl_trigger();
  __shared__ float st[kER + 2][kEP];
  __shared__ float red[kEThreads / 32][kK];
  const int cg = threadIdx.x & 3, col = threadIdx.x >> 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float acc[8][kTaps] = {};
  const long long ntiles = (long long)B * tiles_x * tiles_y;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const EdgeTile t = edge_tile(tile, tiles_x, tiles_y, kEC, H, W);
    __syncthreads();
    stage_field(s, t, H, W, st);
    __syncthreads();
    const int x = t.x0 + col;
    if (x >= W) continue;
    float a[kTaps];
#pragma unroll
    for (int k = 0; k < 6; ++k) a[3 + k] = st[k / 3][col + k % 3];
    const int rows = min(kER, H - t.y0);
    const bf16 *src = xv + (t.f + (long long)t.y0 * W + x) * kC + 8 * cg;
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
#pragma unroll
      for (int k = 0; k < 6; ++k) a[k] = a[k + 3];
#pragma unroll
      for (int k = 0; k < 3; ++k) a[6 + k] = st[r + 2][col + k];
      float v[8];
      unpack8(__ldg(reinterpret_cast<const uint4 *>(src + (long long)r * W * kC)), v);
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int k = 0; k < kTaps; ++k) acc[e][k] = fmaf(v[e], a[k], acc[e][k]);
    }
  }
  // the eight columns of a warp, then the warps, in a fixed order
#pragma unroll
  for (int e = 0; e < 8; ++e)
#pragma unroll
    for (int k = 0; k < kTaps; ++k) {
      float v = acc[e][k];
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane < 4) red[warp][(LAYER == 1 ? k : kTaps - 1 - k) * kC + 8 * cg + e] = v;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < kK; i += kEThreads) {
    float v = 0.0f;
#pragma unroll
    for (int q = 0; q < kEThreads / 32; ++q) v += red[q][i];
    if (isnan(v)) v = wgrad_edge_sum(xv, s, i % kC, LAYER == 1 ? i / kC : kTaps - 1 - i / kC, B, H, W, tiles_x, tiles_y);
    part[(long long)blockIdx.x * kK + i] = v;
  }
}

// 32 bytes to and from global memory in one instruction
__device__ __forceinline__ void ldg32(const void *p, uint32_t (&r)[8]) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void stg32(void *p, const uint32_t (&r)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// 32 accumulators of a pixel -> BF16: ReLU, or the mask of the layer's
// activation.  A lane holds a whole pixel (64 bytes): 16-byte stores write each
// sector in two halves, 32-byte ones (pixels are 64-byte aligned) 8 us a layer
// faster for 4 fields of 512^2.
template <int MODE>
__device__ __forceinline__ void store_mid(const uint32_t (&r)[2][16], const uint32_t (&mk)[2][8], bf16 *out) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v0 = __uint_as_float(r[q][2 * j]), v1 = __uint_as_float(r[q][2 * j + 1]);
      if (MODE == 0) {
        v0 = fmaxf(v0, 0.0f);
        v1 = fmaxf(v1, 0.0f);
      } else {
        const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(&mk[q][j]);
        if (!(__low2float(m) > 0.0f)) v0 = 0.0f;
        if (!(__high2float(m) > 0.0f)) v1 = 0.0f;
      }
      o[j] = pack2(v0, v1);
    }
    stg32(out + 16 * q, o);
  }
}

// --- 32 -> 32 on tensor cores ---------------------------------------------------
// One block: a 16 x 8 pixel tile of one field; warp w computes tile row w
// (M = 16 pixels) for all 32 output channels (4 n-tiles of 8), K = 9 taps x
// 32 input channels in 18 steps of 16.  The halo tile and the weights sit in
// shared memory with padded strides so that the 32-bit fragment loads of a
// warp hit 32 different banks.
// MODE 0: out = bf16(ReLU(Z)).  MODE 1 (backward-data): out = bf16(Z * [mask > 0]).
template <int MODE>
__global__ void __launch_bounds__(256) k_conv_mid(const bf16 *__restrict__ in, const bf16 *__restrict__ wt,
                                                  const bf16 *__restrict__ mask, bf16 *__restrict__ out, int H,
                                                  int W) {
  pdl_wait();
  pdl_trigger();
  __shared__ __align__(16) bf16 sin_[HHT * HWD * PSTR];
  __shared__ __align__(16) bf16 sw[kC * WSTR];
  const int tid = threadIdx.x;
  const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;
  const long long fbase = (long long)blockIdx.z * H * W;
  for (int i = tid; i < kC * (kK / 8); i += 256) {
    const int co = i / (kK / 8), ch = i % (kK / 8);
    *reinterpret_cast<uint4 *>(&sw[co * WSTR + ch * 8]) = *reinterpret_cast<const uint4 *>(&wt[co * kK + ch * 8]);
  }
  for (int i = tid; i < HHT * HWD * 4; i += 256) {
    const int hp = i >> 2, part = i & 3;
    const int gy = y0 - 1 + hp / HWD, gx = x0 - 1 + hp % HWD;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (gy >= 0 && gy < H && gx >= 0 && gx < W)
      v = *reinterpret_cast<const uint4 *>(&in[(fbase + (long long)gy * W + gx) * kC + part * 8]);
    *reinterpret_cast<uint4 *>(&sin_[hp * PSTR + part * 8]) = v;
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  float acc[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[nt][k] = 0.0f;
#pragma unroll
  for (int tap = 0; tap < kTaps; ++tap) {
    const bf16 *rowp = &sin_[((warp + tap / 3) * HWD + tap % 3) * PSTR];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int kc = h * 16 + 2 * t4;
      const uint32_t a0 = *reinterpret_cast<const uint32_t *>(&rowp[g * PSTR + kc]);
      const uint32_t a1 = *reinterpret_cast<const uint32_t *>(&rowp[(g + 8) * PSTR + kc]);
      const uint32_t a2 = *reinterpret_cast<const uint32_t *>(&rowp[g * PSTR + kc + 8]);
      const uint32_t a3 = *reinterpret_cast<const uint32_t *>(&rowp[(g + 8) * PSTR + kc + 8]);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const bf16 *wp = &sw[(nt * 8 + g) * WSTR + tap * kC + kc];
        const uint32_t b0 = *reinterpret_cast<const uint32_t *>(wp);
        const uint32_t b1 = *reinterpret_cast<const uint32_t *>(wp + 8);
        mma_bf16(acc[nt], a0, a1, a2, a3, b0, b1);
      }
    }
  }
  const int y = y0 + warp;
  if (y >= H) return;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int x = x0 + g + 8 * half;
    if (x >= W) continue;
    const long long pix = fbase + (long long)y * W + x;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int ch = nt * 8 + 2 * t4;
      float v0 = acc[nt][2 * half], v1 = acc[nt][2 * half + 1];
      if (MODE == 0) {
        v0 = fmaxf(v0, 0.0f);
        v1 = fmaxf(v1, 0.0f);
      } else {
        const uint32_t m = *reinterpret_cast<const uint32_t *>(&mask[pix * kC + ch]);
        if (!(__uint_as_float(m << 16) > 0.0f)) v0 = 0.0f;
        if (!(__uint_as_float(m & 0xffff0000u) > 0.0f)) v1 = 0.0f;
      }
      *reinterpret_cast<uint32_t *>(&out[pix * kC + ch]) = pack2(v0, v1);
    }
  }
}

// --- 32 -> 32 on the 5th-generation tensor cores (tcgen05, TMEM accumulators) --------
// Persistent blocks, two per SM, with one role per warp: four producer warps
// stage halo tiles, one thread issues the MMAs, eight warps turn accumulators
// into BF16 outputs; tiles pass through mbarriers (kTcStages halo buffers,
// two pairs of accumulators), so loads, MMAs and stores of different tiles
// overlap.  A tile is 16 x 16 pixels, two MMA rows of M = 128 (pixel columns
// 0-7 and 8-15, m = py * 8 + px).  Its 18 x 18 halo lies in shared memory as
// four channel planes (plane c8 holds channels 8 c8 .. 8 c8 + 7 of every halo
// pixel, 16 bytes per pixel).  That is the canonical K-major layout without
// swizzle for every tap at once: a core matrix is 8 consecutive pixels of one
// row (16 bytes apart), the next row is kTcSbo bytes further, the next 8
// channels kTcLbo bytes, and tap (dy, dx) only moves the start address by
// (18 dy + dx) * 16 bytes.  So the A operands of the 18 MMAs of K = 16 (9 taps
// x 2 channel halves, N = 32) are descriptors over one halo tile, with no
// im2col copy.  kTcLbo is 32 mod 128 bytes: the copies of a pixel's four
// planes fall on distinct banks.  The weights (B: 32 x 288; core matrices of 8
// output channels, next 8 input channels kBLbo bytes further) are loaded once
// per block.
// What bounds it: with N = 32 an MMA reads 5 KB of operands for 131072
// multiply-adds, 40 cycles of shared memory against 32 of arithmetic: 22 us for
// 4 fields of 512^2, beside 20 us for the 128 bytes per pixel of memory traffic
// and the producers' copies and fences (about 1300 cycles a tile row of warps).
// There on B200: all 256 threads of a block loading, waiting and storing in
// turn, five blocks per SM, 65 us (72 us with the mask); this form 41 and 46
// us.  Fields wide enough go by rows instead (k_conv_row_tc, 27.5 and 33 us).
constexpr int kTcM = 128;
constexpr int kTcT = 16;                        // tile: 16 x 16 pixels
constexpr int kTcH = kTcT + 2;
constexpr int kTcSbo = kTcH * 16;               // 288: next tile row
constexpr int kTcLbo = kTcH * kTcSbo + 96;      // 5280: next 8 channels (plane)
constexpr int kABytes = (kC / 8) * kTcLbo;      // 21120 per halo buffer
constexpr int kTcStages = 3;
constexpr int kBLbo = (kC / 8) * 128;           // 512: next 8 K-elements of B
constexpr int kBBytes = (kK / 8) * kBLbo;       // 18432
constexpr int kTcBars = 2 * kTcStages + 4;
// Dynamic shared memory: halo buffers, B, the mbarriers and the TMEM slot
constexpr int kTcSmem = kTcStages * kABytes + kBBytes + 8 * kTcBars + 16;
constexpr int kTcBlocksPerSm = 2;
constexpr int kTcEpi = 256, kTcProd = 128;      // epilogue threads first, then producers, then the MMA warp
constexpr int kTcThreads = kTcEpi + kTcProd + 32;
constexpr int kTcTmemCols = 4 * kC;             // two pairs of accumulators
constexpr int kTcChunks = (kTcH * kTcH * 4 + kTcProd - 1) / kTcProd;  // 16-byte copies per producer thread
static_assert(kTcLbo % 128 == 32 && kABytes % 128 == 0, "plane pitch");
// kind::f16 instruction descriptor: FP32 accumulate (bits 4-5 = 1), A and B
// BF16 (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at
// bits 24-28.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kC >> 3) << 17) |
                            ((uint32_t)(kTcM >> 4) << 24);
constexpr long long kTcWaitLimit = 1LL << 20;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// shared-memory matrix descriptor: start, leading (K) and stride (M/N) byte
// offsets in 16-byte units, descriptor version 1 (bit 46), no swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// an MMA from its descriptors' halves: the offsets of an unrolled sequence stay
// immediate 32-bit additions for the one thread that issues it
constexpr uint64_t kSwizzle64 = 4ull << 61;  // layout type, with 8 rows of 64 bytes as the core matrix
__device__ __forceinline__ void tc_mma_lo(uint32_t tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                          uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}\n" ::"r"(tmem),
      "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(acc)
      : "memory");
}
// 16-byte asynchronous copy global -> shared; src_bytes = 0 writes zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(addr), "r"(parity)
      : "memory");
  return done != 0;
}
// bounded wait for the completion of a phase
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
  for (long long k = 0; k < kTcWaitLimit; ++k)
    if (mbar_try(addr, parity)) return true;
  return false;
}
__device__ __forceinline__ void mbar_arrive(uint32_t addr) {
  asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.shared::cta.b64 s, [%0];\n\t}\n" ::"r"(addr) : "memory");
}
// one arrival for a converged warp, after all its lanes' work (an arrival per
// lane is a serial chain of shared-memory updates)
__device__ __forceinline__ void mbar_arrive_warp(uint32_t addr) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(addr);
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}
// a box of the activations (act_map) into shared memory from pixel x, row y of
// field b on; completes on bar (bytes announced by tma_expect)
__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap *map, int x, int y, int b, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];\n" ::"r"(dst),
      "l"(map), "r"(0), "r"(x), "r"(y), "r"(b), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 s, [%0], %1;\n\t}\n" ::"r"(bar), "r"(bytes)
               : "memory");
}
// 16 accumulator columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr)
      : "memory");
}

// MODE 0: out = bf16(ReLU(Z)).  MODE 1 (backward-data): out = bf16(Z * [mask > 0]).
// A wait that gives up sets *err; every role then leaves its loop (the others
// by their own limits) and the block frees its TMEM.
template <int MODE>
__global__ void __launch_bounds__(kTcThreads, kTcBlocksPerSm)
    k_conv_mid_tc(const bf16 *__restrict__ in, const bf16 *__restrict__ wt, const bf16 *__restrict__ mask,
                  bf16 *__restrict__ out, int B, int H, int W, int tiles_x, int tiles_y, unsigned *__restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sB = smem + kTcStages * kABytes;
  const uint32_t aBase = smem_u32(smem), bBase = smem_u32(sB), bars = bBase + kBBytes;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + kBBytes + 8 * kTcBars);
  const uint32_t full = bars, empty = bars + 8 * kTcStages, tfull = bars + 16 * kTcStages, tempty = tfull + 16;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // B: element (n = co, k) at (k / 8) * kBLbo + co * 16 + (k % 8) * 2
  for (int i = tid; i < kC * (kK / 8); i += kTcThreads) {
    const int co = i % kC, kc = i / kC;
    *reinterpret_cast<uint4 *>(sB + kc * kBLbo + co * 16) = *reinterpret_cast<const uint4 *>(&wt[co * kK + kc * 8]);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                 "r"(kTcTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int k = 0; k < kTcBars; ++k) {
      // full: the producer warps; empty and tfull: one commit; tempty: the epilogue warps
      const int count = k < kTcStages ? kTcProd / 32 : (k < 2 * kTcStages + 2 ? 1 : kTcEpi / 32);
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bars + 8 * k), "r"(count) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  pdl_wait();
  pdl_trigger();
  const uint32_t taddr = *tslot;
  const long long per_field = (long long)tiles_x * tiles_y;
  const long long ntiles = per_field * B;
  bool ok = true;
  if (tid < kTcEpi) {
    // lanes 32 (warp % 4) .. of the pair's accumulator warp / 4
    const int half = warp >> 2, m = 32 * (warp & 3) + lane;
    const int px = 8 * half + (m & 7), py = m >> 3;
    int it = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
      const int acc = it & 1;
      const int b = (int)(tile / per_field), rem = (int)(tile % per_field);
      const int gx = (rem % tiles_x) * kTcT + px, gy = (rem / tiles_x) * kTcT + py;
      const bool in_f = gx < W && gy < H;
      const long long pix = (long long)b * H * W + (long long)gy * W + gx;
      uint32_t mk[2][8];
      if (MODE == 1 && in_f)
#pragma unroll
        for (int q = 0; q < 2; ++q) ldg32(mask + pix * kC + 16 * q, mk[q]);
      ok = __all_sync(0xffffffffu, mbar_wait(tfull + 8 * acc, (it >> 1) & 1));  // the warp stays converged
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      uint32_t r[2][16];
      const uint32_t ta = taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(2 * kC * acc + kC * half);
      tmem_ld16(ta, r[0]);
      tmem_ld16(ta + 16, r[1]);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      mbar_arrive_warp(tempty + 8 * acc);
      if (in_f) store_mid<MODE>(r, mk, out + pix * kC);
    }
  } else if (tid < kTcEpi + kTcProd) {
    // chunk j of this thread: plane c8 of halo pixel hp0 + 32 j
    const int pt = tid - kTcEpi, c8 = pt & 3, hp0 = pt >> 2;
    int rel[kTcChunks];
#pragma unroll
    for (int j = 0; j < kTcChunks; ++j) {
      const int hp = hp0 + 32 * j;
      rel[j] = ((hp / kTcH) * W + hp % kTcH) * kC;
    }
    const uint32_t d0 = aBase + c8 * kTcLbo + hp0 * 16;
    int it = 0;
    auto publish = [&](int k) {  // tile k's copies by this thread are complete
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      mbar_arrive_warp(full + 8 * (k % kTcStages));
    };
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
      const int st = it % kTcStages;
      if (!(ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * st, ((it / kTcStages) & 1) ^ 1)))) break;
      const int b = (int)(tile / per_field), rem = (int)(tile % per_field);
      const int hx0 = (rem % tiles_x) * kTcT - 1, hy0 = (rem / tiles_x) * kTcT - 1;
      const bf16 *src = in + ((long long)b * H * W + (long long)hy0 * W + hx0) * kC + 8 * c8;
      const uint32_t dst = d0 + st * kABytes;
      if (hx0 >= 0 && hy0 >= 0 && hx0 + kTcH <= W && hy0 + kTcH <= H) {
#pragma unroll
        for (int j = 0; j < kTcChunks; ++j)
          if (hp0 + 32 * j < kTcH * kTcH) cp_async16(dst + 512 * j, src + rel[j], 16u);
      } else {
#pragma unroll
        for (int j = 0; j < kTcChunks; ++j) {
          const int hp = hp0 + 32 * j, gx = hx0 + hp % kTcH, gy = hy0 + hp / kTcH;
          const bool inside = gx >= 0 && gx < W && gy >= 0 && gy < H;
          if (hp < kTcH * kTcH) cp_async16(dst + 512 * j, inside ? src + rel[j] : in, inside ? 16u : 0u);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      if (it > 0) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        publish(it - 1);
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (ok && it > 0) publish(it - 1);
  } else if (lane == 0) {
    const uint64_t a0 = smem_desc(aBase, kTcLbo, kTcSbo), b0 = smem_desc(bBase, kBLbo, 128);
    const uint32_t alo = (uint32_t)a0, ahi = (uint32_t)(a0 >> 32), blo = (uint32_t)b0, bhi = (uint32_t)(b0 >> 32);
    int it = 0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
      const int st = it % kTcStages, acc = it & 1;
      if (!(ok = mbar_wait(full + 8 * st, (it / kTcStages) & 1))) break;
      if (!(ok = mbar_wait(tempty + 8 * acc, ((it >> 1) & 1) ^ 1))) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int ks = 0; ks < kK / 16; ++ks) {
          const int t = ks >> 1, h = ks & 1;
          tc_mma_lo(taddr + 2 * kC * acc + kC * half,
                    alo + st * (kABytes / 16) + 2 * h * (kTcLbo / 16) + (t / 3) * kTcH + t % 3 + 8 * half, ahi,
                    blo + 2 * ks * (kBLbo / 16), bhi, kIdesc, ks > 0 ? 1u : 0u);
        }
      tc_commit(empty + 8 * st);
      tc_commit(tfull + 8 * acc);
    }
    if (!ok && it > 0) mbar_wait(tfull + 8 * ((it - 1) & 1), ((it - 1) >> 1) & 1);  // MMAs in flight, before the TMEM is freed
  }
  if (!ok) atomicExch(err, 1u);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(kTcTmemCols) : "memory");
}

// --- 32 -> 32, 128 pixels of a row per MMA ------------------------------------------
// The tile kernel above spends an MMA on every tap; here one MMA does three.
// A is 128 consecutive pixels of one input row as a TMA copy leaves them: 64
// bytes per pixel with the 64-byte swizzle, core matrices of 8 pixels (512
// bytes); tap dx moves the start address by a pixel (the swizzle follows the
// address, so it moves along).  B stacks the three dy taps along N = 96: its
// products belong to three consecutive output rows, whose accumulators (32
// TMEM columns each) lie side by side in a ring of kRSlots rows.  Input row q
// of a strip takes 6 MMAs (3 dx x 2 channel halves) and one more to start
// output row q from zero; where the ring wraps an MMA splits in two, and the
// first and last two input rows take the N = 32 and 64 parts they need.  Rows,
// their accumulators and the unrolled MMA sequence share the index it %
// kRStages, so every offset is an immediate.  Blocks walk down strips of 128
// columns; one thread issues the copies, one the MMAs, and two groups of four
// warps turn alternate output rows into BF16.
// What bounds it: 7 KB of operands per MMA (N = 96) are 56 cycles, 13 us of the
// tensor core for 4 fields of 512^2; the memory traffic is 20 us, and about 7
// us pass before the first row and after the last.  On B200 (ReLU, mask):
// the tile kernel 51 and 55 us; rows staged by cp.async into planes of 8
// channels (no swizzle) 42 us, with every thread's proxy fence and arrival
// per row on the critical path; by TMA into such planes, 16 bytes at a time,
// 36 us; this form 27.5 and 33 us.
constexpr int kRM = 128;
constexpr int kRBytes = (kRM + 2) * 2 * kC;     // 8320 per input row
constexpr int kRRow = 9216;                     // staged, 1024-byte aligned
constexpr int kRStages = 8;
constexpr int kRSlots = kRStages;               // row it: stage and accumulator it % kRStages
constexpr int kRBLbo = 3 * kC * 16;             // 1536: next 8 K-elements of B
constexpr int kRBBytes = 3 * (kC / 8) * kRBLbo; // 18432
constexpr int kRBars = 2 * kRStages + 2 * kRSlots + 1;
constexpr int kRSmem = kRStages * kRRow + kRBBytes + 8 * kRBars + 16;
constexpr int kRTmemCols = kRSlots * kC;
constexpr uint32_t kRIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kRM >> 4) << 24);  // N is added
static_assert(kRRow >= kRBytes && kRRow % 1024 == 0, "the swizzle repeats every 512 bytes of address");
// Rows of 128 pixels or tiles of 16: by the pixels each computes, a tile's
// costing half as much again (4 fields of 512 rows: 64 columns 12.0 and 11.4 us,
// 96 columns 12.2 and 14.2, 512 columns 27.5 and 41).
inline bool by_rows(int W) { return 2 * ((W + kRM - 1) / kRM) * kRM < 3 * ((W + kTcT - 1) / kTcT) * kTcT; }
constexpr int kRThreads = kTcEpi + 64;          // epilogue warps, the producer's and the MMAs'

// the MMAs of an input row in stage PH that ends output row it - 2, continues
// it - 1 and starts it (slots PH - 2 .. PH of the ring)
template <int PH>
__device__ __forceinline__ void row_mmas(uint32_t taddr, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi) {
  constexpr int s0 = (PH + kRSlots - 2) % kRSlots, n1 = s0 + 3 <= kRSlots ? 3 : kRSlots - s0;
  auto mm = [&](int ks, int j, int cnt, int slot, uint32_t acc) {
    tc_mma_lo(taddr + kC * slot, alo + PH * (kRRow / 16) + 2 * (ks & 1) + 2 * kC / 16 * (ks >> 1), ahi,
              blo + 2 * ks * (kRBLbo / 16) + j * kC, bhi, kRIdesc | ((uint32_t)(cnt * (kC >> 3)) << 17), acc);
  };
  mm(0, 2, 1, PH, 0u);
  if (n1 == 1) {
    mm(0, 0, 1, s0, 1u);
    mm(0, 1, 1, 0, 1u);
  } else {
    mm(0, 0, 2, s0, 1u);
  }
#pragma unroll
  for (int ks = 1; ks < 6; ++ks) {
    mm(ks, 0, n1, s0, 1u);
    if (n1 < 3) mm(ks, n1, 3 - n1, 0, 1u);
  }
}

// MODE as k_conv_mid_tc; item = strip of 128 columns, rows [R chunk, R (chunk + 1))
template <int MODE>
__global__ void __launch_bounds__(kRThreads, kTcBlocksPerSm)
    k_conv_row_tc(const __grid_constant__ CUtensorMap in, const bf16 *__restrict__ wt, const bf16 *__restrict__ mask,
                  bf16 *__restrict__ out, int H, int W, int strips, int chunks, int R, int nitems,
                  unsigned *__restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sB = smem + kRStages * kRRow;
  const uint32_t aBase = smem_u32(smem), bBase = smem_u32(sB), bars = bBase + kRBBytes;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + kRBBytes + 8 * kRBars);
  const uint32_t full = bars, empty = bars + 8 * kRStages, tfull = bars + 16 * kRStages, tempty = tfull + 8 * kRSlots,
                 drain = tempty + 8 * kRSlots;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // B: column n = 32 j + co is tap row dy = 2 - j; element (n, k = 32 dx + ci)
  // at (k / 8) * kRBLbo + n * 16 + (k % 8) * 2
  for (int i = tid; i < kC * (kK / 8); i += kRThreads) {
    const int co = i % kC, r = i / kC, t = r >> 2, c8 = r & 3, dy = t / 3, dx = t % 3;
    *reinterpret_cast<uint4 *>(sB + (4 * dx + c8) * kRBLbo + ((2 - dy) * kC + co) * 16) =
        *reinterpret_cast<const uint4 *>(&wt[co * kK + t * kC + c8 * 8]);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                 "r"(kRTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int k = 0; k < kRBars; ++k) {
      // full: the producer; empty, tfull and drain: one commit; tempty: a group of epilogue warps
      const int te = 2 * kRStages + kRSlots;
      const int count = k >= te && k < te + kRSlots ? kTcEpi / 64 : 1;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bars + 8 * k), "r"(count) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  pdl_wait();
  pdl_trigger();
  const uint32_t taddr = *tslot;
  bool ok = true;
  // item -> field, first column and row, rows
  struct Item {
    int x0, y0, rows, b;
  };
  auto item_at = [&](int item) {
    const int sx = item % strips, r = item / strips, c = r % chunks, b = r / chunks;
    return Item{sx * kRM, c * R, min(R, H - c * R), b};
  };
  if (tid < kTcEpi) {
    const int group = warp >> 2, px = 32 * (warp & 3) + lane;
    int it = 0;  // input rows so far: output row k of an item is its slot's row it + k
    for (int item = blockIdx.x; ok && item < nitems; item += gridDim.x) {
      const Item t = item_at(item);
      const int gx = t.x0 + px;
      const int first = it;
      it += t.rows + 2;
      for (int k = first + ((first ^ group) & 1); k < it; k += 2) {
        const int slot = k & (kRSlots - 1);
        const bool in_f = gx < W && k - first < t.rows;  // the last two rows start no output
        const long long pix = ((long long)t.b * H + t.y0 + k - first) * W + gx;
        uint32_t mk[2][8];
        if (MODE == 1 && in_f)
#pragma unroll
          for (int q = 0; q < 2; ++q) ldg32(mask + pix * kC + 16 * q, mk[q]);
        ok = __all_sync(0xffffffffu, mbar_wait(tfull + 8 * slot, (k / kRSlots) & 1));  // the warp stays converged
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        uint32_t r[2][16];
        const uint32_t ta = taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(kC * slot);
        tmem_ld16(ta, r[0]);
        tmem_ld16(ta + 16, r[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        mbar_arrive_warp(tempty + 8 * slot);
        if (in_f) store_mid<MODE>(r, mk, out + pix * kC);
      }
    }
  } else if (warp == kTcEpi / 32) {
    if (elect_one()) {
      int it = 0;
      for (int item = blockIdx.x; ok && item < nitems; item += gridDim.x) {
        const Item t = item_at(item);
        for (int q = 0; q < t.rows + 2; ++q, ++it) {
          const int st = it % kRStages;
          if (!(ok = mbar_wait(empty + 8 * st, ((it / kRStages) & 1) ^ 1))) break;
          tma_expect(full + 8 * st, kRBytes);
          tma_box(aBase + st * kRRow, &in, t.x0 - 1, t.y0 - 1 + q, t.b, full + 8 * st);
        }
      }
      // the last copies have landed before the block leaves, whatever the other roles met
      for (int k = max(0, it - kRStages); k < it; ++k) ok &= mbar_wait(full + 8 * (k % kRStages), (k / kRStages) & 1);
    }
    ok = __all_sync(0xffffffffu, ok);
  } else {
    const bool leader = elect_one();
    const uint64_t a0 = smem_desc(aBase, 16, 8 * 2 * kC) | kSwizzle64, b0 = smem_desc(bBase, kRBLbo, 128);
    const uint32_t alo = (uint32_t)a0, ahi = (uint32_t)(a0 >> 32), blo = (uint32_t)b0, bhi = (uint32_t)(b0 >> 32);
    int it = 0;
    for (int item = blockIdx.x; ok && item < nitems; item += gridDim.x) {
      const int rows = item_at(item).rows;
      for (int q = 0; q < rows + 2; ++q, ++it) {
        const int ph = it & (kRSlots - 1), par = (it / kRSlots) & 1;
        ok = mbar_wait(full + 8 * ph, par) && mbar_wait(tempty + 8 * ph, par ^ 1);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (!leader) continue;
        if (q >= 2 && q < rows) {
          switch (ph) {
            case 0: row_mmas<0>(taddr, alo, ahi, blo, bhi); break;
            case 1: row_mmas<1>(taddr, alo, ahi, blo, bhi); break;
            case 2: row_mmas<2>(taddr, alo, ahi, blo, bhi); break;
            case 3: row_mmas<3>(taddr, alo, ahi, blo, bhi); break;
            case 4: row_mmas<4>(taddr, alo, ahi, blo, bhi); break;
            case 5: row_mmas<5>(taddr, alo, ahi, blo, bhi); break;
            case 6: row_mmas<6>(taddr, alo, ahi, blo, bhi); break;
            default: row_mmas<7>(taddr, alo, ahi, blo, bhi); break;
          }
        } else {  // one or two of the three output rows, an MMA each
          for (int j = max(2 - q, 0); j <= min(2, rows + 1 - q); ++j)
            for (int ks = 0; ks < 6; ++ks)
              tc_mma_lo(taddr + kC * ((ph + j + kRSlots - 2) & (kRSlots - 1)),
                        alo + ph * (kRRow / 16) + 2 * (ks & 1) + 2 * kC / 16 * (ks >> 1), ahi,
                        blo + 2 * ks * (kRBLbo / 16) + j * kC, bhi, kRIdesc | ((uint32_t)(kC >> 3) << 17),
                        j < 2 || ks > 0 ? 1u : 0u);
        }
        tc_commit(empty + 8 * ph);
        if (q >= 2) tc_commit(tfull + 8 * ((ph + kRSlots - 2) & (kRSlots - 1)));
      }
      if (!ok) break;
      if (!leader) continue;
      // the slots of the last two rows hold no output
      tc_commit(tfull + 8 * ((it + kRSlots - 2) & (kRSlots - 1)));
      tc_commit(tfull + 8 * ((it + kRSlots - 1) & (kRSlots - 1)));
    }
    if (!ok && leader) {  // MMAs in flight, before the TMEM is freed
      tc_commit(drain);
      mbar_wait(drain, 0);
    }
  }
  if (!ok) atomicExch(err, 1u);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(kRTmemCols) : "memory");
}

// --- 32 -> 1 on tensor cores (the default path) --------------------------------------
// y = scale sum_t sum_c W6[t][c] a5[p + t][c] with FP32 weights: each weight is
// the sum of three BF16 values (24 bits, exact up to its last), so one row of
// 128 pixels is two MMAs (K = 32 channels) with N = 32 columns: tap t's parts at
// 3 t .. 3 t + 2, products exact, sums in FP32.  An epilogue thread adds a
// pixel's parts, keeps per dx the running sums of the three rows it belongs to
// and exchanges the finished row's with its neighbours through shared memory.
// Rows come by TMA as in k_conv_row_tc; 126 outputs of 128 columns.  Bound by
// the epilogue's adds and barriers, near its 67 MB of reads (10 us) for 4 fields
// of 512^2: 15.5 us on B200, against 40 us on the FP32 cores (k_conv_out).
// Parts of an infinite activation cancel (or meet a zero part), and a weight
// beyond BF16's range has infinite parts: a result that is not finite is formed
// again from the FP32 weights (conv_out_pixel).
constexpr int kOStages = 4;                     // staged rows and accumulators
constexpr int kORow = kRM * 2 * kC;             // 8192
constexpr int kOBBytes = kC * kC * 2;
constexpr int kOW = kRM - 2;                    // output columns of a strip
constexpr int kOBars = 4 * kOStages + 1;
constexpr int kOSmem = kOStages * kORow + kOBBytes + 2 * 3 * kRM * 4 + 8 * kOBars + 16;
constexpr int kOThreads = 192, kOBlocksPerSm = 4;

// layer 6 at pixel (x, y) of the field at a: FP32 sums over the taps inside it
__device__ __noinline__ float conv_out_pixel(const bf16 *__restrict__ a, const float *__restrict__ w6, float scale,
                                             int x, int y, int H, int W) {
  float s = 0.0f;
  for (int t = 0; t < kTaps; ++t) {
    const int xx = x + t % 3 - 1, yy = y + t / 3 - 1;
    if (xx < 0 || xx >= W || yy < 0 || yy >= H) continue;
    const uint4 *p = reinterpret_cast<const uint4 *>(a + ((long long)yy * W + xx) * kC);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v[8];
      unpack8(__ldg(p + q), v);
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(__ldg(w6 + t * kC + 8 * q + e), v[e], s);
    }
    if (isnan(s)) break;  // whatever follows
  }
  return scale * s;
}

__global__ void __launch_bounds__(kOThreads, kOBlocksPerSm)
    k_conv_out_tc(const __grid_constant__ CUtensorMap a5, const bf16 *__restrict__ act, const float *__restrict__ w6,
                  float scale, float *__restrict__ y, int H, int W, int strips, int chunks, int R, int nitems,
                  unsigned *__restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sB = smem + kOStages * kORow;
  float(*sv)[3][kRM] = reinterpret_cast<float(*)[3][kRM]>(sB + kOBBytes);
  const uint32_t aBase = smem_u32(smem), bBase = smem_u32(sB), bars = bBase + kOBBytes + 2 * 3 * kRM * 4;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sB + kOBBytes + 2 * 3 * kRM * 4 + 8 * kOBars);
  const uint32_t full = bars, empty = bars + 8 * kOStages, tfull = bars + 16 * kOStages, tempty = bars + 24 * kOStages,
                 drain = bars + 32 * kOStages;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                 "r"(kOStages * kC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int k = 0; k < kOBars; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bars + 8 * k),
                   "r"(k >= 3 * kOStages && k < 4 * kOStages ? 4 : 1)
                   : "memory");  // tempty: the four epilogue warps
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // B: element (n = 3 t + part, k = c) at (c / 8) * 512 + n * 16 + (c % 8) * 2
  for (int i = tid; i < kC * kC; i += kOThreads) {
    const int n = i / kC, c = i % kC, t = n / 3, part = n % 3;
    float w = t < kTaps ? __ldg(w6 + t * kC + c) : 0.0f;
    for (int q = 0; q < part; ++q) w -= __bfloat162float(__float2bfloat16_rn(w));
    *reinterpret_cast<bf16 *>(sB + (c >> 3) * 512 + n * 16 + (c & 7) * 2) = __float2bfloat16_rn(w);
  }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t taddr = *tslot;
  pdl_wait();
  pdl_trigger();
  bool ok = true;
  int it = 0;  // rows so far: stage and accumulator it % kOStages
  struct Item {
    int x0, y0, rows, b;
  };
  auto item_at = [&](int item) {
    const int sx = item % strips, r = item / strips, c = r % chunks, b = r / chunks;
    return Item{sx * kOW, c * R, min(R, H - c * R), b};
  };
  if (warp < 4) {
    // a wait that gave up leaves the loop running without waits: the four
    // warps meet at every row's barrier
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
      const Item t = item_at(item);
      float up[3] = {0.0f, 0.0f, 0.0f}, mid[3] = {0.0f, 0.0f, 0.0f};  // rows q - 1 and q without their later taps
      float *dst = y + ((long long)t.b * H + t.y0) * W + t.x0 + tid;
      const bool store = tid < kOW && t.x0 + tid < W;
      for (int q = 0; q < t.rows + 2; ++q, ++it) {
        const int st = it % kOStages;
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(tfull + 8 * st, (it / kOStages) & 1));
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        uint32_t r[2][16];
        const uint32_t ta = taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)(kC * st);
        tmem_ld16(ta, r[0]);
        tmem_ld16(ta + 16, r[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        mbar_arrive_warp(tempty + 8 * st);
        float v[kTaps];
#pragma unroll
        for (int k = 0; k < kTaps; ++k) {
          auto d = [&](int n) { return __uint_as_float(r[n >> 4][n & 15]); };
          v[k] = (d(3 * k + 2) + d(3 * k + 1)) + d(3 * k);
        }
        float o[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          o[k] = up[k] + v[6 + k];  // this row is dy = +1 of output row q - 2
          up[k] = mid[k] + v[3 + k];
          mid[k] = v[k];
        }
        if (q < 2) continue;  // the same for all four warps
#pragma unroll
        for (int k = 0; k < 3; ++k) sv[it & 1][k][tid] = o[k];
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        if (store) {
          float s = scale * (sv[it & 1][0][tid] + sv[it & 1][1][tid + 1] + sv[it & 1][2][tid + 2]);
          if (!isfinite(s))
            s = conv_out_pixel(act + (long long)t.b * H * W * kC, w6, scale, t.x0 + tid, t.y0 + q - 2, H, W);
          dst[(long long)(q - 2) * W] = s;
        }
      }
    }
  } else if (warp == 4) {
    if (elect_one()) {
      for (int item = blockIdx.x; ok && item < nitems; item += gridDim.x) {
        const Item t = item_at(item);
        for (int q = 0; q < t.rows + 2; ++q, ++it) {
          const int st = it % kOStages;
          if (!(ok = mbar_wait(empty + 8 * st, ((it / kOStages) & 1) ^ 1))) break;
          tma_expect(full + 8 * st, kORow);
          tma_box(aBase + st * kORow, &a5, t.x0 - 1, t.y0 - 1 + q, t.b, full + 8 * st);
        }
      }
      // the last copies have landed before the block leaves, whatever the other roles met
      for (int k = max(0, it - kOStages); k < it; ++k) ok &= mbar_wait(full + 8 * (k % kOStages), (k / kOStages) & 1);
    }
    ok = __all_sync(0xffffffffu, ok);
  } else {
    const bool leader = elect_one();
    const uint64_t a0 = smem_desc(aBase, 16, 8 * 2 * kC) | kSwizzle64, b0 = smem_desc(bBase, 512, 128);
    const uint32_t alo = (uint32_t)a0, ahi = (uint32_t)(a0 >> 32), blo = (uint32_t)b0, bhi = (uint32_t)(b0 >> 32);
    for (int item = blockIdx.x; ok && item < nitems; item += gridDim.x) {
      const int rows = item_at(item).rows;
      for (int q = 0; q < rows + 2; ++q, ++it) {
        const int st = it % kOStages, par = (it / kOStages) & 1;
        ok = mbar_wait(full + 8 * st, par) && mbar_wait(tempty + 8 * st, par ^ 1);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (!leader) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          tc_mma_lo(taddr + kC * st, alo + st * (kORow / 16) + 2 * h, ahi, blo + 2 * h * (512 / 16), bhi, kIdesc, (uint32_t)h);
        tc_commit(empty + 8 * st);
        tc_commit(tfull + 8 * st);
      }
    }
    if (!ok && leader) {  // MMAs in flight, before the TMEM is freed
      tc_commit(drain);
      mbar_wait(drain, 0);
    }
  }
  if (!ok) atomicExch(err, 1u);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(kOStages * kC) : "memory");
}

// --- block reductions (fixed order: deterministic) ----------------------------
template <int NQ>
__device__ void block_sum(double (&v)[NQ], const bool (&is_max)[NQ], double *out) {
  __shared__ double sh[32][NQ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    for (int off = 16; off > 0; off >>= 1) {
      const double o = __shfl_down_sync(0xffffffffu, v[q], off);
      v[q] = is_max[q] ? fmax(v[q], o) : v[q] + o;
    }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) sh[warp][q] = v[q];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double a = sh[0][q];
      for (int w = 1; w < nw; ++w) a = is_max[q] ? fmax(a, sh[w][q]) : a + sh[w][q];
      out[q] = a;
    }
}

// out[q] = combination over rows of part[row * NQ + q] (one block, fixed order)
template <int NQ>
__global__ void k_finish(const double *__restrict__ part, int rows, const int max_mask, double *__restrict__ out) {
  pdl_wait();
  pdl_trigger();
  bool is_max[NQ];
  double v[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    is_max[q] = (max_mask >> q) & 1;
    v[q] = is_max[q] ? -INFINITY : 0.0;
  }
  for (int r = threadIdx.x; r < rows; r += blockDim.x)
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = is_max[q] ? fmax(v[q], part[r * NQ + q]) : v[q] + part[r * NQ + q];
  block_sum<NQ>(v, is_max, out);
}

// loss = sum (y - tgt)^2 / n; dy = dL/d(layer-6 output) = 2 (y - tgt) / n * scale
__global__ void __launch_bounds__(256) k_loss(const float *__restrict__ y, const float *__restrict__ tgt,
                                              float *__restrict__ dy, float gscale, long long n,
                                              double *__restrict__ part) {
  pdl_wait();
  pdl_trigger();
  double v[1] = {0.0};
  const bool mx[1] = {false};
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const float d = y[p] - tgt[p];
    dy[p] = gscale * d;
    v[0] += (double)d * d;
  }
  block_sum<1>(v, mx, part + blockIdx.x);
}

// The pressure Laplacian A = M Om^-1 G of a context (its 1D row tables, the
// form of lap() in device.cuh) applied to one FP32 field
__device__ __forceinline__ float lap_f(const DevOps &P, const float *__restrict__ f, int i, int j) {
  const int32_t *cx = P.TX.c + kT * i;
  const double *wx = P.TX.w + kT * i;
  const int32_t *cy = P.TY.c + kT * j;
  const double *wy = P.TY.w + kT * j;
  const long long row = (long long)j * P.Npx;
  const float sx = (float)__ldg(wx) * f[row + __ldg(cx)] + (float)__ldg(wx + 1) * f[row + __ldg(cx + 1)] +
                   (float)__ldg(wx + 2) * f[row + __ldg(cx + 2)];
  const float sy = (float)__ldg(wy) * f[(long long)__ldg(cy) * P.Npx + i] +
                   (float)__ldg(wy + 1) * f[(long long)__ldg(cy + 1) * P.Npx + i] +
                   (float)__ldg(wy + 2) * f[(long long)__ldg(cy + 2) * P.Npx + i];
  return -((float)__ldg(P.hy + j) * sx + (float)__ldg(P.hx + i) * sy);
}

// residual loss, pass 1: d = A y - diag(A) in per field (in = f / (diag(A) s),
// so diag(A) in = f / s); partial sums of d^2
__global__ void __launch_bounds__(256) k_res_loss(const __grid_constant__ DevOps P, const float *__restrict__ y,
                                                  const float *__restrict__ in, float *__restrict__ d, int B,
                                                  double *__restrict__ part) {
  double v[1] = {0.0};
  const bool mx[1] = {false};
  const long long n = (long long)B * P.Np;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const long long b = k / P.Np, kk = k % P.Np;
    const int i = (int)(kk % P.Npx), j = (int)(kk / P.Npx);
    const float dv = lap_f(P, y + b * P.Np, i, j) - (float)lap_diag(P, i, j) * in[k];
    d[k] = dv;
    v[0] += (double)dv * dv;
  }
  block_sum<1>(v, mx, part + blockIdx.x);
}
// pass 2: dy = g A d (A is symmetric)
__global__ void __launch_bounds__(256) k_res_grad(const __grid_constant__ DevOps P, const float *__restrict__ d,
                                                  float *__restrict__ dy, float g, int B) {
  const long long n = (long long)B * P.Np;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const long long b = k / P.Np, kk = k % P.Np;
    dy[k] = g * lap_f(P, d + b * P.Np, (int)(kk % P.Npx), (int)(kk / P.Npx));
  }
}

// Weight gradient of a 32 -> 32 layer on tensor cores: D[co][t, ci] =
// sum_p dZ[p][co] A[p + t][ci], K = the 128 pixels of a 16 x 8 tile in 8 steps
// of one tile row.  The tiles are copied as they lie in memory (pixel by
// channel, cp.async, two buffers); ldmatrix.trans transposes both operands
// into fragments, and a tap is another row address.  Twelve warps: warp
// (dy, kg) takes the three taps of row dy and every fourth step, so the dZ
// fragments of a step serve three taps (96 FP32 sums per thread).  The four
// step groups' sums are added in order, one partial sum per block.
// Bound by the mma.sync rate (576 instructions per tile); the first version
// transposed by 2-byte shared-memory stores and read dZ fragments per tap:
// 124 us per layer for 4 fields of 512^2 on B200, now 104 us, and the sum of
// a quarter of the partial rows 4 instead of 8.6 us.
constexpr int kWgWarps = 12, kWgThreads = 32 * kWgWarps, kWgGroups = 4;
constexpr int kWgDz = TW * TH * PSTR, kWgA = HHT * HWD * PSTR;  // bf16 per buffer
constexpr int kWgSmem = 2 * (kWgDz + kWgA) * (int)sizeof(bf16);
static_assert(kWgSmem >= kSzWm * (int)sizeof(float), "the partial sums reuse the tiles' memory");

__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad_mid(const bf16 *__restrict__ dz, const bf16 *__restrict__ a,
                                                             float *__restrict__ part, int B, int H, int W,
                                                             int tiles_x, int tiles_y) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) uint8_t wsm[];
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(wsm);
  constexpr uint32_t kBuf = (kWgDz + kWgA) * sizeof(bf16), kAOff = kWgDz * sizeof(bf16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int dy = warp >> 2, kg = warp & 3;
  float acc[3][2][4][4] = {};
  const long long per_field = (long long)tiles_x * tiles_y;
  const long long ntiles = per_field * B;
  auto copy16 = [](uint32_t dst, const bf16 *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
  };
  auto load = [&](long long tile, int buf) {
    const int b = (int)(tile / per_field), rem = (int)(tile % per_field);
    const int x0 = (rem % tiles_x) * TW, y0 = (rem / tiles_x) * TH;
    const long long fb = (long long)b * H * W;
    const uint32_t d0 = base + buf * kBuf;
    for (int i = tid; i < TW * TH * 4; i += kWgThreads) {
      const int pix = i >> 2, prt = i & 3, gx = x0 + (pix & (TW - 1)), gy = y0 + pix / TW;
      const bool in = gx < W && gy < H;
      copy16(d0 + (pix * PSTR + prt * 8) * 2, in ? &dz[(fb + (long long)gy * W + gx) * kC + prt * 8] : dz, in);
    }
    for (int i = tid; i < HHT * HWD * 4; i += kWgThreads) {
      const int hp = i >> 2, prt = i & 3, gy = y0 - 1 + hp / HWD, gx = x0 - 1 + hp % HWD;
      const bool in = gy >= 0 && gy < H && gx >= 0 && gx < W;
      copy16(d0 + kAOff + (hp * PSTR + prt * 8) * 2, in ? &a[(fb + (long long)gy * W + gx) * kC + prt * 8] : a, in);
    }
  };
  if ((long long)blockIdx.x < ntiles) load(blockIdx.x, 0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  int buf = 0;
  // row of an 8 x 8 matrix this lane addresses (matrix lane / 8): pixels
  // (matrix bit 1 for dZ, bit 0 for A: + 8) by channels (the other bit: + 8)
  const int r8 = lane & 7, m0 = (lane >> 3) & 1, m1 = lane >> 4;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
    if (tile + gridDim.x < ntiles) load(tile + gridDim.x, buf ^ 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const uint32_t sd = base + buf * kBuf, sa = sd + kAOff;
#pragma unroll
    for (int u = 0; u < TH / kWgGroups; ++u) {
      const int ks = kg + u * kWgGroups;  // tile row
      uint32_t af[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)  // a0 (k, m), a1 (k, m + 8), a2 (k + 8, m), a3 (k + 8, m + 8)
        ldsm4t(af[mt], sd + ((ks * TW + r8 + 8 * m1) * PSTR + mt * 16 + 8 * m0) * 2);
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        uint32_t bfr[2][4];
        const int hp = (ks + dy) * HWD + dx + r8 + 8 * m0;
#pragma unroll
        for (int np = 0; np < 2; ++np)  // two n-tiles: b0 (k), b1 (k + 8) each
          ldsm4t(bfr[np], sa + (hp * PSTR + np * 16 + 8 * m1) * 2);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
            mma_bf16(acc[dx][mt][nt], af[mt][0], af[mt][1], af[mt][2], af[mt][3], bfr[nt >> 1][2 * (nt & 1)],
                     bfr[nt >> 1][2 * (nt & 1) + 1]);
      }
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  float *sum = reinterpret_cast<float *>(wsm);
  for (int q = 0; q < kWgGroups; ++q) {
    __syncthreads();
    if (kg != q) continue;
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int co = mt * 16 + g + 8 * (k >> 1), ci = nt * 8 + 2 * t4 + (k & 1);
            float *d = sum + co * kK + (dy * 3 + dx) * kC + ci;
            *d = q == 0 ? acc[dx][mt][nt][k] : *d + acc[dx][mt][nt][k];
          }
  }
  __syncthreads();
  for (int i = tid; i < kSzWm; i += kWgThreads) part[(long long)blockIdx.x * kSzWm + i] = sum[i];
}

// The same on tcgen05 (the default path).  K = 16 pixels of a row; A is four rows
// of dZ (M = 4 rows x 32 channels), B five rows of the activations (N = 160),
// shifted by tap dx: the accumulator of dZ row i and activation row q is tap
// row dy = q - i of the gradient.  The first three dZ rows use their three taps
// of the five rows, so an MMA does nine useful row pairs of twenty; what the
// others hold (the fourth dZ row is whatever follows in shared memory) is never
// read.  Both operands lie as the copies leave them, 64 bytes per pixel with
// the 64-byte swizzle, M/N-major: 8 pixels 512 bytes, the next image row a row
// pitch further, dx 64 bytes.  The three dx accumulators (480 TMEM columns) stay
// for all of a block's tiles of 64 x 6 pixels (kGStages in flight); at the end
// three warps read their dZ row's lanes and the three rows are added in order.
// What bounds it: 9 KB of operands per MMA, 72 cycles: 17 us of the tensor core
// for 4 fields of 512^2, and 20 us of memory traffic.  There on B200: the
// mma.sync form 104 us, this one 32 us.
constexpr int kGW = 64, kGRows = 6;                   // dZ tile
constexpr int kGPitch = kGW * 2 * kC;                 // 4096 per dZ row
constexpr int kGXPitch = (kGW + 2) * 2 * kC;          // 4224 per activation row
constexpr int kGOff = kGRows * kGPitch;               // the activation rows of a stage
constexpr int kGStage = kGOff + (kGRows + 2) * kGXPitch;
constexpr int kGStages = 3;
constexpr int kGN = 5 * kC;                           // 160
constexpr int kGSumLd = kK + 1;
constexpr int kGBars = 2 * kGStages + 1;
constexpr int kGSmem = kGStages * kGStage + 8 * kGBars + 16;
constexpr int kGThreads = 192;                        // four epilogue warps, the producer's and the MMAs'
constexpr uint32_t kGIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                             ((uint32_t)(kGN >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);  // both M/N-major
static_assert(kGStage % 1024 == 0 && kGOff % 1024 == 0, "the swizzle repeats every 512 bytes of address");
static_assert(kGPitch <= (kGRows + 2) * kGXPitch, "the unused fourth dZ row lies within the stage");
static_assert(3 * kC * kGSumLd * (int)sizeof(float) <= kGStages * kGStage, "the row sums reuse the stages");

__global__ void __launch_bounds__(kGThreads, 1)
    k_wgrad_tc(const __grid_constant__ CUtensorMap dz, const __grid_constant__ CUtensorMap a, float *__restrict__ part,
               int tiles_x, int tiles_y, int ntiles, unsigned *__restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem), bars = base + kGStages * kGStage;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + kGStages * kGStage + 8 * kGBars);
  const uint32_t full = bars, empty = bars + 8 * kGStages, done = bars + 16 * kGStages;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(tslot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int k = 0; k < kGBars; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bars + 8 * k) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  pdl_wait();
  pdl_trigger();
  const uint32_t taddr = *tslot;
  bool ok = true;
  if (warp == 4) {
    if (elect_one()) {
      int it = 0;
      for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int st = it % kGStages, r = tile / tiles_x, b = r / tiles_y;
        const int x = (tile % tiles_x) * kGW, y = (r % tiles_y) * kGRows;
        if (!(ok = mbar_wait(empty + 8 * st, ((it / kGStages) & 1) ^ 1))) break;
        tma_expect(full + 8 * st, kGStage);
        tma_box(base + st * kGStage, &dz, x, y, b, full + 8 * st);
        tma_box(base + st * kGStage + kGOff, &a, x - 1, y - 1, b, full + 8 * st);
      }
      // the last copies have landed before the block leaves, whatever the other roles met
      for (int k = max(0, it - kGStages); k < it; ++k) ok &= mbar_wait(full + 8 * (k % kGStages), (k / kGStages) & 1);
    }
    ok = __all_sync(0xffffffffu, ok);
  } else if (warp == 5) {
    const bool leader = elect_one();
    const uint64_t a0 = smem_desc(base, kGPitch, 512) | kSwizzle64, b0 = smem_desc(base + kGOff, kGXPitch, 512) | kSwizzle64;
    const uint32_t alo = (uint32_t)a0, ahi = (uint32_t)(a0 >> 32), blo = (uint32_t)b0, bhi = (uint32_t)(b0 >> 32);
    int it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
      const int st = it % kGStages;
      if (!(ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * st, (it / kGStages) & 1)))) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      if (!leader) continue;
      const uint32_t as = alo + st * (kGStage / 16), bs = blo + st * (kGStage / 16);
#pragma unroll
      for (int u = 0; u < kGRows / 3; ++u)
#pragma unroll
        for (int kb = 0; kb < kGW / 16; ++kb)
#pragma unroll
          for (int dx = 0; dx < 3; ++dx)
            tc_mma_lo(taddr + kGN * dx, as + (3 * u * kGPitch + 1024 * kb) / 16, ahi,
                      bs + (3 * u * kGXPitch + 1024 * kb + 64 * dx) / 16, bhi, kGIdesc,
                      it > 0 || u > 0 || kb > 0 ? 1u : 0u);
      tc_commit(empty + 8 * st);
    }
    if (leader) tc_commit(done);
  }
  if (warp != 4) {  // every MMA, before the TMEM is freed; the wait spans all tiles
    bool fin = false;
    for (int k = 0; k < 64 && !fin; ++k) fin = __all_sync(0xffffffffu, mbar_wait(done, 0));
    ok &= fin;
  }
  __syncthreads();
  float *sum = reinterpret_cast<float *>(smem);
  if (warp < 3) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    float *d = sum + (warp * kC + lane) * kGSumLd;  // dZ row i = warp, co = lane
#pragma unroll 1
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int dy = 0; dy < 3; ++dy) {
        uint32_t r[2][16];
        const uint32_t ta = taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)(kGN * dx + kC * (warp + dy));
        tmem_ld16(ta, r[0]);
        tmem_ld16(ta + 16, r[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
        for (int ci = 0; ci < kC; ++ci) d[(3 * dy + dx) * kC + ci] = __uint_as_float(r[ci >> 4][ci & 15]);
      }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  }
  if (!ok) atomicExch(err, 1u);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(taddr) : "memory");
  for (int i = tid; i < kSzWm; i += kGThreads) {
    const float *d = sum + (i / kK) * kGSumLd + i % kK;
    part[(long long)blockIdx.x * kSzWm + i] = (d[0] + d[kC * kGSumLd]) + d[2 * kC * kGSumLd];
  }
}

// out[j] = sum over rows of part[row * cols + j]: a block takes 32 columns, its
// eight warps every eighth row each, combined in a fixed order (one thread per
// column summing its rows waited for each load: 41 us for 592 rows of 9216
// columns, 8.6 us so);
// remap9 maps the edge kernel's (t*32 + c) index to W1's [c][t] layout
__global__ void __launch_bounds__(256) k_reduce_rows(const float *__restrict__ part, int rows, int cols,
                                                     float *__restrict__ out, int remap9) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sh[8][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, j = blockIdx.x * 32 + lane;
  float s = 0.0f;
  if (j < cols) {
#pragma unroll 8
    for (int r = g; r < rows; r += 8) s += __ldg(part + (long long)r * cols + j);
  }
  sh[g][lane] = s;
  __syncthreads();
  if (g == 0 && j < cols) {
#pragma unroll
    for (int q = 1; q < 8; ++q) s += sh[q][lane];
    out[remap9 ? (j & 31) * kTaps + (j >> 5) : j] = s;
  }
}

// BF16 copies of the 32 -> 32 weights: forward [co][t][ci] and the
// backward-data form [ci][8 - t][co]
__global__ void k_pack(const float *__restrict__ w, bf16 *__restrict__ wf, bf16 *__restrict__ wb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMid * kSzWm) return;
  const int l = i / kSzWm, r = i % kSzWm;
  const int co = r / kK, t = (r / kC) % kTaps, ci = r % kC;
  const bf16 v = __float2bfloat16_rn(w[kOffWm + i]);
  wf[i] = v;
  wb[l * kSzWm + ci * kK + (kTaps - 1 - t) * kC + co] = v;
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, int n, float lr, float b1, float b2, float c1, float c2, float eps) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// --- inputs from (f, p) --------------------------------------------------------
__global__ void __launch_bounds__(256) k_prep_stats(const __grid_constant__ DevOps P, const double *__restrict__ f,
                                                    const double *__restrict__ p, double *__restrict__ part) {
  double v[2] = {0.0, 0.0};
  const bool mx[2] = {false, false};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < P.Np; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k % P.Npx), j = (int)(k / P.Npx);
    const double s = f[k] / lap_diag(P, i, j);
    v[0] += s * s;
    if (p) v[1] += p[k];
  }
  block_sum<2>(v, mx, part + 2 * blockIdx.x);
}

__global__ void __launch_bounds__(256) k_prep_write(const __grid_constant__ DevOps P, const double *__restrict__ f,
                                                    const double *__restrict__ p, int center,
                                                    const double *__restrict__ stats, float *__restrict__ in,
                                                    float *__restrict__ tgt) {
  const double n = (double)P.Np;
  const double rms = sqrt(stats[0] / n);
  const double inv = rms > 0.0 ? 1.0 / rms : 1.0;
  const double mean = center ? stats[1] / n : 0.0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < P.Np; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k % P.Npx), j = (int)(k / P.Npx);
    in[k] = (float)(f[k] / lap_diag(P, i, j) * inv);
    if (tgt) tgt[k] = (float)((p[k] - mean) * inv);
  }
}

// second field of a pair = -first (the odd part of the network needs both)
__global__ void k_negate(float *__restrict__ a, long long n) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    a[n + k] = -a[k];
}

// standard normal values from a counter-based generator (splitmix64 of the
// index and the seed, Box-Muller), for the noise fields of training batches
__device__ __forceinline__ double u01(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return ((z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}
__global__ void k_gaussian(float *__restrict__ a, long long n, unsigned long long seed) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double u1 = u01(seed ^ (2ull * (unsigned long long)k)), u2 = u01(seed ^ (2ull * (unsigned long long)k + 1));
    a[k] = (float)(sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2));
  }
}
__global__ void __launch_bounds__(256) k_sumsq_f(const float *__restrict__ a, long long n, double *__restrict__ part) {
  double v[1] = {0.0};
  const bool mx[1] = {false};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    v[0] += (double)a[k] * a[k];
  block_sum<1>(v, mx, part + blockIdx.x);
}

__global__ void __launch_bounds__(256) k_dots(long long n, const double *__restrict__ x, const double *__restrict__ f,
                                              const double *__restrict__ q, double *__restrict__ part) {
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  const bool mx[4] = {false, false, false, true};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double xv = x[k], fv = f[k];
    v[0] += xv * fv;
    v[1] += xv * q[k];
    v[2] += fv * fv;
    v[3] = fmax(v[3], fabs(fv));
  }
  block_sum<4>(v, mx, part + 4 * blockIdx.x);
}

__global__ void __launch_bounds__(256) k_resid(long long n, const double *__restrict__ f, const double *__restrict__ q,
                                               double a, double *__restrict__ x, double *__restrict__ r,
                                               double *__restrict__ part) {
  double v[2] = {0.0, 0.0};
  const bool mx[2] = {false, true};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double rv = f[k] - a * q[k];
    r[k] = rv;
    x[k] *= a;
    v[0] += rv * rv;
    v[1] = fmax(v[1], fabs(rv));
  }
  block_sum<2>(v, mx, part + 2 * blockIdx.x);
}

struct EdgeGrid {
  unsigned blocks;
  int tx, ty;
};
EdgeGrid edge_grid(const ins2d_cnn *net, int B, int H, int W, int step_x) {
  EdgeGrid g;
  g.tx = (W + step_x - 1) / step_x;
  g.ty = (H + kER - 1) / kER;
  g.blocks = (unsigned)std::min({(long long)g.tx * g.ty * B, (long long)kEBlocksPerSm * net->sms, (long long)kWgBlocks});
  return g;
}

// A BF16 activation array of B fields as {channel, pixel, row, field} for copies
// of npx pixels by nrows rows, 64 bytes a pixel with the 64-byte swizzle; zeros
// outside the field
CUtensorMap act_map(const bf16 *p, int B, int H, int W, int npx, int nrows) {
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !f) throw CudaError("cnn: no cuTensorMapEncodeTiled in this driver");
    return (Encode)f;
  }();
  CUtensorMap m;
  const cuuint64_t w = (cuuint64_t)W, h = (cuuint64_t)H;
  const cuuint64_t dims[4] = {kC, w, h, (cuuint64_t)B};
  const cuuint64_t strides[3] = {2 * kC, 2 * kC * w, 2 * kC * w * h};
  const cuuint32_t box[4] = {kC, (cuuint32_t)npx, (cuuint32_t)nrows, 1}, es[4] = {1, 1, 1, 1};
  if (encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16 *>(p), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    throw CudaError("cnn: the activations' tensor map was refused");
  return m;
}

// Rows per item for `per` strips of H rows on up to cap blocks: the fewest row
// steps (R + 2 an item) of the busiest block
int item_rows(long long per, int H, int cap) {
  int R = H;
  long long best = -1;
  for (int c = 1; c <= (H + 3) / 4 && (c == 1 || per * (c - 1) < 2LL * cap); ++c) {
    const int r = (H + c - 1) / c;
    const long long cost = ((per * ((H + r - 1) / r) + cap - 1) / cap) * (r + 2);
    if (best < 0 || cost < best) best = cost, R = r;
  }
  return R;
}

// Opts a kernel in to its dynamic shared memory on the network's device at its
// first launch there: the call loads the kernel, and a network launches three
// of the seven (all of them at set-up: 3.0 instead of 1.8 ms for a process's
// first network).
template <typename K>
void opt_in(ins2d_cnn *net, unsigned bit, K k, int bytes) {
  if (net->opted & bit) return;
  CK(cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  net->opted |= bit;
}

template <int MODE>
void launch_mid(ins2d_cnn *net, const bf16 *in, const bf16 *wt, const bf16 *mask, bf16 *out, int B, int H, int W,
                cudaStream_t s) {
  if (net->path == INS2D_CNN_PATH_TCGEN05 && by_rows(W)) {
    const int strips = (W + kRM - 1) / kRM, cap = kTcBlocksPerSm * net->sms;
    const long long per = (long long)strips * B;
    const int R = item_rows(per, H, cap);
    const int chunks = (H + R - 1) / R;
    const int nitems = (int)(per * chunks), grid = std::min(nitems, cap);
    opt_in(net, 1u << MODE, k_conv_row_tc<MODE>, kRSmem);
    launch_kp(true, k_conv_row_tc<MODE>, grid, kRThreads, kRSmem, s, act_map(in, B, H, W, kRM + 2, 1), wt, mask, out, H,
              W, strips, chunks, R, nitems, net->flag);
  } else if (net->path == INS2D_CNN_PATH_TCGEN05) {
    const int tx = (W + kTcT - 1) / kTcT, ty = (H + kTcT - 1) / kTcT;
    const long long nt = (long long)tx * ty * B;
    const int grid = (int)std::min<long long>(nt, (long long)kTcBlocksPerSm * net->sms);
    opt_in(net, 4u << MODE, k_conv_mid_tc<MODE>, kTcSmem);
    launch_kp(true, k_conv_mid_tc<MODE>, grid, kTcThreads, kTcSmem, s, in, wt, mask, out, B, H, W, tx, ty, net->flag);
  } else {
    const int tiles_x = (W + TW - 1) / TW, tiles_y = (H + TH - 1) / TH;
    launch_kp(true, k_conv_mid<MODE>, dim3(tiles_x, tiles_y, B), 256, 0, s, in, wt, mask, out, H, W);
  }
}

// z = rms * y: the network output rescaled by the rms of its unscaled input
// (stats[0] = sum of squares over n_stat cells), so z = M(r) is homogeneous
// of degree one in r
// x = s (y[k] - y[n + k]) / 2: the odd part of the network over the pair
// (r, -r), rescaled by s = rms of the unscaled input (stats[0] = its sum of
// squares over n_stat cells) when stats is given, so that the result is odd
// and homogeneous of degree one in r
__global__ void k_widen_odd(const float *__restrict__ y, double *__restrict__ x, long long n,
                            const double *__restrict__ stats, double n_stat) {
  const double s = stats ? sqrt(stats[0] / n_stat) : 1.0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    x[k] = 0.5 * s * ((double)y[k] - (double)y[n + k]);
}

// flexible CG vector steps (each with its block partials)
__global__ void __launch_bounds__(256) k_fcg_pq(long long n, const double *__restrict__ p,
                                                const double *__restrict__ q, const double *__restrict__ r,
                                                double *__restrict__ part) {
  double v[2] = {0.0, 0.0};
  const bool mx[2] = {false, false};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double pv = p[k];
    v[0] += pv * q[k];
    v[1] += pv * r[k];
  }
  block_sum<2>(v, mx, part + 2 * blockIdx.x);
}
__global__ void __launch_bounds__(256) k_fcg_update(long long n, double a, double *__restrict__ x,
                                                    double *__restrict__ r, const double *__restrict__ p,
                                                    const double *__restrict__ q, double *__restrict__ part) {
  double v[2] = {0.0, 0.0};
  const bool mx[2] = {false, true};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    x[k] += a * p[k];
    const double rv = r[k] - a * q[k];
    r[k] = rv;
    v[0] += rv * rv;
    v[1] = fmax(v[1], fabs(rv));
  }
  block_sum<2>(v, mx, part + 2 * blockIdx.x);
}
__global__ void __launch_bounds__(256) k_fcg_zq(long long n, const double *__restrict__ z,
                                                const double *__restrict__ q, double *__restrict__ part) {
  double v[1] = {0.0};
  const bool mx[1] = {false};
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    v[0] += z[k] * q[k];
  block_sum<1>(v, mx, part + blockIdx.x);
}
__global__ void k_fcg_p(long long n, double b, const double *__restrict__ z, double *__restrict__ p) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    p[k] = z[k] + b * p[k];
}

unsigned stride_blocks(long long n, int per_sm = 8) {
  long long b = (n + 255) / 256;
  const long long cap = std::min<long long>(148LL * per_sm, kRedBlocks);
  if (b > cap) b = cap;
  return (unsigned)(b < 1 ? 1 : b);
}

void pack(ins2d_cnn *net, cudaStream_t s) {
  if (net->packed) return;
  k_pack<<<(kMid * kSzWm + 255) / 256, 256, 0, s>>>(net->w, net->wf, net->wb);
  CK(cudaGetLastError());
  net->packed = true;
}

}  // namespace

void check(ins2d_cnn *net, cudaStream_t s);

void reserve(ins2d_cnn *net, long long pixels) {
  if (pixels <= net->cap) return;
  for (auto *&a : net->act) cudaFree(a), a = nullptr;
  for (auto *&a : net->dz) cudaFree(a), a = nullptr;
  cudaFree(net->y);
  cudaFree(net->dy);
  cudaFree(net->dres);
  net->y = net->dy = net->dres = nullptr;
  net->cap = 0;
  const size_t nb = (size_t)pixels * kC * sizeof(bf16);
  for (auto *&a : net->act)
    if (cudaMalloc(&a, nb) != cudaSuccess) throw std::bad_alloc();
  for (auto *&a : net->dz)
    if (cudaMalloc(&a, nb) != cudaSuccess) throw std::bad_alloc();
  if (cudaMalloc(&net->y, pixels * sizeof(float)) != cudaSuccess) throw std::bad_alloc();
  if (cudaMalloc(&net->dy, pixels * sizeof(float)) != cudaSuccess) throw std::bad_alloc();
  if (cudaMalloc(&net->dres, pixels * sizeof(float)) != cudaSuccess) throw std::bad_alloc();
  net->cap = pixels;
}

// The kernels of a pass follow each other by programmatic dependent launches:
// set-up (barriers, TMEM, weights, which are packed two launches earlier at
// least) runs beside the end of the kernel before, everything else behind
// pdl_wait.  26 launches of 4 fields of 512^2, loss and gradient: 0.901 ->
// 0.811 ms.
void forward(ins2d_cnn *net, const float *in, int B, int H, int W, cudaStream_t s) {
  const long long n = (long long)B * H * W;
  reserve(net, n);
  pack(net, s);
  const EdgeGrid e = edge_grid(net, B, H, W, kEC);
  launch_kp(true, k_expand<0>, e.blocks, kEThreads, 0, s, in, net->w + kOffW1, nullptr, net->act[0], B, H, W, e.tx, e.ty);
  for (int l = 0; l < kMid; ++l)
    launch_mid<0>(net, net->act[l], net->wf + l * kSzWm, nullptr, net->act[l + 1], B, H, W, s);
  if (net->path == INS2D_CNN_PATH_TCGEN05) {
    const int strips = (W + kOW - 1) / kOW, cap = kOBlocksPerSm * net->sms;
    const long long per = (long long)strips * B;
    const int R = item_rows(per, H, cap), chunks = (H + R - 1) / R, nitems = (int)(per * chunks);
    opt_in(net, 16u, k_conv_out_tc, kOSmem);
    launch_kp(true, k_conv_out_tc, std::min(nitems, cap), kOThreads, kOSmem, s, act_map(net->act[4], B, H, W, kRM, 1),
              net->act[4], net->w + kOffW6, net->out_scale, net->y, H, W, strips, chunks, R, nitems, net->flag);
  } else {
    const EdgeGrid eo = edge_grid(net, B, H, W, kEC - 2);
    launch_kp(true, k_conv_out, eo.blocks, kEThreads, 0, s, net->act[4], net->w + kOffW6, net->out_scale, net->y, B, H,
              W, eo.tx, eo.ty);
  }
  CK(cudaGetLastError());
}

// loss (returned, after a stream synchronisation) and the gradient in net->g
double loss_grad(ins2d_cnn *net, const float *in, const float *tgt, int B, int H, int W, cudaStream_t s,
                 const DevOps *P) {
  const long long n = (long long)B * H * W;
  forward(net, in, B, H, W, s);
  const unsigned gb = stride_blocks(n, 16);
  double *part = net->red, *res = net->red + 4 * kRedBlocks;
  const float g = (float)(2.0 / (double)n) * net->out_scale;
  if (P) {
    k_res_loss<<<gb, 256, 0, s>>>(*P, net->y, in, net->dres, B, part);
    k_res_grad<<<gb, 256, 0, s>>>(*P, net->dres, net->dy, g, B);
  } else {
    launch_kp(true, k_loss, gb, 256, 0, s, net->y, tgt, net->dy, g, n, part);
  }
  launch_kp(true, k_finish<1>, 1, 256, 0, s, part, (int)gb, 0, res);
  // layer 6
  const EdgeGrid e = edge_grid(net, B, H, W, kEC);
  launch_kp(true, k_expand<1>, e.blocks, kEThreads, 0, s, net->dy, net->w + kOffW6, net->act[4], net->dz[0], B, H,
            W, e.tx, e.ty);
  launch_kp(true, k_wgrad_edge<6>, e.blocks, kEThreads, 0, s, net->act[4], net->dy, net->partials, B, H, W, e.tx, e.ty);
  launch_kp(true, k_reduce_rows, kK / 32, 256, 0, s, net->partials, (int)e.blocks, kK, net->g + kOffW6, 0);
  // layers 5..2: dZ_l in dz[cur]; weight gradient from (dZ_l, A_{l-1}); dZ_{l-1}
  const bool tc = net->path == INS2D_CNN_PATH_TCGEN05;
  const int tw = tc ? kGW : TW, th = tc ? kGRows : TH;
  const int tiles_x = (W + tw - 1) / tw, tiles_y = (H + th - 1) / th;
  const long long ntiles = (long long)tiles_x * tiles_y * B;
  const int wb = (int)std::min({(long long)kWgBlocks, (long long)net->sms, ntiles});
  int cur = 0;
  if (tc)
    opt_in(net, 32u, k_wgrad_tc, kGSmem);
  else
    opt_in(net, 64u, k_wgrad_mid, kWgSmem);
  for (int l = kMid - 1; l >= 0; --l) {
    // layer index l: input act[l], output act[l + 1], gradient dZ in dz[cur]
    if (tc)
      launch_kp(true, k_wgrad_tc, wb, kGThreads, kGSmem, s, act_map(net->dz[cur], B, H, W, kGW, kGRows),
                act_map(net->act[l], B, H, W, kGW + 2, kGRows + 2), net->partials, tiles_x, tiles_y, (int)ntiles,
                net->flag);
    else
      launch_kp(true, k_wgrad_mid, wb, kWgThreads, kWgSmem, s, net->dz[cur], net->act[l], net->partials, B, H, W,
                tiles_x, tiles_y);
    launch_kp(true, k_reduce_rows, kSzWm / 32, 256, 0, s, net->partials, wb, kSzWm, net->g + kOffWm + l * kSzWm, 0);
    launch_mid<1>(net, net->dz[cur], net->wb + l * kSzWm, net->act[l], net->dz[cur ^ 1], B, H, W, s);
    cur ^= 1;
  }
  // layer 1
  launch_kp(true, k_wgrad_edge<1>, e.blocks, kEThreads, 0, s, net->dz[cur], in, net->partials, B, H, W, e.tx, e.ty);
  launch_kp(true, k_reduce_rows, kK / 32, 256, 0, s, net->partials, (int)e.blocks, kK, net->g + kOffW1, 1);
  CK(cudaGetLastError());
  double h = 0.0;
  CK(cudaMemcpyAsync(&h, res, sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  check(net, s);
  return h / (double)n;
}

void check(ins2d_cnn *net, cudaStream_t s) {
  unsigned f = 0;
  CK(cudaMemcpyAsync(&f, net->flag, sizeof f, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (f) {
    CK(cudaMemsetAsync(net->flag, 0, sizeof(unsigned), s));
    throw CudaError("cnn: a tensor-core wait gave up (tcgen05 MMA did not complete)");
  }
}

void adam(ins2d_cnn *net, float lr, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f;
  net->adam_t += 1;
  const float c1 = 1.0f - std::pow(b1, (float)net->adam_t), c2 = 1.0f - std::pow(b2, (float)net->adam_t);
  k_adam<<<(kNParam + 255) / 256, 256, 0, s>>>(net->w, net->g, net->m, net->v, kNParam, lr, b1, b2, c1, c2, 1e-8f);
  CK(cudaGetLastError());
  net->packed = false;
}

void prepare(const DevOps &P, const double *f, const double *p, int center, float *in, float *tgt, double *red,
             cudaStream_t s) {
  const unsigned gb = stride_blocks(P.Np);
  double *part = red, *res = red + 4 * kRedBlocks;
  k_prep_stats<<<gb, 256, 0, s>>>(P, f, p, part);
  k_finish<2><<<1, 256, 0, s>>>(part, (int)gb, 0, res);
  k_prep_write<<<gb, 256, 0, s>>>(P, f, p, center, res, in, tgt);
  CK(cudaGetLastError());
}

namespace {
// the network's odd part applied to the prepared field v (f or r):
// out = scaled (N(v) - N(-v)) / 2, one forward pass over the pair
void apply_odd(ins2d_cnn *net, const DevOps &P, const double *v, double *out, bool rescale, cudaStream_t s) {
  reserve(net, 2 * P.Np);
  if (net->in1_cap < 2 * P.Np) {
    cudaFree(net->in1);
    net->in1 = nullptr;
    net->in1_cap = 0;
    if (cudaMalloc(&net->in1, 2 * P.Np * sizeof(float)) != cudaSuccess) throw std::bad_alloc();
    net->in1_cap = 2 * P.Np;
  }
  prepare(P, v, nullptr, 0, net->in1, nullptr, net->red, s);
  k_negate<<<stride_blocks(P.Np), 256, 0, s>>>(net->in1, P.Np);
  forward(net, net->in1, 2, P.Npy, P.Npx, s);
  k_widen_odd<<<stride_blocks(P.Np), 256, 0, s>>>(net->y, out, P.Np, rescale ? net->red + 4 * kRedBlocks : nullptr,
                                                   (double)P.Np);
  CK(cudaGetLastError());
}
}  // namespace

void guess(ins2d_cnn *net, const DevOps &P, const double *f, double *x0, cudaStream_t s) {
  apply_odd(net, P, f, x0, false, s);
}

void precond(ins2d_cnn *net, const DevOps &P, const double *r, double *z, cudaStream_t s) {
  apply_odd(net, P, r, z, true, s);
}

namespace {
void finish_read(int nq, unsigned gb, int max_mask, double *red, double *d, cudaStream_t s) {
  double *part = red, *res = red + 4 * kRedBlocks;
  if (nq == 1)
    k_finish<1><<<1, 256, 0, s>>>(part, (int)gb, max_mask, res);
  else
    k_finish<2><<<1, 256, 0, s>>>(part, (int)gb, max_mask, res);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(d, res, nq * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
}
}  // namespace

void fcg_pq(long long n, const double *p, const double *q, const double *r, double *red, double d[2],
            cudaStream_t s) {
  const unsigned gb = stride_blocks(n);
  k_fcg_pq<<<gb, 256, 0, s>>>(n, p, q, r, red);
  finish_read(2, gb, 0, red, d, s);
}
void fcg_update(long long n, double a, double *x, double *r, const double *p, const double *q, double *red,
                double d[2], cudaStream_t s) {
  const unsigned gb = stride_blocks(n);
  k_fcg_update<<<gb, 256, 0, s>>>(n, a, x, r, p, q, red);
  finish_read(2, gb, 2, red, d, s);
}
double fcg_zq(long long n, const double *z, const double *q, double *red, cudaStream_t s) {
  const unsigned gb = stride_blocks(n);
  k_fcg_zq<<<gb, 256, 0, s>>>(n, z, q, red);
  double d = 0.0;
  finish_read(1, gb, 0, red, &d, s);
  return d;
}
void fcg_p(long long n, double b, const double *z, double *p, cudaStream_t s) {
  k_fcg_p<<<stride_blocks(n), 256, 0, s>>>(n, b, z, p);
  CK(cudaGetLastError());
}

void negate_tail(float *a, long long n, cudaStream_t s) {
  k_negate<<<stride_blocks(n), 256, 0, s>>>(a, n);
  CK(cudaGetLastError());
}

void gaussian(float *a, long long n, uint64_t seed, cudaStream_t s) {
  k_gaussian<<<stride_blocks(n), 256, 0, s>>>(a, n, (unsigned long long)seed);
  CK(cudaGetLastError());
}

double sumsq(const float *a, long long n, double *red, cudaStream_t s) {
  const unsigned gb = stride_blocks(n);
  double *part = red, *res = red + 4 * kRedBlocks;
  k_sumsq_f<<<gb, 256, 0, s>>>(a, n, part);
  k_finish<1><<<1, 256, 0, s>>>(part, (int)gb, 0, res);
  CK(cudaGetLastError());
  double h = 0.0;
  CK(cudaMemcpyAsync(&h, res, sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return h;
}

void dots(long long n, const double *x, const double *f, const double *q, double *red, double d[4], cudaStream_t s) {
  const unsigned gb = stride_blocks(n);
  double *part = red, *res = red + 4 * kRedBlocks;
  k_dots<<<gb, 256, 0, s>>>(n, x, f, q, part);
  k_finish<4><<<1, 256, 0, s>>>(part, (int)gb, 8, res);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(d, res, 4 * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
}

void residual(long long n, const double *f, const double *q, double a, double *x, double *r, double *red,
              double d[2], cudaStream_t s) {
  const unsigned gb = stride_blocks(n);
  double *part = red, *res = red + 4 * kRedBlocks;
  k_resid<<<gb, 256, 0, s>>>(n, f, q, a, x, r, part);
  k_finish<2><<<1, 256, 0, s>>>(part, (int)gb, 2, res);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(d, res, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
}

size_t red_doubles() { return 4 * (size_t)kRedBlocks + 8; }

}  // namespace cnn
}  // namespace ins2d

// ---------------------------------------------------------------------------
// C-ABI: the network object
using namespace ins2d;
using cnn::CudaError;

namespace {

int cnn_fail(ins2d_cnn *n, int code, const std::string &msg) {
  if (n) n->err = msg;
  return code;
}

// He-normal initial weights from a seeded generator (splitmix64 + Box-Muller)
void init_weights(std::vector<float> &w, uint64_t seed) {
  uint64_t st = seed;
  auto next = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return ((z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
  };
  auto normal = [&]() {
    const double u1 = next(), u2 = next();
    return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
  };
  w.assign(cnn::kNParam, 0.0f);
  for (int i = 0; i < cnn::kOffWm; ++i) w[i] = (float)(normal() * std::sqrt(2.0 / cnn::kTaps));
  for (int i = cnn::kOffWm; i < cnn::kOffW6; ++i) w[i] = (float)(normal() * std::sqrt(2.0 / cnn::kK));
  for (int i = cnn::kOffW6; i < cnn::kNParam; ++i) w[i] = (float)(normal() * std::sqrt(1.0 / cnn::kK));
}

bool dev_ptr(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

int check_shape(ins2d_cnn *n, const void *a, const void *b, int32_t B, int32_t H, int32_t W) {
  if (B < 1 || H < 1 || W < 1) return cnn_fail(n, INS2D_EINVAL, "cnn: batch and field sizes must be positive");
  if ((long long)B * H * W > (1LL << 31) / cnn::kC)
    return cnn_fail(n, INS2D_EINVAL, "cnn: B*H*W too large (at most 2^26 pixels per call)");
  if (H > 8 * 65535 || B > 65535) return cnn_fail(n, INS2D_EINVAL, "cnn: H or B beyond the launch limits");
  if (!a || !dev_ptr(a) || (b && !dev_ptr(b)))
    return cnn_fail(n, INS2D_EINVAL, "cnn: inputs, targets and outputs must be device arrays");
  return INS2D_OK;
}

}  // namespace

extern "C" {

int ins2d_cnn_create(int32_t device, uint64_t seed, ins2d_cnn **out) {
  if (!out) return INS2D_EINVAL;
  *out = nullptr;
  ins2d_cnn *n = new (std::nothrow) ins2d_cnn();
  if (!n) return INS2D_ENOMEM;
  try {
    n->device = device;
    DeviceGuard dg(device);
    CK(dg.err);
    const size_t pb = cnn::kNParam * sizeof(float);
    for (float **p : {&n->w, &n->g, &n->m, &n->v})
      if (cudaMalloc(p, pb) != cudaSuccess) throw std::bad_alloc();
    if (cudaMalloc(&n->wf, cnn::kMid * cnn::kSzWm * sizeof(__nv_bfloat16)) != cudaSuccess) throw std::bad_alloc();
    if (cudaMalloc(&n->wb, cnn::kMid * cnn::kSzWm * sizeof(__nv_bfloat16)) != cudaSuccess) throw std::bad_alloc();
    if (cudaMalloc(&n->partials, (size_t)cnn::kWgBlocks * cnn::kSzWm * sizeof(float)) != cudaSuccess)
      throw std::bad_alloc();
    if (cudaMalloc(&n->red, cnn::red_doubles() * sizeof(double)) != cudaSuccess) throw std::bad_alloc();
    if (cudaMalloc(&n->flag, sizeof(unsigned)) != cudaSuccess) throw std::bad_alloc();
    CK(cudaMemset(n->flag, 0, sizeof(unsigned)));
    CK(cudaDeviceGetAttribute(&n->sms, cudaDevAttrMultiProcessorCount, device));
    std::vector<float> w;
    init_weights(w, seed);
    CK(cudaMemcpy(n->w, w.data(), pb, cudaMemcpyHostToDevice));
    CK(cudaMemset(n->m, 0, pb));
    CK(cudaMemset(n->v, 0, pb));
    CK(cudaMemset(n->g, 0, pb));
  } catch (const std::bad_alloc &) {
    ins2d_cnn_destroy(n);
    return INS2D_ENOMEM;
  } catch (const std::exception &) {
    ins2d_cnn_destroy(n);
    return INS2D_ECUDA;
  }
  *out = n;
  return INS2D_OK;
}

int ins2d_cnn_destroy(ins2d_cnn *n) {
  if (!n) return INS2D_OK;
  DeviceGuard dg(n->device);
  for (float *p : {n->w, n->g, n->m, n->v, n->y, n->dy, n->dres, n->in1, n->partials}) cudaFree(p);
  cudaFree(n->wf);
  cudaFree(n->wb);
  cudaFree(n->red);
  cudaFree(n->flag);
  for (auto *a : n->act) cudaFree(a);
  for (auto *a : n->dz) cudaFree(a);
  delete n;
  return INS2D_OK;
}

const char *ins2d_cnn_last_error(const ins2d_cnn *n) { return n ? n->err.c_str() : "null network"; }

int ins2d_cnn_set_stream(ins2d_cnn *n, void *stream) {
  if (!n) return INS2D_EINVAL;
  n->stream = (cudaStream_t)stream;
  return INS2D_OK;
}

int ins2d_cnn_set_path(ins2d_cnn *n, int32_t path) {
  if (!n) return INS2D_EINVAL;
  if (path != INS2D_CNN_PATH_TCGEN05 && path != INS2D_CNN_PATH_MMA_SYNC)
    return cnn_fail(n, INS2D_EINVAL, "cnn_set_path: unknown tensor-core path");
  n->path = path;
  return INS2D_OK;
}

int ins2d_cnn_get_params(ins2d_cnn *n, float *w, float *out_scale) {
  if (!n) return INS2D_EINVAL;
  try {
    DeviceGuard dg(n->device);
    CK(dg.err);
    if (w) {
      CK(cudaMemcpyAsync(w, n->w, cnn::kNParam * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
      CK(cudaStreamSynchronize(n->stream));
    }
    if (out_scale) *out_scale = n->out_scale;
  } catch (const std::exception &e) {
    return cnn_fail(n, INS2D_ECUDA, e.what());
  }
  return INS2D_OK;
}

int ins2d_cnn_set_params(ins2d_cnn *n, const float *w, float out_scale) {
  if (!n) return INS2D_EINVAL;
  if (!(out_scale > 0.0f) || !std::isfinite(out_scale)) return cnn_fail(n, INS2D_EINVAL, "cnn: out_scale must be > 0");
  try {
    DeviceGuard dg(n->device);
    CK(dg.err);
    if (w) {
      CK(cudaMemcpyAsync(n->w, w, cnn::kNParam * sizeof(float), cudaMemcpyHostToDevice, n->stream));
      CK(cudaStreamSynchronize(n->stream));
      n->packed = false;
    }
    n->out_scale = out_scale;
  } catch (const std::exception &e) {
    return cnn_fail(n, INS2D_ECUDA, e.what());
  }
  return INS2D_OK;
}

int ins2d_cnn_forward(ins2d_cnn *n, const float *in, float *y, int32_t B, int32_t H, int32_t W) {
  if (!n) return INS2D_EINVAL;
  int rc = check_shape(n, in, y, B, H, W);
  if (rc) return rc;
  if (!y) return cnn_fail(n, INS2D_EINVAL, "cnn_forward: null output");
  try {
    DeviceGuard dg(n->device);
    CK(dg.err);
    cnn::forward(n, in, B, H, W, n->stream);
    CK(cudaMemcpyAsync(y, n->y, (size_t)B * H * W * sizeof(float), cudaMemcpyDeviceToDevice, n->stream));
    CK(cudaStreamSynchronize(n->stream));
    cnn::check(n, n->stream);
  } catch (const std::bad_alloc &) {
    return cnn_fail(n, INS2D_ENOMEM, "cnn_forward: out of device memory");
  } catch (const std::exception &e) {
    return cnn_fail(n, INS2D_ECUDA, e.what());
  }
  return INS2D_OK;
}

int ins2d_cnn_get_activations(ins2d_cnn *n, int32_t layer, int64_t pixels, uint16_t *out) {
  if (!n) return INS2D_EINVAL;
  if (layer < 1 || layer > 5 || !out || pixels < 1 || pixels > n->cap)
    return cnn_fail(n, INS2D_EINVAL, "cnn_get_activations: layer 1..5, pixels of the last forward pass");
  try {
    DeviceGuard dg(n->device);
    CK(dg.err);
    CK(cudaMemcpyAsync(out, n->act[layer - 1], (size_t)pixels * cnn::kC * sizeof(uint16_t), cudaMemcpyDeviceToHost,
                       n->stream));
    CK(cudaStreamSynchronize(n->stream));
  } catch (const std::exception &e) {
    return cnn_fail(n, INS2D_ECUDA, e.what());
  }
  return INS2D_OK;
}

int ins2d_cnn_loss_grad(ins2d_cnn *n, const float *in, const float *tgt, int32_t B, int32_t H, int32_t W,
                        double *loss, float *grad) {
  if (!n) return INS2D_EINVAL;
  int rc = check_shape(n, in, tgt, B, H, W);
  if (rc) return rc;
  if (!tgt) return cnn_fail(n, INS2D_EINVAL, "cnn_loss_grad: null targets");
  try {
    DeviceGuard dg(n->device);
    CK(dg.err);
    const double l = cnn::loss_grad(n, in, tgt, B, H, W, n->stream, nullptr);
    if (loss) *loss = l;
    if (grad) {
      CK(cudaMemcpyAsync(grad, n->g, cnn::kNParam * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
      CK(cudaStreamSynchronize(n->stream));
    }
  } catch (const std::bad_alloc &) {
    return cnn_fail(n, INS2D_ENOMEM, "cnn_loss_grad: out of device memory");
  } catch (const std::exception &e) {
    return cnn_fail(n, INS2D_ECUDA, e.what());
  }
  return INS2D_OK;
}

int ins2d_cnn_train_step(ins2d_cnn *n, const float *in, const float *tgt, int32_t B, int32_t H, int32_t W, float lr,
                         double *loss) {
  if (!n) return INS2D_EINVAL;
  int rc = check_shape(n, in, tgt, B, H, W);
  if (rc) return rc;
  if (!tgt) return cnn_fail(n, INS2D_EINVAL, "cnn_train_step: null targets");
  if (!(lr > 0.0f) || !std::isfinite(lr)) return cnn_fail(n, INS2D_EINVAL, "cnn_train_step: lr must be > 0");
  try {
    DeviceGuard dg(n->device);
    CK(dg.err);
    const double l = cnn::loss_grad(n, in, tgt, B, H, W, n->stream, nullptr);
    if (!std::isfinite(l)) return cnn_fail(n, INS2D_ENONFINITE, "cnn_train_step: non-finite loss");
    cnn::adam(n, lr, n->stream);
    if (loss) *loss = l;
  } catch (const std::bad_alloc &) {
    return cnn_fail(n, INS2D_ENOMEM, "cnn_train_step: out of device memory");
  } catch (const std::exception &e) {
    return cnn_fail(n, INS2D_ECUDA, e.what());
  }
  return INS2D_OK;
}

}  // extern "C"
