// Device bodies of the fused model kernels (see model_ops.cu / model_ops.h).  Kept in a header so
// that the same source is compiled by nvcc into the sm_100a kernels and by the host compiler
// (-DBAGUA_HOST_EMULATION, host_emulation.h) into tests/cpp/model_ops_emulation.cc, which runs
// them thread for thread against the host restatement.  Shared memory is handed in by the caller.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "host_emulation.h"

namespace bagua {
namespace model_ops {
namespace bodies {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 148 * 4;

__device__ __forceinline__ void unpack8(const uint4& x, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 v = __bfloat1622float2(h[k]);
    f[2 * k] = v.x;
    f[2 * k + 1] = v.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 r;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
  return r;
}

// Two bf16 values of one sign per word, compared as 16-bit integers: activations behind a ReLU are
// not negative, and their bit patterns are ordered like their values.
#ifdef BAGUA_HOST_EMULATION
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  const uint32_t lo = (a & 0xffffu) > (b & 0xffffu) ? a : b, hi = (a >> 16) > (b >> 16) ? a : b;
  return (lo & 0xffffu) | (hi & 0xffff0000u);
}
__device__ __forceinline__ uint32_t eq_u16x2(uint32_t a, uint32_t b) {
  const uint32_t d = a ^ b;
  return ((d & 0xffffu) ? 0u : 0xffffu) | ((d >> 16) ? 0u : 0xffff0000u);
}
#else
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) { return __vmaxu2(a, b); }
__device__ __forceinline__ uint32_t eq_u16x2(uint32_t a, uint32_t b) { return __vcmpeq2(a, b); }
#endif

// max(x + b, 0) of two bf16 values, rounded once: the bits of an addition in fp32 that is rounded to bf16 afterwards (where
// that one is inexact, the smaller operand is too small for a tie).  Comparisons are masks of 0xffff.
#ifdef BAGUA_HOST_EMULATION
__device__ __forceinline__ float bf16_value(uint32_t half) {
  const uint32_t u = half << 16;
  float f;
  memcpy(&f, &u, 4);
  return f;
}
__device__ __forceinline__ uint32_t bias_relu_x2(uint32_t x, uint32_t b) {
  uint32_t r = 0;
  for (int k = 0; k < 32; k += 16) {
    const __nv_bfloat16 v = __float2bfloat16_rn(fmaxf(bf16_value(x >> k & 0xffffu) + bf16_value(b >> k & 0xffffu), 0.f));
    uint16_t u;
    memcpy(&u, &v, 2);
    r |= (uint32_t)u << k;
  }
  return r & 0x7fff7fffu;
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) { return max_u16x2(a, b); }
__device__ __forceinline__ uint32_t eq_bf16x2(uint32_t a, uint32_t b) { return eq_u16x2(a, b); }
#else
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t v) { return *reinterpret_cast<const __nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t bits_of(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ uint32_t bias_relu_x2(uint32_t x, uint32_t b) {
  return bits_of(__hmax2(__hadd2(as_bf162(x), as_bf162(b)), as_bf162(0u))) & 0x7fff7fffu;
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) { return bits_of(__hmax2(as_bf162(a), as_bf162(b))); }
__device__ __forceinline__ uint32_t eq_bf16x2(uint32_t a, uint32_t b) { return __heq2_mask(as_bf162(a), as_bf162(b)); }
#endif

__device__ __forceinline__ uint4 clear_signs(const uint4& a) {
  return make_uint4(a.x & 0x7fff7fffu, a.y & 0x7fff7fffu, a.z & 0x7fff7fffu, a.w & 0x7fff7fffu);
}

// What a backward pass wants of eight 16-bit values is one bit each: bit 2 k + half of the result is set where half `half` of
// mask k is (masks of 0xffff or 0 per half) ...
__device__ __forceinline__ uint32_t gather_bits(uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  const uint32_t a = (m0 & 0x00010001u) | (m1 & 0x00040004u) | (m2 & 0x00100010u) | (m3 & 0x00400040u);
  return (a | (a >> 15)) & 0xffu;
}
// ... and mask k again.
__device__ __forceinline__ uint32_t spread_bits(uint32_t bits, int k) {
  const uint32_t b = bits >> (2 * k);
  return ((0u - (b & 1u)) & 0x0000ffffu) | ((0u - ((b >> 1) & 1u)) & 0xffff0000u);
}

// Of eight values those whose bit is set.
__device__ __forceinline__ uint4 keep_bits(const uint4& v, uint32_t bits) {
  return make_uint4(v.x & spread_bits(bits, 0), v.y & spread_bits(bits, 1), v.z & spread_bits(bits, 2), v.w & spread_bits(bits, 3));
}

// ---- forward ----------------------------------------------------------------------
__device__ __forceinline__ uint4 bias_relu_vec(const uint4& x, const float* b) {
  float f[8];
  unpack8(x, f);
#pragma unroll
  for (int k = 0; k < 8; ++k) f[k] = fmaxf(f[k] + b[k], 0.f);
  return pack8(f);
}

// The 8 bias values of channel group cg.
__device__ __forceinline__ void load_bias8(const __nv_bfloat16* __restrict__ bias, int cg, float (&b)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) b[k] = __bfloat162float(bias[cg * 8 + k]);
}

// cgroups = C / 8 vectors per row.  cgroups divides kThreads, hence the grid stride too, so all
// vectors a thread visits belong to one channel group: its bias stays in registers and the loop
// has no division.  kSigns: which values are positive is left in `signs`, a byte per vector.
template <bool kSigns = false>
__device__ __forceinline__ void bias_relu_body(uint4* __restrict__ z, const __nv_bfloat16* __restrict__ bias,
                                               int64_t nvec, int cgroups, uint8_t* __restrict__ signs = nullptr) {
  float bs[8];
  load_bias8(bias, (int)(threadIdx.x % cgroups), bs);
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  auto one = [&](int64_t at, const uint4& in) {
    const uint4 r = bias_relu_vec(in, bs);
    z[at] = r;
    if constexpr (kSigns) {
      const uint4 y = clear_signs(r);  // -0 is not positive
      signs[at] = (uint8_t)gather_bits(~eq_u16x2(y.x, 0u), ~eq_u16x2(y.y, 0u), ~eq_u16x2(y.z, 0u), ~eq_u16x2(y.w, 0u));
    }
  };
  for (; v + 3 * stride < nvec; v += 4 * stride) {
    const uint4 a = z[v], b = z[v + stride], c = z[v + 2 * stride], d = z[v + 3 * stride];
    one(v, a);
    one(v + stride, b);
    one(v + 2 * stride, c);
    one(v + 3 * stride, d);
  }
  for (; v < nvec; v += stride) one(v, z[v]);
}

// ---- backward ---------------------------------------------------------------------
__device__ __forceinline__ uint4 relu_mask_acc(const uint4& dy, const uint4& y, float (&acc)[8]) {
  float g[8], o[8];
  unpack8(dy, g);
  unpack8(y, o);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    g[k] = o[k] > 0.f ? g[k] : 0.f;
    acc[k] += g[k];
  }
  return pack8(g);
}

// Threads are laid out [rows_per_iter][cgroups]: thread (ro, cg) visits rows ro, ro + R, ...
// (R = gridDim.x * rows_per_iter apart) and always the same 8 channels.  cgroups divides kThreads.
// kSigns: `signs` as the forward left them stand in for y, a sixteenth of its bytes.
template <bool kSigns = false>
__device__ __forceinline__ void bias_relu_backward_body(const uint4* dy, const uint4* __restrict__ y, uint4* dz,
                                                        float* __restrict__ partial, int64_t rows, int cgroups,
                                                        float* s_acc, const uint8_t* __restrict__ signs = nullptr) {
  const int rows_per_iter = kThreads / cgroups;
  const int cg = threadIdx.x % cgroups, ro = threadIdx.x / cgroups;
  const int64_t step = (int64_t)gridDim.x * rows_per_iter;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  int64_t row = (int64_t)blockIdx.x * rows_per_iter + ro;
  if constexpr (kSigns) {
    auto one = [&](const uint4& g, uint32_t bits) {
      const uint4 r = keep_bits(g, bits);
      float f[8];
      unpack8(r, f);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += f[k];
      return r;
    };
    for (; row + 3 * step < rows; row += 4 * step) {
      const int64_t v0 = row * cgroups + cg, dv = step * cgroups;
      const uint4 a0 = dy[v0], a1 = dy[v0 + dv], a2 = dy[v0 + 2 * dv], a3 = dy[v0 + 3 * dv];
      const uint32_t b0 = signs[v0], b1 = signs[v0 + dv], b2 = signs[v0 + 2 * dv], b3 = signs[v0 + 3 * dv];
      dz[v0] = one(a0, b0);
      dz[v0 + dv] = one(a1, b1);
      dz[v0 + 2 * dv] = one(a2, b2);
      dz[v0 + 3 * dv] = one(a3, b3);
    }
    for (; row < rows; row += step) {
      const int64_t v0 = row * cgroups + cg;
      dz[v0] = one(dy[v0], signs[v0]);
    }
  } else {
    for (; row + step < rows; row += 2 * step) {
      const int64_t v0 = row * cgroups + cg, v1 = (row + step) * cgroups + cg;
      const uint4 a0 = dy[v0], b0 = y[v0], a1 = dy[v1], b1 = y[v1];
      dz[v0] = relu_mask_acc(a0, b0, acc);
      dz[v1] = relu_mask_acc(a1, b1, acc);
    }
    for (; row < rows; row += step) {
      const int64_t v0 = row * cgroups + cg;
      dz[v0] = relu_mask_acc(dy[v0], y[v0], acc);
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s_acc[threadIdx.x * 8 + k] = acc[k];
  __syncthreads();
  const int C = cgroups * 8;
  for (int c = threadIdx.x; c < C; c += kThreads) {
    const int g = c >> 3, k = c & 7;
    float s = 0.f;
    for (int r = 0; r < rows_per_iter; ++r) s += s_acc[(r * cgroups + g) * 8 + k];
    partial[(size_t)blockIdx.x * C + c] = s;
  }
}

// Column sums of the blocks' partial rows.  A thread owns column blockIdx.x * blockDim.x + threadIdx.x and
// every blockDim.y-th row; the blockDim.y sums of a column are then added in order through s_acc
// (blockDim.x * blockDim.y floats; unused when blockDim.y is 1).
//
// Latency-bound: the partial rows sit in L2 (592 x 64 floats = 150 KB for the widest activation of VGG-16), so
// what counts is the length of a thread's chain of loads.  One thread per column walked all 592 rows in 17.7 us;
// 32 x 32 threads per block walk 19 rows each.
__device__ __forceinline__ void bias_grad_finish_body(const float* __restrict__ partial, float* __restrict__ db,
                                                      int blocks, int C, float* s_acc = nullptr,
                                                      bool accumulate = false) {
  const int c = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int rows_at_once = blockDim.y > 1 ? (int)blockDim.y : 1;
  float s = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int b = (int)threadIdx.y; b < blocks; b += rows_at_once) s += partial[(size_t)b * C + c];
  }
  if (rows_at_once > 1) {
    s_acc[threadIdx.y * blockDim.x + threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0) return;
    s = 0.f;
    for (int r = 0; r < rows_at_once; ++r) s += s_acc[r * blockDim.x + threadIdx.x];
  }
  if (c < C) db[c] = accumulate ? db[c] + s : s;
}

// Column sums of x [rows, 8 * cgroups] in bf16, for any number of channel groups: warp (threadIdx.x / 32) of a
// block takes every (blockDim.x / 32)-th row of its slice and 32 channel groups (512 contiguous bytes); the
// warps' sums meet in s_acc (8 floats per thread) and the block leaves one partial row (or adds to it).
__device__ __forceinline__ void column_sum_body(const uint4* __restrict__ x, float* __restrict__ partial, int64_t rows,
                                                int cgroups, float* s_acc, bool accumulate) {
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, warps = (int)blockDim.x >> 5;
  const int cg = (int)blockIdx.x * 32 + lane;
  const int64_t per = (rows + gridDim.y - 1) / gridDim.y;
  const int64_t lo = (int64_t)blockIdx.y * per, hi = lo + per < rows ? lo + per : rows;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  if (cg < cgroups) {
#pragma unroll 4
    for (int64_t r = lo + warp; r < hi; r += warps) {
      float f[8];
      unpack8(x[r * cgroups + cg], f);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += f[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s_acc[threadIdx.x * 8 + k] = acc[k];
  __syncthreads();
  // thread t adds the warps' sums of column t of the block's 256
  const int c = (int)blockIdx.x * 256 + (int)threadIdx.x;
  if ((int)threadIdx.x < 256 && c < cgroups * 8) {
    float s = 0.f;
    for (int w = 0; w < warps; ++w) s += s_acc[w * 256 + threadIdx.x];
    float* out = partial + (size_t)blockIdx.y * cgroups * 8 + c;
    *out = accumulate ? *out + s : s;
  }
}

// ---- 2x2 / stride-2 max pooling -------------------------------------------------------
// Vector indices are [n][h][w][cg] with cg fastest, so a warp reads whole pixels of contiguous
// channels.  Index arithmetic divides in 32 bits whenever the value fits: the 64-bit division
// costs several times as many instructions, enough to show next to the handful of 16-byte
// accesses a thread makes per output vector.
__device__ __forceinline__ void div_mod(int64_t a, int64_t d, int64_t& quot, int64_t& rem) {
  if (a <= 0xffffffffLL && d <= 0xffffffffLL) {
    const uint32_t a32 = (uint32_t)a, d32 = (uint32_t)d, q32 = a32 / d32;
    quot = q32;
    rem = a32 - q32 * d32;
  } else {
    quot = a / d;
    rem = a - quot * d;
  }
}

struct PoolIndex {
  int64_t x00;  // vector index of the window's top-left input pixel
  int64_t dw, dh;  // vector strides to the right / lower neighbour
};
// Pooled pixel p = (n * Ho + ho) * Wo + wo of an [N, 2 Ho, W, C] input: its window starts at
// input row 2 (n * Ho + ho), column 2 wo, so one division by Wo is all it takes.
__device__ __forceinline__ PoolIndex pool_index(int64_t p, int64_t cg, int64_t Wo, int64_t W, int cgroups) {
  int64_t q, wo;
  div_mod(p, Wo, q, wo);
  PoolIndex r;
  r.dw = cgroups;
  r.dh = W * cgroups;
  r.x00 = (2 * q * W + 2 * wo) * cgroups + cg;
  return r;
}

// One thread per output vector (8 channels of one output pixel); any number of channel groups.
__device__ __forceinline__ void maxpool2x2_forward_body(const uint4* __restrict__ x, uint4* __restrict__ y,
                                                        int64_t nvec_out, int64_t Wo, int64_t W, int cgroups) {
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < nvec_out; v += stride) {
    int64_t pixel, cg;
    div_mod(v, cgroups, pixel, cg);
    const PoolIndex p = pool_index(pixel, cg, Wo, W, cgroups);
    const uint4 a = x[p.x00], b = x[p.x00 + p.dw], c = x[p.x00 + p.dh], d = x[p.x00 + p.dh + p.dw];
    float fa[8], fb[8], fc[8], fd[8];
    unpack8(a, fa);
    unpack8(b, fb);
    unpack8(c, fc);
    unpack8(d, fd);
#pragma unroll
    for (int k = 0; k < 8; ++k) fa[k] = fmaxf(fmaxf(fa[k], fb[k]), fmaxf(fc[k], fd[k]));
    y[v] = pack8(fa);
  }
}

__device__ __forceinline__ void maxpool2x2_backward_body(const uint4* __restrict__ x, const uint4* __restrict__ dy,
                                                         uint4* __restrict__ dx, int64_t nvec_out, int64_t Wo,
                                                         int64_t W, int cgroups) {
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < nvec_out; v += stride) {
    int64_t pixel, cg;
    div_mod(v, cgroups, pixel, cg);
    const PoolIndex p = pool_index(pixel, cg, Wo, W, cgroups);
    const uint4 a = x[p.x00], b = x[p.x00 + p.dw], c = x[p.x00 + p.dh], d = x[p.x00 + p.dh + p.dw];
    const uint4 g4 = dy[v];
    float fa[8], fb[8], fc[8], fd[8], g[8];
    unpack8(a, fa);
    unpack8(b, fb);
    unpack8(c, fc);
    unpack8(d, fd);
    unpack8(g4, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      // first maximum in scan order (0,0) (0,1) (1,0) (1,1): a later element wins only if strictly larger
      float m = fa[k];
      int idx = 0;
      if (fb[k] > m) {
        m = fb[k];
        idx = 1;
      }
      if (fc[k] > m) {
        m = fc[k];
        idx = 2;
      }
      if (fd[k] > m) idx = 3;
      fa[k] = idx == 0 ? g[k] : 0.f;
      fb[k] = idx == 1 ? g[k] : 0.f;
      fc[k] = idx == 2 ? g[k] : 0.f;
      fd[k] = idx == 3 ? g[k] : 0.f;
    }
    dx[p.x00] = pack8(fa);
    dx[p.x00 + p.dw] = pack8(fb);
    dx[p.x00 + p.dh] = pack8(fc);
    dx[p.x00 + p.dh + p.dw] = pack8(fd);
  }
}

// ---- bias + ReLU with the 2x2 pooling that follows it -----------------------------------
// Forward: y = max(z + bias, 0) in place on the [N, H, W, C] convolution output, and
// p = 2x2 max of y, both from one read of z.  One thread per pooled vector; cgroups divides
// kThreads, so a thread keeps its channel group (and its bias, in registers) and walks pooled
// pixels that are a fixed number apart.
__device__ __forceinline__ void bias_relu_pool_body(uint4* __restrict__ y, uint4* __restrict__ p,
                                                    const __nv_bfloat16* __restrict__ bias, int64_t pooled_pixels,
                                                    int64_t Wo, int64_t W, int cgroups) {
  const int cg = (int)(threadIdx.x % cgroups);
  float b[8];
  load_bias8(bias, cg, b);
  const int64_t pixel_step = (int64_t)gridDim.x * (kThreads / cgroups);
  for (int64_t px = (int64_t)blockIdx.x * (kThreads / cgroups) + threadIdx.x / cgroups; px < pooled_pixels;
       px += pixel_step) {
    const PoolIndex q = pool_index(px, cg, Wo, W, cgroups);
    const uint4 a0 = y[q.x00], a1 = y[q.x00 + q.dw], a2 = y[q.x00 + q.dh], a3 = y[q.x00 + q.dh + q.dw];
    const uint4 r0 = bias_relu_vec(a0, b), r1 = bias_relu_vec(a1, b), r2 = bias_relu_vec(a2, b), r3 = bias_relu_vec(a3, b);
    y[q.x00] = r0;
    y[q.x00 + q.dw] = r1;
    y[q.x00 + q.dh] = r2;
    y[q.x00 + q.dh + q.dw] = r3;
    float f0[8], f1[8], f2[8], f3[8];
    unpack8(r0, f0);
    unpack8(r1, f1);
    unpack8(r2, f2);
    unpack8(r3, f3);
#pragma unroll
    for (int k = 0; k < 8; ++k) f0[k] = fmaxf(fmaxf(f0[k], f1[k]), fmaxf(f2[k], f3[k]));
    p[px * cgroups + cg] = pack8(f0);
  }
}

// The maximum of four positions, none of them negative; in their places, masks that are set at the first one that holds it, if
// it is not zero.
__device__ __forceinline__ uint32_t first_max(uint32_t& y0, uint32_t& y1, uint32_t& y2, uint32_t& y3) {
  const uint32_t m = max_bf16x2(max_bf16x2(y0, y1), max_bf16x2(y2, y3)), none = eq_bf16x2(m, 0u);
  const uint32_t e0 = eq_bf16x2(y0, m), e01 = e0 | eq_bf16x2(y1, m), e012 = e01 | eq_bf16x2(y2, m);
  y0 = e0 & ~none;
  y1 = e01 & ~e0 & ~none;
  y2 = e012 & ~e01 & ~none;
  y3 = ~e012 & ~none;
  return m;
}

// The same maximum without the activation: z is only read, and only the pooled output is written.  kCodes: with what the
// backward needs of the activation, in four bytes per pooled vector: byte `position` has a bit for every channel whose first
// maximum, if it is positive, is at that position of the window.  (64 channels at 224 x 224, batch 32, us: forward / backward
// 43.5 / 76.6 where the backward makes the activation again from z and the bias, 48.0 / 43.9 with codes.)
template <bool kCodes = false>
__device__ __forceinline__ void bias_relu_pool_only_body(const uint4* __restrict__ z, uint4* __restrict__ p,
                                                         const __nv_bfloat16* __restrict__ bias, int64_t pooled_pixels,
                                                         int64_t Wo, int64_t W, int cgroups, uint32_t* __restrict__ codes = nullptr) {
  const int cg = (int)(threadIdx.x % cgroups);
  float b[8];
  load_bias8(bias, cg, b);
  const uint4 b2 = pack8(b);
  const int64_t pixel_step = (int64_t)gridDim.x * (kThreads / cgroups);
  for (int64_t px = (int64_t)blockIdx.x * (kThreads / cgroups) + threadIdx.x / cgroups; px < pooled_pixels;
       px += pixel_step) {
    const PoolIndex q = pool_index(px, cg, Wo, W, cgroups);
    uint4 a0 = z[q.x00], a1 = z[q.x00 + q.dw], a2 = z[q.x00 + q.dh], a3 = z[q.x00 + q.dh + q.dw];
    if constexpr (kCodes) {
      // two channels an instruction: one at a time, as below, the instructions took 57 us where memory takes 43
      auto active = [&](const uint4& v) {
        return make_uint4(bias_relu_x2(v.x, b2.x), bias_relu_x2(v.y, b2.y), bias_relu_x2(v.z, b2.z), bias_relu_x2(v.w, b2.w));
      };
      a0 = active(a0);
      a1 = active(a1);
      a2 = active(a2);
      a3 = active(a3);
      uint4 m;
      m.x = first_max(a0.x, a1.x, a2.x, a3.x);
      m.y = first_max(a0.y, a1.y, a2.y, a3.y);
      m.z = first_max(a0.z, a1.z, a2.z, a3.z);
      m.w = first_max(a0.w, a1.w, a2.w, a3.w);
      p[px * cgroups + cg] = m;
      codes[px * cgroups + cg] = gather_bits(a0.x, a0.y, a0.z, a0.w) | gather_bits(a1.x, a1.y, a1.z, a1.w) << 8 |
                                 gather_bits(a2.x, a2.y, a2.z, a2.w) << 16 | gather_bits(a3.x, a3.y, a3.z, a3.w) << 24;
      continue;
    }
    float f0[8], f1[8], f2[8], f3[8];
    unpack8(a0, f0);
    unpack8(a1, f1);
    unpack8(a2, f2);
    unpack8(a3, f3);
    // adding the bias, clamping and rounding are monotonic: the maximum may be taken first
#pragma unroll
    for (int k = 0; k < 8; ++k) f0[k] = fmaxf(fmaxf(fmaxf(f0[k], f1[k]), fmaxf(f2[k], f3[k])) + b[k], 0.f);
    p[px * cgroups + cg] = pack8(f0);
  }
}

// g for the first of four positions that holds the maximum, zero for the others; nothing where the maximum is zero.
__device__ __forceinline__ uint32_t route_to_first_max(uint32_t& y0, uint32_t& y1, uint32_t& y2, uint32_t& y3, uint32_t g) {
  first_max(y0, y1, y2, y3);
  const uint32_t any = y0 | y1 | y2 | y3;
  y0 &= g;
  y1 &= g;
  y2 &= g;
  y3 &= g;
  return g & any;
}

// Backward of the pair: dz = dp routed to each window's first maximum of y, masked by y > 0,
// zero elsewhere; db[c] = column sums of dz.  Thread (ro, cg) visits pooled pixels ro, ro + R, ...
// and always the same 8 channels, like the un-pooled backward.  kFromZ: `y` holds the convolution's
// output z, and the activation max(z + bias, 0), rounded as the forward rounds it, is made again here.
// (Blocks train through bias_relu_pool_backward_codes_body; these two forms are what it is compared with.)
template <bool kFromZ = false>
__device__ __forceinline__ void bias_relu_pool_backward_body(const uint4* __restrict__ dp, const uint4* __restrict__ y,
                                                             uint4* __restrict__ dz, float* __restrict__ partial,
                                                             int64_t pooled_rows, int64_t Wo, int64_t W, int cgroups,
                                                             float* s_acc,
                                                             const __nv_bfloat16* __restrict__ bias = nullptr) {
  const int rows_per_iter = kThreads / cgroups;
  const int cg = threadIdx.x % cgroups, ro = threadIdx.x / cgroups;
  const int64_t step = (int64_t)gridDim.x * rows_per_iter;
  float acc[8], bs[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  if constexpr (kFromZ) load_bias8(bias, cg, bs);
  for (int64_t pr = (int64_t)blockIdx.x * rows_per_iter + ro; pr < pooled_rows; pr += step) {
    const int64_t v = pr * cgroups + cg;
    const PoolIndex q = pool_index(pr, cg, Wo, W, cgroups);
    uint4 a0 = y[q.x00], a1 = y[q.x00 + q.dw], a2 = y[q.x00 + q.dh], a3 = y[q.x00 + q.dh + q.dw];
    const uint4 g4 = dp[v];
    if constexpr (kFromZ) {
      // two channels per word throughout: half the instructions of the per-channel form below, so that making
      // the activation again costs nothing (512 channels at 28 x 28, batch 32: 16.6 us; 18.8 us from the stored
      // activation per channel)
      a0 = clear_signs(bias_relu_vec(a0, bs));  // -0 would be the largest of all
      a1 = clear_signs(bias_relu_vec(a1, bs));
      a2 = clear_signs(bias_relu_vec(a2, bs));
      a3 = clear_signs(bias_relu_vec(a3, bs));
      uint4 gr;
      gr.x = route_to_first_max(a0.x, a1.x, a2.x, a3.x, g4.x);
      gr.y = route_to_first_max(a0.y, a1.y, a2.y, a3.y, g4.y);
      gr.z = route_to_first_max(a0.z, a1.z, a2.z, a3.z, g4.z);
      gr.w = route_to_first_max(a0.w, a1.w, a2.w, a3.w, g4.w);
      dz[q.x00] = a0;
      dz[q.x00 + q.dw] = a1;
      dz[q.x00 + q.dh] = a2;
      dz[q.x00 + q.dh + q.dw] = a3;
      float g[8];
      unpack8(gr, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += g[k];
      continue;
    }
    float f0[8], f1[8], f2[8], f3[8], g[8];
    unpack8(a0, f0);
    unpack8(a1, f1);
    unpack8(a2, f2);
    unpack8(a3, f3);
    unpack8(g4, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float m = f0[k];
      int idx = 0;
      if (f1[k] > m) {
        m = f1[k];
        idx = 1;
      }
      if (f2[k] > m) {
        m = f2[k];
        idx = 2;
      }
      if (f3[k] > m) {
        m = f3[k];
        idx = 3;
      }
      const float gv = m > 0.f ? g[k] : 0.f;  // the ReLU mask of the element the gradient goes to
      acc[k] += gv;
      f0[k] = idx == 0 ? gv : 0.f;
      f1[k] = idx == 1 ? gv : 0.f;
      f2[k] = idx == 2 ? gv : 0.f;
      f3[k] = idx == 3 ? gv : 0.f;
    }
    dz[q.x00] = pack8(f0);
    dz[q.x00 + q.dw] = pack8(f1);
    dz[q.x00 + q.dh] = pack8(f2);
    dz[q.x00 + q.dh + q.dw] = pack8(f3);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s_acc[threadIdx.x * 8 + k] = acc[k];
  __syncthreads();
  const int C = cgroups * 8;
  for (int c = threadIdx.x; c < C; c += kThreads) {
    const int g = c >> 3, k = c & 7;
    float s = 0.f;
    for (int r = 0; r < rows_per_iter; ++r) s += s_acc[(r * cgroups + g) * 8 + k];
    partial[(size_t)blockIdx.x * C + c] = s;
  }
}

// The same from the forward's codes: neither z nor the activation is read.
__device__ __forceinline__ void bias_relu_pool_backward_codes_body(const uint4* __restrict__ dp, const uint32_t* __restrict__ codes,
                                                                   uint4* __restrict__ dz, float* __restrict__ partial, int64_t pooled_rows,
                                                                   int64_t Wo, int64_t W, int cgroups, float* s_acc) {
  const int rows_per_iter = kThreads / cgroups;
  const int cg = threadIdx.x % cgroups, ro = threadIdx.x / cgroups;
  const int64_t step = (int64_t)gridDim.x * rows_per_iter;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
#pragma unroll 2
  for (int64_t pr = (int64_t)blockIdx.x * rows_per_iter + ro; pr < pooled_rows; pr += step) {
    const int64_t v = pr * cgroups + cg;
    const uint4 g = dp[v];
    const uint32_t code = codes[v];
    const PoolIndex q = pool_index(pr, cg, Wo, W, cgroups);
    uint4 sum = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int at = 0; at < 4; ++at) {
      const uint4 r = keep_bits(g, code >> (8 * at));
      dz[q.x00 + (at & 1 ? q.dw : 0) + (at & 2 ? q.dh : 0)] = r;
      sum = make_uint4(sum.x | r.x, sum.y | r.y, sum.z | r.z, sum.w | r.w);  // a channel goes to one position at most
    }
    float f[8];
    unpack8(sum, f);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] += f[k];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s_acc[threadIdx.x * 8 + k] = acc[k];
  __syncthreads();
  const int C = cgroups * 8;
  for (int c = threadIdx.x; c < C; c += kThreads) {
    const int g = c >> 3, k = c & 7;
    float s = 0.f;
    for (int r = 0; r < rows_per_iter; ++r) s += s_acc[(r * cgroups + g) * 8 + k];
    partial[(size_t)blockIdx.x * C + c] = s;
  }
}

}  // namespace bodies
}  // namespace model_ops
}  // namespace bagua
