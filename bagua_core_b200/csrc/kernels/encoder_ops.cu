// See encoder_ops.h.  All kernels are latency- and bandwidth-bound streams over activations of a few MB that
// mostly sit in L2: 16-byte vectors, one warp per row for everything that needs row statistics (shuffles
// instead of block barriers), column sums kept in registers over the rows a warp visits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../common.h"
#include "encoder_ops.h"
#include "launch.cuh"
#include "model_ops_bodies.cuh"

namespace bagua {
namespace encoder_ops {

namespace {

using kernels::launch_overlapped;
using kernels::sm_count;
using kernels::wait_for_predecessor;
using model_ops::bodies::pack8;
using model_ops::bodies::unpack8;

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxVecs = 4;  // H <= 32 lanes * 8 columns * kMaxVecs

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 8 floats from an address that is 4-byte aligned; `vec`: 16-byte aligned.
__device__ __forceinline__ void load8(const float* p, bool vec, float (&f)[8]) {
  if (vec) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w;
    f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = p[k];
  }
}

template <int NV>
struct Row {
  float v[NV][8];
};
// Mean and reciprocal deviation of a row spread over a warp.
template <int NV>
__device__ __forceinline__ void statistics(const Row<NV>& x, int nvec, int lane, float eps, int H, float& mean, float& rstd) {
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j)
    if (j * 32 + lane < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) s += x.v[j][k];
    }
  mean = warp_sum(s) / (float)H;
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j)
    if (j * 32 + lane < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = x.v[j][k] - mean;
        q += d * d;
      }
    }
  rstd = rsqrtf(warp_sum(q) / (float)H + eps);
}

template <int NV>
__global__ void __launch_bounds__(kThreads)
    add_layer_norm_kernel(const uint4* __restrict__ x, const uint4* __restrict__ r, const float* __restrict__ gamma,
                          const float* __restrict__ beta, float eps, uint4* __restrict__ sum, uint4* __restrict__ y,
                          float* __restrict__ mean, float* __restrict__ rstd, int64_t rows, int H, bool vec) {
  wait_for_predecessor();
  const int lane = (int)threadIdx.x & 31, nvec = H / 8;
  const int64_t row = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  Row<NV> a;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = j * 32 + lane;
    if (v >= nvec) continue;
    unpack8(x[row * nvec + v], a.v[j]);
    if (r) {
      float b[8];
      unpack8(r[row * nvec + v], b);
#pragma unroll
      for (int k = 0; k < 8; ++k) a.v[j][k] += b[k];
      const uint4 packed = pack8(a.v[j]);  // the sum as a bf16 residual stream holds it
      sum[row * nvec + v] = packed;
      unpack8(packed, a.v[j]);
    }
  }
  float m, rs;
  statistics<NV>(a, nvec, lane, eps, H, m, rs);
  if (lane == 0) {
    mean[row] = m;
    rstd[row] = rs;
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = j * 32 + lane;
    if (v >= nvec) continue;
    float g[8], b[8];
    load8(gamma + v * 8, vec, g);
    load8(beta + v * 8, vec, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) a.v[j][k] = (a.v[j][k] - m) * rs * g[k] + b[k];
    y[row * nvec + v] = pack8(a.v[j]);
  }
}

// tok[id] + pos[p] + typ, in this order, in fp32
template <int NV>
__device__ __forceinline__ void gather_row(const int64_t* ids, int64_t vocab, const float* tok, const float* pos,
                                           const float* typ, int64_t row, int64_t seq, int H, int nvec, int lane, bool vec,
                                           Row<NV>& a) {
  const int64_t id = ids[row];
  const bool known = id >= 0 && id < vocab;  // an id outside the table gives a row of NaN
  const float* t = tok + (known ? id : 0) * H;
  const float* p = pos + (row % seq) * H;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = j * 32 + lane;
    if (v >= nvec) continue;
    float b[8], c[8];
    load8(t + v * 8, vec, a.v[j]);
    load8(p + v * 8, vec, b);
    load8(typ + v * 8, vec, c);
#pragma unroll
    for (int k = 0; k < 8; ++k) a.v[j][k] = known ? a.v[j][k] + b[k] + c[k] : nanf("");
  }
}

template <int NV>
__global__ void __launch_bounds__(kThreads)
    embed_layer_norm_kernel(const int64_t* __restrict__ ids, int64_t vocab, const float* __restrict__ tok,
                            const float* __restrict__ pos,
                            const float* __restrict__ typ, const float* __restrict__ gamma, const float* __restrict__ beta,
                            float eps, uint4* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd, int64_t rows,
                            int64_t seq, int H, bool vec) {
  wait_for_predecessor();
  const int lane = (int)threadIdx.x & 31, nvec = H / 8;
  const int64_t row = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  Row<NV> a;
  gather_row<NV>(ids, vocab, tok, pos, typ, row, seq, H, nvec, lane, vec, a);
  float m, rs;
  statistics<NV>(a, nvec, lane, eps, H, m, rs);
  if (lane == 0) {
    mean[row] = m;
    rstd[row] = rs;
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = j * 32 + lane;
    if (v >= nvec) continue;
    float g[8], b[8];
    load8(gamma + v * 8, vec, g);
    load8(beta + v * 8, vec, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) a.v[j][k] = (a.v[j][k] - m) * rs * g[k] + b[k];
    y[row * nvec + v] = pack8(a.v[j]);
  }
}

// Backward of a row: ds = rstd * (g dy - mean(g dy) - xhat * mean(g dy xhat)); column sums of dy xhat and dy, and with
// kEmbed of ds, over the rows a warp visits, then over the block's warps, one partial row per block.
template <int NV, bool kEmbed>
__global__ void __launch_bounds__(kThreads)
    layer_norm_backward_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ sum, const int64_t* __restrict__ ids,
                               int64_t vocab, const float* __restrict__ tok, const float* __restrict__ pos, const float* __restrict__ typ,
                               const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
                               uint4* __restrict__ ds, float* __restrict__ ds32, float* __restrict__ partial, int64_t rows,
                               int64_t seq, int H, bool vec) {
  constexpr int kSums = kEmbed ? 3 : 2;
  extern __shared__ float s_sum[];  // [kSums][H]
  wait_for_predecessor();
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5, nvec = H / 8;
  float acc[kSums][NV][8];
#pragma unroll
  for (int q = 0; q < kSums; ++q)
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[q][j][k] = 0.f;
  for (int64_t row = (int64_t)blockIdx.x * kWarps + warp; row < rows; row += (int64_t)gridDim.x * kWarps) {
    const float m = mean[row], rs = rstd[row];
    Row<NV> x, g;  // xhat, then g dy
    if constexpr (kEmbed) gather_row<NV>(ids, vocab, tok, pos, typ, row, seq, H, nvec, lane, vec, x);
    float c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = j * 32 + lane;
      if (v >= nvec) continue;
      if constexpr (!kEmbed) unpack8(sum[row * nvec + v], x.v[j]);
      float w[8];
      unpack8(dy[row * nvec + v], g.v[j]);
      load8(gamma + v * 8, vec, w);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        x.v[j][k] = (x.v[j][k] - m) * rs;
        acc[0][j][k] += g.v[j][k] * x.v[j][k];
        acc[1][j][k] += g.v[j][k];
        g.v[j][k] *= w[k];
        c1 += g.v[j][k];
        c2 += g.v[j][k] * x.v[j][k];
      }
    }
    c1 = warp_sum(c1) / (float)H;
    c2 = warp_sum(c2) / (float)H;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = j * 32 + lane;
      if (v >= nvec) continue;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        g.v[j][k] = rs * (g.v[j][k] - c1 - x.v[j][k] * c2);
        if constexpr (kEmbed) acc[2][j][k] += g.v[j][k];
      }
      if constexpr (kEmbed) {
        float4* o = reinterpret_cast<float4*>(ds32 + row * H + v * 8);
        o[0] = make_float4(g.v[j][0], g.v[j][1], g.v[j][2], g.v[j][3]);
        o[1] = make_float4(g.v[j][4], g.v[j][5], g.v[j][6], g.v[j][7]);
      } else {
        ds[row * nvec + v] = pack8(g.v[j]);
      }
    }
  }
  // the block's warps add up in order
  for (int w = 0; w < kWarps; ++w) {
    if (warp == w) {
#pragma unroll
      for (int q = 0; q < kSums; ++q)
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int v = j * 32 + lane;
          if (v >= nvec) continue;
          float* o = s_sum + q * H + v * 8;
#pragma unroll
          for (int k = 0; k < 8; ++k) o[k] = w == 0 ? acc[q][j][k] : o[k] + acc[q][j][k];
        }
    }
    __syncthreads();
  }
  for (int c = (int)threadIdx.x; c < kSums * H; c += kThreads) partial[(size_t)blockIdx.x * kSums * H + c] = s_sum[c];
}

// Column sums of `blocks` partial rows of several vectors of H columns each, to as many destinations.
constexpr int kFoldCols = 32, kFoldRows = 16;
struct FoldTargets {
  float* out[3];
  bool add[3];
};
__global__ void __launch_bounds__(kFoldCols * kFoldRows)
    fold_kernel(const float* __restrict__ partial, FoldTargets to, int blocks, int H, int vectors) {
  __shared__ float s_acc[kFoldRows][kFoldCols];
  wait_for_predecessor();
  const int C = H * vectors, c = (int)(blockIdx.x * kFoldCols + threadIdx.x);
  float s = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int b = (int)threadIdx.y; b < blocks; b += kFoldRows) s += partial[(size_t)b * C + c];
  }
  s_acc[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || c >= C) return;
  s = 0.f;
#pragma unroll
  for (int r = 0; r < kFoldRows; ++r) s += s_acc[r][threadIdx.x];
  const int q = c / H;
  float* o = to.out[q] + (c - q * H);
  *o = to.add[q] ? *o + s : s;
}
void fold(const float* partial, const FoldTargets& to, int blocks, int H, int vectors, cudaStream_t s) {
  launch_overlapped(fold_kernel, dim3((H * vectors + kFoldCols - 1) / kFoldCols), dim3(kFoldCols, kFoldRows), s, partial, to,
                    blocks, H, vectors);
}

// ---- gradients of the embedding tables ------------------------------------------------------------
// Block i belongs to token i of the batch.  Its occurrences are found by looking over all ids (T of them, from
// L2); the first of every kMaxOrdered occurrences adds up that many rows, in order.  Blocks of the first
// sequence also add up their position over the batch.  The framework's path writes a dense gradient of the
// whole table (zero fill, scatter, addition: about 240 us for 30522 x 1024 and 3072 tokens); this touches the
// rows that occur.
__global__ void __launch_bounds__(kThreads)
    embed_scatter_kernel(const int64_t* __restrict__ ids, int64_t vocab, const float* __restrict__ ds, float* __restrict__ dtok,
                         float* __restrict__ dpos, int64_t batch, int64_t seq, int H) {
  __shared__ int s_list[kMaxOrdered];
  __shared__ int s_warp[kWarps];
  wait_for_predecessor();
  const int T = (int)(batch * seq), i = (int)blockIdx.x, tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (i < seq) {
    for (int c = tid; c < H; c += kThreads) {
      float s = 0.f;
#pragma unroll 4
      for (int64_t b = 0; b < batch; ++b) s += ds[(b * seq + i) * H + c];
      dpos[(size_t)i * H + c] += s;
    }
  }
  const int64_t id = ids[i];
  if (id < 0 || id >= vocab) return;
  int before = 0;
  for (int j = tid; j < i; j += kThreads) before += ids[j] == id;
  // exact rank of this occurrence, when it is not the first
  int rank = 0;
  if (__syncthreads_or(before)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) s_warp[warp] = before;
    __syncthreads();
    for (int w = 0; w < kWarps; ++w) rank += s_warp[w];
    __syncthreads();
  }
  if (rank % kMaxOrdered != 0) return;
  // this and the next kMaxOrdered - 1 occurrences, in order
  int found = 0;
  bool more = false;
  for (int j0 = i; j0 < T; j0 += kThreads) {
    const int j = j0 + tid;
    const bool hit = j < T && ids[j] == id;
    const unsigned ballot = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) s_warp[warp] = __popc(ballot);
    __syncthreads();
    int at = found, total = 0;
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) at += s_warp[w];
      total += s_warp[w];
    }
    at += __popc(ballot & ((1u << lane) - 1u));
    if (hit && at < kMaxOrdered) s_list[at] = j;
    found += total;
    __syncthreads();
    if (found > kMaxOrdered) {
      more = true;
      break;
    }
  }
  const int n = found < kMaxOrdered ? found : kMaxOrdered;
  const bool shared = more || rank > 0;  // several blocks add to this row
  float* out = dtok + (size_t)id * H;
  for (int c = tid; c < H; c += kThreads) {
    float s = 0.f;
#pragma unroll 8
    for (int k = 0; k < n; ++k) s += ds[(size_t)s_list[k] * H + c];
    if (shared)
      atomicAdd(out + c, s);
    else
      out[c] += s;
  }
}

// ---- GELU -------------------------------------------------------------------------------------------
constexpr float kSqrtHalf = 0.70710678118654752440f, kInvSqrt2Pi = 0.39894228040143267794f;

__global__ void __launch_bounds__(kThreads) gelu_kernel(const uint4* __restrict__ z, uint4* __restrict__ y, int64_t nvec) {
  wait_for_predecessor();
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < nvec; v += stride) {
    float f[8];
    unpack8(z[v], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = f[k] * 0.5f * (1.f + erff(f[k] * kSqrtHalf));
    y[v] = pack8(f);
  }
}

// Warps on rows, lanes on 8 columns each, as in the column sum of a linear layer's bias gradient.
__global__ void __launch_bounds__(kThreads)
    gelu_backward_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ z, uint4* __restrict__ dz,
                         float* __restrict__ partial, int64_t rows, int cgroups) {
  __shared__ float s_acc[kThreads * 8];
  wait_for_predecessor();
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
  const int cg = (int)blockIdx.x * 32 + lane;
  const int64_t per = (rows + gridDim.y - 1) / gridDim.y;
  const int64_t lo = (int64_t)blockIdx.y * per, hi = min(lo + per, rows);
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  if (cg < cgroups) {
#pragma unroll 2
    for (int64_t r = lo + warp; r < hi; r += kWarps) {
      float f[8], g[8];
      unpack8(z[r * cgroups + cg], f);
      unpack8(dy[r * cgroups + cg], g);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float cdf = 0.5f * (1.f + erff(f[k] * kSqrtHalf));
        const float pdf = expf(-0.5f * f[k] * f[k]) * kInvSqrt2Pi;
        g[k] *= cdf + f[k] * pdf;
      }
      const uint4 packed = pack8(g);
      dz[r * cgroups + cg] = packed;
      unpack8(packed, g);  // the sums are those of what was written
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += g[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s_acc[threadIdx.x * 8 + k] = acc[k];
  __syncthreads();
  const int c = (int)blockIdx.x * 256 + (int)threadIdx.x;
  if (c < cgroups * 8) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += s_acc[w * 256 + threadIdx.x];
    partial[(size_t)blockIdx.y * cgroups * 8 + c] = s;
  }
}
int gelu_splits(int64_t rows, int C) {
  const int col_blocks = (C / 8 + 31) / 32;
  return (int)std::max<int64_t>(1, std::min<int64_t>((rows + kWarps - 1) / kWarps, 4 * 148 / col_blocks));
}

// ---- attention gradients ------------------------------------------------------------------------------
struct MergeArgs {
  const uint4* src[3];
  HeadStrides stride[3];  // in vectors of 8
};
__global__ void __launch_bounds__(kThreads)
    merge_heads_kernel(const __grid_constant__ MergeArgs a, uint4* __restrict__ out, int64_t nvec, int64_t seq, int heads, int dvecs) {
  wait_for_predecessor();
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < nvec; v += stride) {
    uint32_t t = (uint32_t)v;
    const uint32_t d = t % (uint32_t)dvecs;
    t /= (uint32_t)dvecs;
    const uint32_t h = t % (uint32_t)heads;
    t /= (uint32_t)heads;
    const uint32_t q = t % 3u;
    t /= 3u;
    const uint32_t s = t % (uint32_t)seq, b = t / (uint32_t)seq;
    const HeadStrides& st = a.stride[q];
    out[v] = a.src[q][b * st.batch + h * st.head + s * st.seq + d];
  }
}

// Blocks of the row kernels whose warps each walk several rows: enough for every SM, few enough partial rows to fold.
int walk_blocks(int64_t rows) { return (int)std::max<int64_t>(1, std::min<int64_t>((rows + kWarps - 1) / kWarps, sm_count())); }

bool aligned16(const float* a, const float* b, const float* c = nullptr, const float* d = nullptr, const float* e = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d | (uintptr_t)e) & 15u) == 0;
}

// The instantiation for H: 256 columns per vector of a lane.
template <typename F>
void with_vecs(int H, F&& f) {
  switch ((H + 255) / 256) {
    case 1: f(std::integral_constant<int, 1>{}); return;
    case 2: f(std::integral_constant<int, 2>{}); return;
    case 3: f(std::integral_constant<int, 3>{}); return;
    default: f(std::integral_constant<int, 4>{}); return;
  }
}

}  // namespace

void add_layer_norm_forward(const void* x, const void* r, const float* gamma, const float* beta, float eps, void* sum, void* y,
                            float* mean, float* rstd, int64_t rows, int H, cudaStream_t s) {
  BAGUA_CHECK(row_supported(rows, H), Tensor, "layer norm: unsupported shape [" << rows << ", " << H << "]");
  with_vecs(H, [&](auto nv) {
    launch_overlapped(add_layer_norm_kernel<nv.value>, dim3((unsigned)((rows + kWarps - 1) / kWarps)), dim3(kThreads), s,
                      (const uint4*)x, (const uint4*)r, gamma, beta, eps, (uint4*)sum, (uint4*)y, mean, rstd, rows, H,
                      aligned16(gamma, beta));
  });
}

size_t layer_norm_backward_scratch_bytes(int64_t rows, int H) { return (size_t)walk_blocks(rows) * 2 * H * sizeof(float); }
void layer_norm_backward(const void* dy, const void* sum, const float* gamma, const float* mean, const float* rstd, void* ds,
                         float* dgamma, float* dbeta, bool add_gamma, bool add_beta, void* scratch, int64_t rows, int H,
                         cudaStream_t s) {
  BAGUA_CHECK(row_supported(rows, H), Tensor, "layer norm: unsupported shape [" << rows << ", " << H << "]");
  const int blocks = walk_blocks(rows);
  with_vecs(H, [&](auto nv) {
    kernels::launch_overlapped_shared(layer_norm_backward_kernel<nv.value, false>, dim3(blocks), dim3(kThreads),
                                      (size_t)2 * H * sizeof(float), s, (const uint4*)dy, (const uint4*)sum,
                                      (const int64_t*)nullptr, (int64_t)0, (const float*)nullptr, (const float*)nullptr,
                                      (const float*)nullptr, gamma, mean, rstd, (uint4*)ds, (float*)nullptr, (float*)scratch,
                                      rows, (int64_t)1, H, aligned16(gamma, gamma));
  });
  fold((const float*)scratch, FoldTargets{{dgamma, dbeta, nullptr}, {add_gamma, add_beta, false}}, blocks, H, 2, s);
}

void embed_layer_norm_forward(const int64_t* ids, int64_t vocab, const float* tok, const float* pos, const float* typ, const float* gamma,
                              const float* beta, float eps, void* y, float* mean, float* rstd, int64_t batch, int64_t seq, int H,
                              cudaStream_t s) {
  const int64_t rows = batch * seq;
  BAGUA_CHECK(row_supported(rows, H), Tensor, "embedding: unsupported shape [" << rows << ", " << H << "]");
  with_vecs(H, [&](auto nv) {
    launch_overlapped(embed_layer_norm_kernel<nv.value>, dim3((unsigned)((rows + kWarps - 1) / kWarps)), dim3(kThreads), s, ids,
                      vocab, tok, pos, typ, gamma, beta, eps, (uint4*)y, mean, rstd, rows, seq, H,
                      aligned16(gamma, beta, tok, pos, typ));
  });
}

size_t embed_backward_scratch_bytes(int64_t rows, int H) { return (size_t)walk_blocks(rows) * 3 * H * sizeof(float); }
void embed_layer_norm_backward(const void* dy, const int64_t* ids, int64_t vocab, const float* tok, const float* pos, const float* typ,
                               const float* gamma, const float* mean, const float* rstd, float* ds, float* dtok, float* dpos,
                               float* dtyp, float* dgamma, float* dbeta, void* scratch, int64_t batch, int64_t seq, int H,
                               cudaStream_t s) {
  const int64_t rows = batch * seq;
  BAGUA_CHECK(row_supported(rows, H) && rows <= kMaxTokens, Tensor,
              "embedding backward: unsupported shape [" << rows << ", " << H << "]");
  const int blocks = walk_blocks(rows);
  with_vecs(H, [&](auto nv) {
    kernels::launch_overlapped_shared(layer_norm_backward_kernel<nv.value, true>, dim3(blocks), dim3(kThreads),
                                      (size_t)3 * H * sizeof(float), s, (const uint4*)dy, (const uint4*)nullptr, ids, vocab, tok, pos,
                                      typ, gamma, mean, rstd, (uint4*)nullptr, ds, (float*)scratch, rows, seq, H,
                                      aligned16(gamma, gamma, tok, pos, typ));
  });
  fold((const float*)scratch, FoldTargets{{dgamma, dbeta, dtyp}, {true, true, true}}, blocks, H, 3, s);
  launch_overlapped(embed_scatter_kernel, dim3((unsigned)rows), dim3(kThreads), s, ids, vocab, (const float*)ds, dtok, dpos, batch, seq,
                    H);
}

void gelu_forward(const void* z, void* y, int64_t n, cudaStream_t s) {
  BAGUA_CHECK(n % 8 == 0 && n > 0, Tensor, "gelu: " << n << " elements");
  const int64_t blocks = (n / 8 + kThreads - 1) / kThreads;
  launch_overlapped(gelu_kernel, dim3((unsigned)std::min<int64_t>(blocks, (int64_t)sm_count() * 8)), dim3(kThreads), s,
                    (const uint4*)z, (uint4*)y, n / 8);
}
size_t gelu_backward_scratch_bytes(int64_t rows, int C) { return (size_t)gelu_splits(rows, C) * C * sizeof(float); }
void gelu_backward(const void* dy, const void* z, void* dz, float* db, bool accumulate, void* scratch, int64_t rows, int C,
                   cudaStream_t s) {
  BAGUA_CHECK(rows > 0 && C % 8 == 0, Tensor, "gelu backward: unsupported shape [" << rows << ", " << C << "]");
  const int splits = gelu_splits(rows, C);
  launch_overlapped(gelu_backward_kernel, dim3((C / 8 + 31) / 32, splits), dim3(kThreads), s, (const uint4*)dy, (const uint4*)z,
                    (uint4*)dz, (float*)scratch, rows, C / 8);
  fold((const float*)scratch, FoldTargets{{db, nullptr, nullptr}, {accumulate, false, false}}, splits, C, 1, s);
}

void merge_heads(const void* const src[3], const HeadStrides stride[3], void* out, int64_t batch, int64_t seq, int heads,
                 int dim, cudaStream_t s) {
  const int64_t nvec = batch * seq * 3 * heads * (dim / 8);
  BAGUA_CHECK(dim % 8 == 0 && nvec > 0 && nvec < (1ll << 32), Tensor, "merge_heads: unsupported shape");
  MergeArgs a;
  for (int q = 0; q < 3; ++q) {
    a.src[q] = (const uint4*)src[q];
    a.stride[q] = HeadStrides{stride[q].batch / 8, stride[q].head / 8, stride[q].seq / 8};
  }
  const int64_t blocks = (nvec + kThreads - 1) / kThreads;
  launch_overlapped(merge_heads_kernel, dim3((unsigned)std::min<int64_t>(blocks, (int64_t)sm_count() * 8)), dim3(kThreads), s, a,
                    (uint4*)out, nvec, seq, heads, dim / 8);
}

}  // namespace encoder_ops
}  // namespace bagua
