// See encoder_ops.h.  All kernels are latency- and bandwidth-bound streams over activations of a few MB that
// mostly sit in L2: 16-byte vectors, enough blocks for every SM, column sums kept in registers over the rows a warp
// visits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>

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
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Column sums of `blocks` partial rows.
constexpr int kFoldCols = 32, kFoldRows = 16;
__global__ void __launch_bounds__(kFoldCols * kFoldRows)
    fold_kernel(const float* __restrict__ partial, float* __restrict__ out, int blocks, int C, bool accumulate) {
  __shared__ float s_acc[kFoldRows][kFoldCols];
  wait_for_predecessor();
  const int c = (int)(blockIdx.x * kFoldCols + threadIdx.x);
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
  out[c] = accumulate ? out[c] + s : s;
}
void fold(const float* partial, float* out, int blocks, int C, bool accumulate, cudaStream_t s) {
  launch_overlapped(fold_kernel, dim3((C + kFoldCols - 1) / kFoldCols), dim3(kFoldCols, kFoldRows), s, partial, out, blocks, C,
                    accumulate);
}

// ---- indices outside their table -------------------------------------------------------------------
// A kernel skips them and leaves the last one here, in host memory: the value first, then that there is one.
struct IndexReport {
  long long value[2];  // by kind: a token's id, a span's target
  unsigned int seen[2];
};
enum { kTokenId = 0, kSpanTarget = 1 };
__device__ __noinline__ void report_index(IndexReport* r, int kind, int64_t value) {
  *(volatile long long*)&r->value[kind] = value;
  __threadfence_system();
  *(volatile unsigned int*)&r->seen[kind] = 1u;
}
// One per device, never given back: a captured graph keeps its address.
IndexReport* index_report() {
  static std::atomic<IndexReport*> reports[64] = {};
  static std::mutex mu;
  int dev = 0;
  BAGUA_CUDA_CHECK(cudaGetDevice(&dev));
  BAGUA_CHECK(dev >= 0 && dev < 64, Tensor, "device index " << dev << " out of range");
  if (IndexReport* r = reports[dev].load(std::memory_order_acquire)) return r;
  std::lock_guard<std::mutex> g(mu);
  if (!reports[dev].load()) {
    // allowed while a stream is being captured, as nothing is enqueued
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    BAGUA_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
    IndexReport* r = nullptr;
    const cudaError_t e = cudaHostAlloc((void**)&r, sizeof(IndexReport), cudaHostAllocMapped);
    BAGUA_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
    BAGUA_CUDA_CHECK(e);
    std::memset(r, 0, sizeof(IndexReport));
    reports[dev].store(r, std::memory_order_release);
  }
  return reports[dev].load();
}

// ---- embedding ------------------------------------------------------------------------------------
// x[row] = (tok[id] + pos[position]) + typ, in this order, in fp32; an id outside the table gives a row of NaN.
__global__ void __launch_bounds__(kThreads)
    embed_sum_kernel(const int64_t* __restrict__ ids, int64_t vocab, const float* __restrict__ tok, const float* __restrict__ pos,
                     const float* __restrict__ typ, float* __restrict__ x, int64_t seq, int H, IndexReport* report) {
  wait_for_predecessor();
  const int64_t row = blockIdx.x, id = ids[row];
  const bool known = id >= 0 && id < vocab;
  if (!known && threadIdx.x == 0) report_index(report, kTokenId, id);
  const float* t = tok + (known ? id : 0) * H;
  const float* p = pos + (row % seq) * H;
  for (int c = (int)threadIdx.x; c < H; c += kThreads) x[row * H + c] = known ? t[c] + p[c] + typ[c] : nanf("");
}

// Column sums of x [rows, H] in fp32: threads on columns, one partial row per slice of rows.
__global__ void __launch_bounds__(kThreads)
    column_sum_f32_kernel(const float* __restrict__ x, float* __restrict__ partial, int64_t rows, int H) {
  wait_for_predecessor();
  const int c = (int)(blockIdx.x * kThreads + threadIdx.x);
  if (c >= H) return;
  const int64_t per = (rows + gridDim.y - 1) / gridDim.y, lo = (int64_t)blockIdx.y * per, hi = min(lo + per, rows);
  float s = 0.f;
#pragma unroll 8
  for (int64_t r = lo; r < hi; ++r) s += x[r * H + c];
  partial[(size_t)blockIdx.y * H + c] = s;
}
int column_slices(int64_t rows, int H) {
  const int64_t col_blocks = (H + kThreads - 1) / kThreads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(rows / 8, 2 * 148 / col_blocks));
}

// ---- gradients of the embedding tables ------------------------------------------------------------
// Block i belongs to token i of the batch.  Its occurrences are found by looking over all ids (T of them, from
// L2); the first of every kMaxOrdered occurrences adds up that many rows, in order.  Blocks of the first
// sequence also add up their position over the batch.  The framework's path writes a dense gradient of the
// whole table (zero fill, scatter, addition: about 240 us for 30522 x 1024 and 3072 tokens); this touches the
// rows that occur.  Either table may be missing (null): its gradient is not wanted.
__global__ void __launch_bounds__(kThreads)
    embed_scatter_kernel(const int64_t* __restrict__ ids, int64_t vocab, const float* __restrict__ ds, float* __restrict__ dtok,
                         float* __restrict__ dpos, int64_t batch, int64_t seq, int H) {
  __shared__ int s_list[kMaxOrdered];
  __shared__ int s_warp[kWarps];
  wait_for_predecessor();
  const int T = (int)(batch * seq), i = (int)blockIdx.x, tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (dpos && i < seq) {
    for (int c = tid; c < H; c += kThreads) {
      float s = 0.f;
#pragma unroll 4
      for (int64_t b = 0; b < batch; ++b) s += ds[(b * seq + i) * H + c];
      dpos[(size_t)i * H + c] += s;
    }
  }
  const int64_t id = ids[i];
  if (!dtok || id < 0 || id >= vocab) return;
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

// Warps on rows, lanes on 8 columns each, as in the column sum of a linear layer's bias gradient.  `z`: what the
// activation was applied to, or for ReLU its result.
template <bool kGelu>
__global__ void __launch_bounds__(kThreads)
    activation_backward_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ z, uint4* __restrict__ dz,
                               float* __restrict__ partial, int64_t rows, int cgroups, bool accumulate) {
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
        if constexpr (kGelu) {
          const float cdf = 0.5f * (1.f + erff(f[k] * kSqrtHalf));
          const float pdf = expf(-0.5f * f[k] * f[k]) * kInvSqrt2Pi;
          g[k] *= cdf + f[k] * pdf;
        } else {
          g[k] = f[k] > 0.f ? g[k] : 0.f;
        }
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
    float* out = partial + (size_t)blockIdx.y * cgroups * 8 + c;
    *out = accumulate ? *out + s : s;
  }
}
int activation_splits(int64_t rows, int C) {
  const int col_blocks = (C / 8 + 31) / 32;
  if (rows <= 64) return 1;  // the one slice's sums are the result: one launch
  return (int)std::max<int64_t>(1, std::min<int64_t>((rows + kWarps - 1) / kWarps, 4 * 148 / col_blocks));
}

// ---- loss of a span prediction ------------------------------------------------------------------------
// (cross_entropy(logits[..., 0], start) + cross_entropy(logits[..., 1], end)) / 2 with means over the rows whose target
// is not -100.  A few thousand values: one block, a warp per row, both columns of a row from one read.  As framework
// calls: 10 launches forward, 16 backward.  A target outside the sequence gives NaN.
constexpr int kSpanThreads = 1024;
constexpr int64_t kIgnored = -100;
__global__ void __launch_bounds__(kSpanThreads)
    span_loss_kernel(const __nv_bfloat162* __restrict__ logits, const int64_t* __restrict__ start,
                     const int64_t* __restrict__ end, float* __restrict__ loss, float* __restrict__ stats, int batch, int seq,
                     IndexReport* report) {
  // stats: [batch][2] log-sum-exp, then the two counts
  __shared__ float s_loss[32][2];
  __shared__ float s_count[32][2];
  wait_for_predecessor();
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
  float l[2] = {0.f, 0.f}, n[2] = {0.f, 0.f};
  for (int b = warp; b < batch; b += kSpanThreads / 32) {
    const __nv_bfloat162* row = logits + (size_t)b * seq;
    float m0 = -INFINITY, m1 = -INFINITY;
    for (int i = lane; i < seq; i += 32) {
      const float2 v = __bfloat1622float2(row[i]);
      m0 = fmaxf(m0, v.x);
      m1 = fmaxf(m1, v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    }
    float e0 = 0.f, e1 = 0.f;
    for (int i = lane; i < seq; i += 32) {
      const float2 v = __bfloat1622float2(row[i]);
      e0 += expf(v.x - m0);
      e1 += expf(v.y - m1);
    }
    const float lse0 = m0 + logf(warp_sum(e0)), lse1 = m1 + logf(warp_sum(e1));
    if (lane == 0) {
      stats[2 * b] = lse0;
      stats[2 * b + 1] = lse1;
      const int64_t t0 = start[b], t1 = end[b];
      const bool in0 = t0 >= 0 && t0 < seq, in1 = t1 >= 0 && t1 < seq;
      if (t0 != kIgnored) {
        l[0] += in0 ? lse0 - __bfloat162float(row[t0].x) : nanf("");
        n[0] += 1.f;
        if (!in0) report_index(report, kSpanTarget, t0);
      }
      if (t1 != kIgnored) {
        l[1] += in1 ? lse1 - __bfloat162float(row[t1].y) : nanf("");
        n[1] += 1.f;
        if (!in1) report_index(report, kSpanTarget, t1);
      }
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      s_loss[warp][k] = l[k];
      s_count[warp][k] = n[k];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float a[2] = {0.f, 0.f}, c[2] = {0.f, 0.f};
    for (int w = 0; w < 32; ++w)
      for (int k = 0; k < 2; ++k) {
        a[k] += s_loss[w][k];
        c[k] += s_count[w][k];
      }
    stats[2 * batch] = c[0];
    stats[2 * batch + 1] = c[1];
    *loss = (a[0] / c[0] + a[1] / c[1]) / 2.f;
  }
}
__global__ void __launch_bounds__(kThreads)
    span_loss_backward_kernel(const __nv_bfloat162* __restrict__ logits, const int64_t* __restrict__ start,
                              const int64_t* __restrict__ end, const float* __restrict__ stats,
                              const float* __restrict__ dloss, __nv_bfloat162* __restrict__ dlogits, int batch, int seq) {
  wait_for_predecessor();
  const int n = batch * seq;
  const float g = *dloss * 0.5f, g0 = g / stats[2 * batch], g1 = g / stats[2 * batch + 1];
  for (int v = (int)(blockIdx.x * kThreads + threadIdx.x); v < n; v += (int)gridDim.x * kThreads) {
    const int b = v / seq, i = v - b * seq;
    const float2 x = __bfloat1622float2(logits[v]);
    const int64_t t0 = start[b], t1 = end[b];
    const float d0 = t0 == kIgnored ? 0.f : (expf(x.x - stats[2 * b]) - (t0 == i ? 1.f : 0.f)) * g0;
    const float d1 = t1 == kIgnored ? 0.f : (expf(x.y - stats[2 * b + 1]) - (t1 == i ? 1.f : 0.f)) * g1;
    dlogits[v] = __floats2bfloat162_rn(d0, d1);
  }
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

}  // namespace

void check_indices() {
  IndexReport* r = index_report();
  for (int kind : {kTokenId, kSpanTarget}) {
    volatile unsigned int* seen = &r->seen[kind];
    if (*seen == 0) continue;
    const long long value = *(volatile long long*)&r->value[kind];
    *seen = 0;
    throw BaguaError(ErrorKind::Tensor, (kind == kTokenId ? "an earlier call was given the token id " : "an earlier call was given the span target ") +
                                            std::to_string(value) + (kind == kTokenId ? ", which is not in the table" : ", which is not in the sequence"));
  }
}

void embed_sum(const int64_t* ids, int64_t vocab, const float* tok, const float* pos, const float* typ, float* x, int64_t batch,
               int64_t seq, int H, cudaStream_t s) {
  launch_overlapped(embed_sum_kernel, dim3((unsigned)(batch * seq)), dim3(kThreads), s, ids, vocab, tok, pos, typ, x, seq, H,
                    index_report());
}

size_t embed_backward_scratch_bytes(int64_t rows, int H) { return (size_t)column_slices(rows, H) * H * sizeof(float); }
int embed_backward(const float* dx, const int64_t* ids, int64_t vocab, float* dtok, float* dpos, float* dtyp, void* scratch,
                   int64_t batch, int64_t seq, int H, cudaStream_t s) {
  const int64_t rows = batch * seq;
  BAGUA_CHECK(rows > 0 && rows <= kMaxTokens, Tensor, "embedding backward: " << rows << " tokens");
  int launches = 0;
  if (dtyp) {
    const int slices = column_slices(rows, H);
    launch_overlapped(column_sum_f32_kernel, dim3((H + kThreads - 1) / kThreads, slices), dim3(kThreads), s, dx, (float*)scratch,
                      rows, H);
    fold((const float*)scratch, dtyp, slices, H, true, s);
    launches += 2;
  }
  if (dtok || dpos) {
    launch_overlapped(embed_scatter_kernel, dim3((unsigned)(dtok ? rows : seq)), dim3(kThreads), s, ids, vocab, dx, dtok, dpos,
                      batch, seq, H);
    ++launches;
  }
  return launches;
}

void gelu_forward(const void* z, void* y, int64_t n, cudaStream_t s) {
  BAGUA_CHECK(n % 8 == 0 && n > 0, Tensor, "gelu: " << n << " elements");
  const int64_t blocks = (n / 8 + kThreads - 1) / kThreads;
  launch_overlapped(gelu_kernel, dim3((unsigned)std::min<int64_t>(blocks, (int64_t)sm_count() * 8)), dim3(kThreads), s,
                    (const uint4*)z, (uint4*)y, n / 8);
}
size_t activation_backward_scratch_bytes(int64_t rows, int C) {
  const int splits = activation_splits(rows, C);
  return splits == 1 ? 0 : (size_t)splits * C * sizeof(float);
}
void activation_backward(bool gelu, const void* dy, const void* z, void* dz, float* db, bool accumulate, void* scratch,
                         int64_t rows, int C, cudaStream_t s) {
  BAGUA_CHECK(rows > 0 && C % 8 == 0, Tensor, "activation backward: unsupported shape [" << rows << ", " << C << "]");
  const int splits = activation_splits(rows, C);
  const bool direct = splits == 1;
  launch_overlapped(gelu ? activation_backward_kernel<true> : activation_backward_kernel<false>,
                    dim3((C / 8 + 31) / 32, splits), dim3(kThreads), s, (const uint4*)dy, (const uint4*)z, (uint4*)dz,
                    direct ? db : (float*)scratch, rows, C / 8, direct && accumulate);
  if (!direct) fold((const float*)scratch, db, splits, C, accumulate, s);
}

void span_loss_forward(const void* logits, const int64_t* start, const int64_t* end, float* loss, float* stats, int64_t batch,
                       int64_t seq, cudaStream_t s) {
  BAGUA_CHECK(batch > 0 && seq > 0 && batch * seq < (1ll << 30), Tensor, "span loss: unsupported shape");
  launch_overlapped(span_loss_kernel, dim3(1), dim3(kSpanThreads), s, (const __nv_bfloat162*)logits, start, end, loss, stats,
                    (int)batch, (int)seq, index_report());
}
void span_loss_backward(const void* logits, const int64_t* start, const int64_t* end, const float* stats, const float* dloss,
                        void* dlogits, int64_t batch, int64_t seq, cudaStream_t s) {
  const int64_t n = batch * seq;
  launch_overlapped(span_loss_backward_kernel, dim3((unsigned)std::min<int64_t>((n + kThreads - 1) / kThreads, sm_count() * 8)),
                    dim3(kThreads), s, (const __nv_bfloat162*)logits, start, end, stats, dloss, (__nv_bfloat162*)dlogits,
                    (int)batch, (int)seq);
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
