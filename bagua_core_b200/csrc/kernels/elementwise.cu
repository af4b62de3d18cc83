// sm_100a element-wise and chunk-reduce kernels.
//
// All are HBM-bound streaming kernels: 16-byte accesses, 64-bit indexing, grid sized as
// a multiple of the 148 SMs, fp32 arithmetic with one rounding on store.  They replace
// the reference's scalar 4-byte grid-stride kernels and its shared-memory tree reduce
// (bagua-core-internal/kernels/bagua_kernels.cu:196-266,373-400).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels_impl.h"
#include "launch.cuh"

namespace bagua {
namespace kernels {
namespace cuda {

namespace {

constexpr int kThreads = 256;

template <typename T>
struct VecTraits;
template <>
struct VecTraits<float> {
  static constexpr int N = 4;
};
template <>
struct VecTraits<__half> {
  static constexpr int N = 8;
};
template <>
struct VecTraits<__nv_bfloat16> {
  static constexpr int N = 8;
};

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename T>
struct alignas(16) Pack {
  T v[VecTraits<T>::N];
};

// Two items per thread, as many blocks as that takes.  (Large streams are slower through the 1184 blocks that are resident at a time, each
// with a share of the whole: those run apart, and the memory sees all their places at once, while blocks that come and go pass over
// it as one front.  100 M elements, resident / as here, us: average of fp32 191 / 172, of bf16 98 / 88; bf16 added to fp32 165 / 145;
// asynchronous average 277 / 274, but 307 with one item per thread.)
inline int grid_for(int64_t work_items) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((work_items + 2 * kThreads - 1) / (2 * kThreads), 1 << 30));
}

// x[i] = op(x[i], y[i]) (y may be null for unary ops)
template <typename T, typename Op, bool kVec>
__global__ void __launch_bounds__(kThreads) ew_kernel(T* __restrict__ x, const T* __restrict__ y, int64_t n, Op op) {
  constexpr int V = VecTraits<T>::N;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if constexpr (kVec) {
    const int64_t nv = n / V;
    auto* xv = reinterpret_cast<Pack<T>*>(x);
    auto* yv = reinterpret_cast<const Pack<T>*>(y);
    for (int64_t i = tid; i < nv; i += stride) {
      Pack<T> a = xv[i];
      Pack<T> b;
      if (y) b = yv[i];
#pragma unroll
      for (int k = 0; k < V; ++k) a.v[k] = from_f<T>(op(to_f(a.v[k]), y ? to_f(b.v[k]) : 0.f));
      xv[i] = a;
    }
    for (int64_t i = nv * V + tid; i < n; i += stride) x[i] = from_f<T>(op(to_f(x[i]), y ? to_f(y[i]) : 0.f));
  } else {
    for (int64_t i = tid; i < n; i += stride) x[i] = from_f<T>(op(to_f(x[i]), y ? to_f(y[i]) : 0.f));
  }
}

template <typename T, typename Op>
void launch_ew(void* x, const void* y, int64_t n, Op op, cudaStream_t s) {
  const bool aligned = ((uintptr_t)x % 16 == 0) && (y == nullptr || (uintptr_t)y % 16 == 0);
  if (aligned) {
    int grid = grid_for(n / VecTraits<T>::N + 1);
    ew_kernel<T, Op, true><<<grid, kThreads, 0, s>>>((T*)x, (const T*)y, n, op);
  } else {
    int grid = grid_for(n);
    ew_kernel<T, Op, false><<<grid, kThreads, 0, s>>>((T*)x, (const T*)y, n, op);
  }
  BAGUA_CUDA_CHECK(cudaGetLastError());
}

template <typename Op>
void dispatch_ew(void* x, const void* y, DType dt, int64_t n, Op op, cudaStream_t s) {
  switch (dt) {
    case DType::F32: launch_ew<float>(x, y, n, op, s); return;
    case DType::F16: launch_ew<__half>(x, y, n, op, s); return;
    case DType::BF16: launch_ew<__nv_bfloat16>(x, y, n, op, s); return;
    default: throw BaguaError(ErrorKind::Tensor, std::string("kernel does not support dtype ") + dtype_name(dt));
  }
}

struct OpDiv {
  float d;
  __device__ float operator()(float a, float) const { return a / d; }
};
struct OpAdd {
  __device__ float operator()(float a, float b) const { return a + b; }
};
struct OpSub {
  __device__ float operator()(float a, float b) const { return a - b; }
};
struct OpAddMul {
  float f;
  __device__ float operator()(float a, float b) const { return a + b * f; }
};
struct OpAvg {
  __device__ float operator()(float a, float b) const { return (a + b) * 0.5f; }
};

__global__ void __launch_bounds__(kThreads)
    async_avg_kernel(float* __restrict__ t, const float* __restrict__ r, const float* __restrict__ cp, float nranks,
                     int64_t n, bool vec) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if (vec) {
    const int64_t nv = n / 4;
    for (int64_t i = tid; i < nv; i += stride) {
      float4 a = reinterpret_cast<const float4*>(r)[i];
      float4 b = reinterpret_cast<const float4*>(cp)[i];
      float4 d = make_float4(a.x / nranks - b.x, a.y / nranks - b.y, a.z / nranks - b.z, a.w / nranks - b.w);
      // one 16-byte vector reduction instead of four scalar atomics
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(t + 4 * i), "f"(d.x), "f"(d.y), "f"(d.z),
                   "f"(d.w)
                   : "memory");
    }
    for (int64_t i = nv * 4 + tid; i < n; i += stride) atomicAdd(t + i, r[i] / nranks - cp[i]);
  } else {
    for (int64_t i = tid; i < n; i += stride) atomicAdd(t + i, r[i] / nranks - cp[i]);
  }
}

// x += y, y in bf16: 10 bytes per element where a cast to fp32 and an addition move 18.
__global__ void __launch_bounds__(kThreads)
    accumulate_bf16_kernel(float* __restrict__ x0, const __nv_bfloat16* __restrict__ y0, float* __restrict__ x1,
                           const __nv_bfloat16* __restrict__ y1, int64_t n, bool vec) {
  float* x = blockIdx.y == 0 ? x0 : x1;
  const __nv_bfloat16* y = blockIdx.y == 0 ? y0 : y1;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  wait_for_predecessor();
  int64_t done = 0;
  if (vec) {
    const int64_t nv = n / 4;
    for (int64_t i = tid; i < nv; i += stride) {
      float4 a = reinterpret_cast<float4*>(x)[i];
      const uint2 b = reinterpret_cast<const uint2*>(y)[i];
      const float2 lo = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(b.x));
      const float2 hi = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(b.y));
      a.x += lo.x;
      a.y += lo.y;
      a.z += hi.x;
      a.w += hi.y;
      reinterpret_cast<float4*>(x)[i] = a;
    }
    done = nv * 4;
  }
  for (int64_t i = done + tid; i < n; i += stride) x[i] += __bfloat162float(y[i]);
}

// fp32 -> bf16 of a few buffers in one launch: a layer's input, weight and bias under autocast, of which the bias
// alone used to cost a launch.  Tiles as in the SGD kernel, a block each (103 M elements: 87 us, 101 with 1184 resident blocks and four
// vectors per thread).
constexpr int kCastVecs = 2;
constexpr int kCastTile = kThreads * 4 * kCastVecs;
constexpr int kCastSegments = 8;
struct CastTable {
  CastSegment seg[kCastSegments];
  int64_t first_tile[kCastSegments + 1];
  int n;
};
__global__ void __launch_bounds__(kThreads) cast_bf16_kernel(const __grid_constant__ CastTable table) {
  wait_for_predecessor();
  int k = 0;
  while ((int64_t)blockIdx.x >= table.first_tile[k + 1]) ++k;
  const CastSegment& a = table.seg[k];
  const int64_t base = ((int64_t)blockIdx.x - table.first_tile[k]) * kCastTile;
  auto* dst = reinterpret_cast<__nv_bfloat16*>(a.dst);
  const bool vec = ((reinterpret_cast<uintptr_t>(a.src) & 15u) | (reinterpret_cast<uintptr_t>(a.dst) & 7u)) == 0;
  if (vec && base + kCastTile <= a.n) {
    float4 v[kCastVecs];
#pragma unroll
    for (int u = 0; u < kCastVecs; ++u) v[u] = reinterpret_cast<const float4*>(a.src + base)[u * kThreads + threadIdx.x];
#pragma unroll
    for (int u = 0; u < kCastVecs; ++u) {
      uint2 h;
      *reinterpret_cast<__nv_bfloat162*>(&h.x) = __floats2bfloat162_rn(v[u].x, v[u].y);
      *reinterpret_cast<__nv_bfloat162*>(&h.y) = __floats2bfloat162_rn(v[u].z, v[u].w);
      reinterpret_cast<uint2*>(dst + base)[u * kThreads + threadIdx.x] = h;
    }
  } else {
    const int64_t end = base + kCastTile < a.n ? base + kCastTile : a.n;
    for (int64_t i = base + threadIdx.x; i < end; i += kThreads) dst[i] = __float2bfloat16_rn(a.src[i]);
  }
}

// x as [n_chunks][chunk]; each thread owns V adjacent columns and walks the chunks.
template <typename T, bool kVec>
__global__ void __launch_bounds__(kThreads)
    reduce_chunk_kernel(T* __restrict__ x, int64_t chunk, int n_chunks, int target, float mul) {
  constexpr int V = VecTraits<T>::N;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if constexpr (kVec) {
    const int64_t nv = chunk / V;
    for (int64_t i = tid; i < nv; i += stride) {
      float acc[V];
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] = 0.f;
      for (int c = 0; c < n_chunks; ++c) {
        Pack<T> a = reinterpret_cast<const Pack<T>*>(x + (int64_t)c * chunk)[i];
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] += to_f(a.v[k]);
      }
      Pack<T> o;
#pragma unroll
      for (int k = 0; k < V; ++k) o.v[k] = from_f<T>(acc[k] * mul);
      reinterpret_cast<Pack<T>*>(x + (int64_t)target * chunk)[i] = o;
    }
  } else {
    for (int64_t i = tid; i < chunk; i += stride) {
      float acc = 0.f;
      for (int c = 0; c < n_chunks; ++c) acc += to_f(x[(int64_t)c * chunk + i]);
      x[(int64_t)target * chunk + i] = from_f<T>(acc * mul);
    }
  }
}

template <typename T>
void launch_reduce_chunk(void* x, int64_t chunk, int n_chunks, int target, bool average, cudaStream_t s) {
  constexpr int V = VecTraits<T>::N;
  // exact division keeps the mean bit-identical to sum / n for power-of-two n and within
  // 1 ulp otherwise; the host oracle divides, tests compare with a tolerance.
  const float mul = average ? 1.0f / (float)n_chunks : 1.0f;
  const bool vec = ((uintptr_t)x % 16 == 0) && (chunk % V == 0);
  if (vec) {
    reduce_chunk_kernel<T, true><<<grid_for(chunk / V), kThreads, 0, s>>>((T*)x, chunk, n_chunks, target, mul);
  } else {
    reduce_chunk_kernel<T, false><<<grid_for(chunk), kThreads, 0, s>>>((T*)x, chunk, n_chunks, target, mul);
  }
  BAGUA_CUDA_CHECK(cudaGetLastError());
}

__device__ __forceinline__ void sgd_update(const SgdSegment& a, float& pv, float gv, float& bv) {
  // fused multiply-adds spelled out: which of two products is rounded is not left to the compiler
  float d = __fmaf_rn(a.weight_decay, pv, gv);
  if (a.momentum != 0.f) {
    const float b = a.first ? d : __fmaf_rn(1.f - a.dampening, d, __fmul_rn(a.momentum, bv));
    bv = b;
    d = a.nesterov ? __fmaf_rn(a.momentum, b, d) : b;
  }
  pv = __fmaf_rn(-a.lr, d, pv);
}

// SGD steps of several flat buffers in one launch, each with its own hyperparameters: a stream of 20 bytes per
// parameter (22 with the bf16 copy), bound by memory.  One launch per buffer left the chip to drain and fill again
// between buffers of a few MB (10 buckets of 10 MB with bf16 copies: 108 us, 97 in one launch).
// Buffers are cut into tiles of kSgdTile elements, a block each; the table travels with the launch.  (Blocks that stay and take the tiles
// in turn are slower, see grid_for(): 138 M elements 485 us, 397 with a block per tile, 403 with tiles of two vectors per thread; those 10
// buckets of 25.6 M 102.6, 84.7, 88.2; 86 at the rate of a copy.)
constexpr int kSgdVecs = 1;
constexpr int kSgdTile = kThreads * 4 * kSgdVecs;
constexpr int kSgdSegments = 40;
struct SgdTable {
  SgdSegment seg[kSgdSegments];
  int64_t first_tile[kSgdSegments + 1];
  int n;
};

__global__ void __launch_bounds__(kThreads) sgd_kernel(const __grid_constant__ SgdTable table) {
  wait_for_predecessor();
  int k = 0;
  while ((int64_t)blockIdx.x >= table.first_tile[k + 1]) ++k;
  const SgdSegment& a = table.seg[k];
  const int64_t base = ((int64_t)blockIdx.x - table.first_tile[k]) * kSgdTile;
  const bool has_m = a.momentum != 0.f, read_m = has_m && !a.first;
  if (a.vec && base + kSgdTile <= a.n) {
    float4 pv[kSgdVecs], gv[kSgdVecs], bv[kSgdVecs];
#pragma unroll
    for (int u = 0; u < kSgdVecs; ++u) {
      const int64_t i = base / 4 + u * kThreads + threadIdx.x;
      pv[u] = reinterpret_cast<const float4*>(a.p)[i];
      gv[u] = reinterpret_cast<const float4*>(a.g)[i];
      bv[u] = read_m ? reinterpret_cast<const float4*>(a.m)[i] : make_float4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kSgdVecs; ++u) {
      const int64_t i = base / 4 + u * kThreads + threadIdx.x;
      sgd_update(a, pv[u].x, gv[u].x, bv[u].x);
      sgd_update(a, pv[u].y, gv[u].y, bv[u].y);
      sgd_update(a, pv[u].z, gv[u].z, bv[u].z);
      sgd_update(a, pv[u].w, gv[u].w, bv[u].w);
      reinterpret_cast<float4*>(a.p)[i] = pv[u];
      if (has_m) reinterpret_cast<float4*>(a.m)[i] = bv[u];
      if (a.shadow) {
        uint2 h;
        *reinterpret_cast<__nv_bfloat162*>(&h.x) = __floats2bfloat162_rn(pv[u].x, pv[u].y);
        *reinterpret_cast<__nv_bfloat162*>(&h.y) = __floats2bfloat162_rn(pv[u].z, pv[u].w);
        reinterpret_cast<uint2*>(a.shadow)[i] = h;
      }
    }
  } else {
    const int64_t end = base + kSgdTile < a.n ? base + kSgdTile : a.n;
    for (int64_t i = base + threadIdx.x; i < end; i += kThreads) {
      float pv = a.p[i], bv = read_m ? a.m[i] : 0.f;
      sgd_update(a, pv, a.g[i], bv);
      a.p[i] = pv;
      if (has_m) a.m[i] = bv;
      if (a.shadow) reinterpret_cast<__nv_bfloat16*>(a.shadow)[i] = __float2bfloat16_rn(pv);
    }
  }
}

// Zeros for several buffers in one launch (13 buckets of 553 MB together: 112 us as memsets, 78 so; one buffer alone is a memset, which
// is as fast from 40 MB on and 1 us faster below).
constexpr int kFillVecs = 4;
constexpr int kFillTile = kThreads * 4 * kFillVecs;
constexpr int kFillSegments = 40;
struct FillTable {
  FillSegment seg[kFillSegments];
  int64_t first_tile[kFillSegments + 1];
};
__global__ void __launch_bounds__(kThreads) fill_zero_kernel(const __grid_constant__ FillTable table) {
  wait_for_predecessor();
  int k = 0;
  while ((int64_t)blockIdx.x >= table.first_tile[k + 1]) ++k;
  float* p = table.seg[k].p;
  const int64_t base = ((int64_t)blockIdx.x - table.first_tile[k]) * kFillTile, end = min(base + kFillTile, table.seg[k].n);
  if (end - base == kFillTile && reinterpret_cast<uintptr_t>(p) % 16 == 0) {
#pragma unroll
    for (int u = 0; u < kFillVecs; ++u) reinterpret_cast<float4*>(p + base)[u * kThreads + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    for (int64_t i = base + threadIdx.x; i < end; i += kThreads) p[i] = 0.f;
  }
}

}  // namespace

void fill_zero(const FillSegment* segs, int n, cudaStream_t s) {
  for (int at = 0; at < n; at += kFillSegments) {
    FillTable t;
    const int count = std::min(kFillSegments, n - at);
    t.first_tile[0] = 0;
    for (int k = 0; k < count; ++k) {
      t.seg[k] = segs[at + k];
      t.first_tile[k + 1] = t.first_tile[k] + (segs[at + k].n + kFillTile - 1) / kFillTile;
    }
    if (count == 1)
      BAGUA_CUDA_CHECK(cudaMemsetAsync(segs[at].p, 0, (size_t)segs[at].n * sizeof(float), s));
    else if (t.first_tile[count] > 0)
      launch_overlapped(fill_zero_kernel, dim3((unsigned)t.first_tile[count]), dim3(kThreads), s, t);
  }
}
void divide_inplace(void* x, DType dt, int64_t n, float d, cudaStream_t s) {
  dispatch_ew(x, nullptr, dt, n, OpDiv{d}, s);
}
void add_inplace(void* x, const void* y, DType dt, int64_t n, cudaStream_t s) { dispatch_ew(x, y, dt, n, OpAdd{}, s); }
void subtract_inplace(void* x, const void* y, DType dt, int64_t n, cudaStream_t s) {
  dispatch_ew(x, y, dt, n, OpSub{}, s);
}
void addmul_inplace(void* x, const void* y, float f, DType dt, int64_t n, cudaStream_t s) {
  dispatch_ew(x, y, dt, n, OpAddMul{f}, s);
}
void average_inplace(void* x, const void* y, DType dt, int64_t n, cudaStream_t s) {
  dispatch_ew(x, y, dt, n, OpAvg{}, s);
}
void async_model_average(float* t, const float* r, const float* cp, float nranks, int64_t n, cudaStream_t s) {
  const bool vec = ((uintptr_t)t % 16 == 0) && ((uintptr_t)r % 16 == 0) && ((uintptr_t)cp % 16 == 0);
  async_avg_kernel<<<grid_for(vec ? n / 4 + 1 : n), kThreads, 0, s>>>(t, r, cp, nranks, n, vec);
  BAGUA_CUDA_CHECK(cudaGetLastError());
}
void accumulate_bf16(float* x, const void* y, int64_t n, cudaStream_t s) {
  const bool vec = ((uintptr_t)x % 16 == 0) && ((uintptr_t)y % 8 == 0);
  launch_overlapped(accumulate_bf16_kernel, dim3(grid_for(vec ? n / 4 + 1 : n)), dim3(kThreads), s, x,
                    (const __nv_bfloat16*)y, (float*)nullptr, (const __nv_bfloat16*)nullptr, n, vec);
}
void accumulate_bf16_pair(float* x0, const void* y0, float* x1, const void* y1, int64_t n, cudaStream_t s) {
  const bool vec = (((uintptr_t)x0 | (uintptr_t)x1) % 16 == 0) && (((uintptr_t)y0 | (uintptr_t)y1) % 8 == 0);
  launch_overlapped(accumulate_bf16_kernel, dim3(grid_for(vec ? n / 4 + 1 : n), 2), dim3(kThreads), s, x0,
                    (const __nv_bfloat16*)y0, x1, (const __nv_bfloat16*)y1, n, vec);
}
void cast_bf16(const CastSegment* segs, int n, cudaStream_t s) {
  for (int at = 0; at < n; at += kCastSegments) {
    CastTable t;
    t.n = std::min(kCastSegments, n - at);
    t.first_tile[0] = 0;
    for (int k = 0; k < t.n; ++k) {
      t.seg[k] = segs[at + k];
      t.first_tile[k + 1] = t.first_tile[k] + (segs[at + k].n + kCastTile - 1) / kCastTile;
    }
    if (t.first_tile[t.n] == 0) continue;
    launch_overlapped(cast_bf16_kernel, dim3((unsigned)t.first_tile[t.n]), dim3(kThreads), s, t);
  }
}
void copy_bytes(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  BAGUA_CUDA_CHECK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s));
}
void reduce_chunk_inplace(void* x, DType dt, int64_t chunk, int n_chunks, int target, bool average, cudaStream_t s) {
  switch (dt) {
    case DType::F32: launch_reduce_chunk<float>(x, chunk, n_chunks, target, average, s); return;
    case DType::F16: launch_reduce_chunk<__half>(x, chunk, n_chunks, target, average, s); return;
    case DType::BF16: launch_reduce_chunk<__nv_bfloat16>(x, chunk, n_chunks, target, average, s); return;
    default: throw BaguaError(ErrorKind::Tensor, std::string("reduce_chunk: unsupported dtype ") + dtype_name(dt));
  }
}
int sgd_steps(const SgdSegment* segs, int n, cudaStream_t s) {
  int launches = 0;
  for (int at = 0; at < n; at += kSgdSegments) {
    SgdTable t;
    t.n = std::min(kSgdSegments, n - at);
    t.first_tile[0] = 0;
    for (int k = 0; k < t.n; ++k) {
      SgdSegment& a = t.seg[k];
      a = segs[at + k];
      a.vec = ((uintptr_t)a.p % 16 == 0) && ((uintptr_t)a.g % 16 == 0) && ((uintptr_t)a.m % 16 == 0) &&
              ((uintptr_t)a.shadow % 8 == 0);
      t.first_tile[k + 1] = t.first_tile[k] + (a.n + kSgdTile - 1) / kSgdTile;
    }
    if (t.first_tile[t.n] == 0) continue;
    launch_overlapped(sgd_kernel, dim3((unsigned)t.first_tile[t.n]), dim3(kThreads), s, t);
    ++launches;
  }
  return launches;
}
void sgd_momentum_flat_shadow(float* p, const float* g, float* buf, void* shadow, int64_t n, float lr, float momentum,
                              float dampening, float wd, bool nesterov, bool first_step, cudaStream_t s) {
  const SgdSegment a{p, g, buf, shadow, n, lr, momentum, dampening, wd, nesterov, first_step, false};
  sgd_steps(&a, 1, s);
}

}  // namespace cuda
}  // namespace kernels
}  // namespace bagua
