// MinMaxUInt8 compression for sm_100a: per-chunk min/max, quantise, dequantise.
//
// One launch per compress call, whatever the number of chunks.  A chunk belongs to a block, to a cluster of blocks (up to
// 2 MB), or to a set of blocks of a launch that is resident as a whole: each block reads its slice once, they agree on the
// chunk's min and max (through shared memory, or through slots in global memory), and each quantises its slice.  The last 64 KiB that a
// block has read stay in its registers between the two passes, so up to 19 MB (two blocks of 512 threads on each of 148 SMs) the
// input is read once; beyond that chunks are taken a group at a time, a group being what fits L2, and the
// second pass runs backwards over what L2 still holds.
//
// Measured, us, calls back to back, compress / both directions (before clusters, and with the dequantiser's loads behind its table):
// 16 KB of fp32 2.8 / 4.9 (3.0 / 4.8), 1 MB 4.4 / 6.9 (6.2 / 8.7), 10 MB in 8 chunks 7.5 / 11.6 (8.2 / 13.3), 1 M fp16 in 3 odd
// chunks 7.7 / 10.2 (9.9 / 12.9), 411 MB in 8 chunks 112 / 200 (116.3 / 216; 78 / 157 at the copy bandwidth), 206 MB of fp16
// 73.8 / 122.8 (76.6 / 131.6).  Small calls are bound by latency (launch, one read, the exchange); large ones by what lies between the passes: at
// 268 MB memory sees the input and the output once, at half its rate.
//
// The reference issues two CUB DeviceReduce calls per chunk from a host loop
// (bagua-core-internal/kernels/bagua_kernels.cu:312-371,533-560) and quantises one byte per thread
// (455-479).
//
// Numerics are the reference's anchored grid (see MinMaxGrid in kernels.h); the header is stored in
// the tensor dtype and the grid is derived from the stored (rounded) values on both sides.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <map>
#include <mutex>

#include "kernels_impl.h"
#include "launch.cuh"
#include "minmax_device.cuh"
#include "minmax_split.h"

namespace bagua {
namespace kernels {
namespace cuda {

namespace {

using mmdev::from_f;
using mmdev::to_f;
using namespace minmax_split;

// ---- vectors at any alignment --------------------------------------------------------------
// A vector is VE elements (16 bytes of T) and their VE quantised bytes.  Both sides are aligned in
// buffers that were padded for it; elsewhere a chunk's payload and its elements start anywhere.

// VE elements of T from a pointer that is only element-aligned: whole words where it is word-aligned,
// else the words around it shifted by two bytes.
template <bool kAligned, typename T>
__device__ __forceinline__ uint4 load_elems(const T* p) {
  if constexpr (kAligned) return *reinterpret_cast<const uint4*>(p);
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  if ((a & 15u) == 0) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
  if ((a & 3u) == 0) return make_uint4(w[0], w[1], w[2], w[3]);
  // 16-bit elements at an odd element: five words cover the eight elements
  const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
  return make_uint4(__funnelshift_r(w0, w1, 16), __funnelshift_r(w1, w2, 16), __funnelshift_r(w2, w3, 16),
                    __funnelshift_r(w3, w4, 16));
}

// What is used for the last time, or not soon again, leaves L2 first: a second read of the input, and outputs
// larger than L2.
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t policy;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
template <bool kAligned, typename T>
__device__ __forceinline__ uint4 load_elems_last(const T* p, uint64_t policy) {
  if constexpr (!kAligned) return load_elems<kAligned>(p);
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p), "l"(policy));
  return r;
}
__device__ __forceinline__ void store_first(uint32_t* p, uint32_t w, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.u32 [%0], %1, %2;" ::"l"(p), "r"(w), "l"(policy) : "memory");
}
__device__ __forceinline__ void store_first(uint2* p, uint2 w, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.v2.u32 [%0], {%1, %2}, %3;" ::"l"(p), "r"(w.x), "r"(w.y), "l"(policy) : "memory");
}
__device__ __forceinline__ void store_first(uint4* p, uint4 w, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "r"(w.x), "r"(w.y), "r"(w.z),
               "r"(w.w), "l"(policy)
               : "memory");
}

__device__ __forceinline__ void widen(const uint4& r, float (&f)[4], const float*) {
  f[0] = __uint_as_float(r.x);
  f[1] = __uint_as_float(r.y);
  f[2] = __uint_as_float(r.z);
  f[3] = __uint_as_float(r.w);
}
__device__ __forceinline__ void widen(const uint4& r, float (&f)[8], const __half*) {
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 v = __half22float2(h[k]);
    f[2 * k] = v.x;
    f[2 * k + 1] = v.y;
  }
}
__device__ __forceinline__ void widen(const uint4& r, float (&f)[8], const __nv_bfloat16*) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 v = __bfloat1622float2(h[k]);
    f[2 * k] = v.x;
    f[2 * k + 1] = v.y;
  }
}

// The VE bytes at q + VE * vec, q at any address: aligned words and a byte shift.
template <bool kAligned, int VE>
__device__ __forceinline__ typename mmdev::QWord<VE>::type load_bytes(const uint8_t* q, int64_t vec) {
  if constexpr (kAligned) return mmdev::load_qword<VE>(q, vec);
  const uintptr_t a = reinterpret_cast<uintptr_t>(q) + (uintptr_t)(vec * VE);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
  const uint32_t sh = (uint32_t)(a & 3u) * 8;
  // the word behind the last byte is touched only when the bytes reach into it
  if constexpr (VE == 4) {
    const uint32_t w0 = w[0], w1 = sh ? w[1] : 0u;
    return __funnelshift_r(w0, w1, sh);
  } else {
    const uint32_t w0 = w[0], w1 = w[1], w2 = sh ? w[2] : 0u;
    return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
  }
}

// ---- compress ------------------------------------------------------------------------------
constexpr int kThreads = 512;
constexpr int kVecs = 8;                       // vectors a thread keeps between the passes (32 registers)
constexpr int kTile = kThreads * kVecs;        // vectors of a tile: 64 KiB
static_assert(kTileBytes == (int64_t)kTile * 16, "the rules of minmax_split.h assume the kernel's tiles");

// How the blocks of a chunk agree: every block leaves {min, tag} and {max, tag} in a slot of its own, two
// 8-byte words each of which says by its tag that it belongs to this launch, and thread t of every block
// waits for slot t.  No atomics, no fences, nothing to reset: one store and one load across L2, where
// maxima by atomics with an arrival counter took 4 us more with 296 blocks.
// With 148 blocks that is 22 thousand waiting threads on 19 lines of L2 (4.6 us): above kDirect blocks the first
// block collects, and the others wait for its answer (2.3 us; 16 blocks among themselves: 1.5 us).
constexpr int kDirect = 24;

__device__ __forceinline__ void leave_minmax(unsigned long long* slot, float mn, float mx, uint32_t tag) {
  const unsigned long long hi = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(hi | __float_as_uint(mn)),
               "l"(hi | __float_as_uint(mx))
               : "memory");
}
// False when the slot's block did not come in time (it cannot fail to under a cooperative launch).
__device__ __forceinline__ bool wait_minmax(const unsigned long long* slot, float& mn, float& mx, uint32_t tag) {
  for (int spins = 0; spins < (1 << 22); ++spins) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(slot) : "memory");
    if ((uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag) {
      mn = __uint_as_float((uint32_t)a);
      mx = __uint_as_float((uint32_t)b);
      return true;
    }
  }
  return false;
}

// The blocks of a chunk, each with its (mn, mx) in every thread, exchange them through the chunk's slots.  Afterwards
// the chunk's min and max are those over the block's threads.  False in a thread that waited in vain.
__device__ __forceinline__ bool agree(unsigned long long* mine, int part, int per_chunk, uint32_t tag, float& mn, float& mx) {
  const int tid = (int)threadIdx.x;
  if (tid == 0) leave_minmax(mine + 2 * part, mn, mx, tag);
  bool all = true;
  if (per_chunk <= kDirect) {
    if (tid < per_chunk) all = wait_minmax(mine + 2 * tid, mn, mx, tag);
    return all;
  }
  // many blocks: the first one collects and passes the result on
  unsigned long long* result = mine + 2 * per_chunk;
  if (part == 0) {
    if (tid < per_chunk) all = wait_minmax(mine + 2 * tid, mn, mx, tag);
    if (__syncthreads_and(all)) {
      mmdev::block_minmax<kThreads>(mn, mx);
      if (tid == 0) leave_minmax(result, mn, mx, tag);
    }
  } else if (tid == 0) {
    all = wait_minmax(result, mn, mx, tag);
  }
  return all;
}

// Smaller chunks belong to a cluster instead (cluster_blocks()).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The blocks of a cluster, each with its (mn, mx) in every thread, exchange them: afterwards the chunk's are those over the block's
// threads.  The caller waits (cluster_wait) before it leaves, as its neighbours read its memory.
__device__ __forceinline__ void agree_in_cluster(int part, int per_chunk, float& mn, float& mx) {
  __shared__ __align__(8) float2 s_mine;
  const int tid = (int)threadIdx.x;
  if (tid == 0) s_mine = make_float2(mn, mx);
  cluster_arrive();
  cluster_wait();
  if (tid < per_chunk && tid != part) {
    uint32_t there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(&s_mine)), "r"(tid));
    float a, b;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(there) : "memory");
    mn = fminf(mn, a);
    mx = fmaxf(mx, b);
  }
  cluster_arrive();
}

// Running min and max of whole vectors: 16-bit types two values at a time, without widening them.
template <typename T>
struct RunningMinMax;
template <>
struct RunningMinMax<float> {
  float mn = FLT_MAX, mx = -FLT_MAX;
  __device__ __forceinline__ void add(const uint4& r) {
    const float f[4] = {__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mn = fminf(mn, f[k]);
      mx = fmaxf(mx, f[k]);
    }
  }
  __device__ __forceinline__ void result(float& a, float& b) const {
    a = mn;
    b = mx;
  }
};
template <typename T2>
struct RunningMinMax2 {
  T2 mn, mx;
  __device__ __forceinline__ void add(const uint4& r) {
    const T2* h = reinterpret_cast<const T2*>(&r);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mn = __hmin2(mn, h[k]);
      mx = __hmax2(mx, h[k]);
    }
  }
  __device__ __forceinline__ void result(float& a, float& b) const {
    a = fminf(to_f(mn.x), to_f(mn.y));
    b = fmaxf(to_f(mx.x), to_f(mx.y));
  }
};
template <>
struct RunningMinMax<__half> : RunningMinMax2<__half2> {
  __device__ RunningMinMax() {
    mn = __floats2half2_rn(INFINITY, INFINITY);
    mx = __floats2half2_rn(-INFINITY, -INFINITY);
  }
};
template <>
struct RunningMinMax<__nv_bfloat16> : RunningMinMax2<__nv_bfloat162> {
  __device__ RunningMinMax() {
    mn = __floats2bfloat162_rn(INFINITY, INFINITY);
    mx = __floats2bfloat162_rn(-INFINITY, -INFINITY);
  }
};

// The quantiser of one chunk.  Where every level lies well inside 2^22 (|upper| does, unless the values are
// large against their range), x * scale is rounded to a whole number, to even at ties as rintf does, by
// adding 1.5 * 2^23, and the byte is the difference of two bit patterns: two additions in place of a
// rounding and a conversion that both run at a quarter of the rate.
struct Quantiser {
  static constexpr float kShift = 12582912.f;
  mmdev::Grid g;
  float mn, mx;  // the range it was made from, where that is needed later
  float lo, hi;  // lower and upper, shifted
  bool shifted;
  __device__ __forceinline__ explicit Quantiser(const mmdev::Grid& grid) : g(grid) {
    shifted = fabsf(g.upper) < 4194304.f - 1024.f;
    lo = g.lower + kShift;
    hi = g.upper + kShift;
  }
  __device__ __forceinline__ uint32_t bits(float x) const {
    const float t = fmaxf(fminf(__fadd_rn(__fmul_rn(x, g.scale), kShift), hi), lo);
    return __float_as_uint(t) - __float_as_uint(lo);  // 0..255
  }
  __device__ __forceinline__ uint32_t pack4(const float* f) const {
    if (shifted) return bits(f[0]) | (bits(f[1]) << 8) | (bits(f[2]) << 16) | (bits(f[3]) << 24);
    return mmdev::pack_q4(f, g);
  }
  __device__ __forceinline__ uint32_t pack(const float (&f)[4]) const { return pack4(f); }
  __device__ __forceinline__ uint2 pack(const float (&f)[8]) const { return make_uint2(pack4(f), pack4(f + 4)); }
};

// One tile of vectors in the registers of the block: kVecs per thread, kThreads apart.
template <typename T, bool kAligned>
struct Tile {
  static constexpr int VE = mmdev::Vec16<T>::VE;
  uint4 raw[kVecs];

  // [p, p + n * VE), n <= kTile
  __device__ __forceinline__ void load(const T* p, int n) {
    const int tid = (int)threadIdx.x;
    if (n == kTile) {
#pragma unroll
      for (int u = 0; u < kVecs; ++u) raw[u] = load_elems<kAligned>(p + (tid + u * kThreads) * VE);
    } else {
#pragma unroll
      for (int u = 0; u < kVecs; ++u)
        if (tid + u * kThreads < n) raw[u] = load_elems<kAligned>(p + (tid + u * kThreads) * VE);
    }
  }
  // `real`: elements from the tile's first on that count (padding does not)
  __device__ __forceinline__ void minmax_all(int n, int64_t real, RunningMinMax<T>& run, float& mn, float& mx) const {
    const int tid = (int)threadIdx.x;
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      const int v = tid + u * kThreads;
      if (v >= n) continue;
      if (real >= (int64_t)n * VE) {
        run.add(raw[u]);
      } else {
        float f[VE];
        widen(raw[u], f, (const T*)nullptr);
#pragma unroll
        for (int k = 0; k < VE; ++k) {
          if ((int64_t)v * VE + k < real) {
            mn = fminf(mn, f[k]);
            mx = fmaxf(mx, f[k]);
          }
        }
      }
    }
  }
  __device__ __forceinline__ void quantise(int u, uint8_t* q, const Quantiser& g) const {
    float f[VE];
    widen(raw[u], f, (const T*)nullptr);
    mmdev::store_qword(q, (int)threadIdx.x + u * kThreads, g.pack(f));
  }
  __device__ __forceinline__ void quantise_out(int u, uint8_t* q, const Quantiser& g, uint64_t policy) const {
    float f[VE];
    widen(raw[u], f, (const T*)nullptr);
    store_first(reinterpret_cast<typename mmdev::QWord<VE>::type*>(q) + (int)threadIdx.x + u * kThreads, g.pack(f), policy);
  }
  __device__ __forceinline__ void quantise_all(uint8_t* q, int n, const Quantiser& g) const {
#pragma unroll
    for (int u = 0; u < kVecs; ++u)
      if ((int)threadIdx.x + u * kThreads < n) quantise(u, q, g);
  }
};

template <typename T, bool kAligned, bool kCluster>
__global__ void __launch_bounds__(kThreads, kBlocksPerSM)
    compress_kernel(const T* __restrict__ in, int64_t num_real, int64_t chunk, int first_chunk, int count, int sets,
                    int per_group, int per_chunk, uint8_t* __restrict__ out, size_t chunk_offset, unsigned long long* slots, uint32_t tag) {
  constexpr int VE = mmdev::Vec16<T>::VE;
  const int tid = (int)threadIdx.x;
  const int slot = (int)blockIdx.x / per_chunk, part = (int)blockIdx.x % per_chunk;
  let_successor_start();
  wait_for_predecessor();
  for (int ci = slot; ci < count; ci += sets * per_group) {
    if (sets > 1 && ci >= per_group) {
      // after the same block of the other set has read its slice of the group in front: the sets stay out of step
      if (tid == 0) {
        float unused_mn, unused_mx;
        wait_minmax(slots + ((size_t)(ci - per_group) * (per_chunk + 1) + part) * 2, unused_mn, unused_mx, tag);
      }
      __syncthreads();
    }
    const int c = first_chunk + ci;
    const T* p = in + (int64_t)c * chunk;
    uint8_t* base = out + (size_t)c * chunk_offset;
    uint8_t* q = base + kCompressHeaderBytes;
    int64_t real = num_real - (int64_t)c * chunk;
    real = real < 0 ? 0 : (real > chunk ? chunk : real);
    // elements in front of the first vector (whose bytes start a word), whole vectors, elements behind the last
    const int64_t head = kAligned ? 0 : min(chunk, (int64_t)((0 - reinterpret_cast<uintptr_t>(q)) & (uintptr_t)(VE - 1)));
    const int64_t nvec = (chunk - head) / VE;
    const int64_t tail = head + nvec * VE;
    const int64_t per = ((nvec + per_chunk - 1) / per_chunk + 31) & ~(int64_t)31;  // slices start on 512 bytes
    // Blocks of several tiles take every per_chunk-th of the chunk's, and the last block what is left: together they pass over memory as
    // one front (411 MB in 8 chunks 115.7 us in slices, 112.0 so; half as much fp16 76.6, 73.8; but unaligned 103 MB in 2 chunks 60.1, 63.3).
    // Blocks of fewer have a slice each.
    const bool front = kAligned && real == chunk && nvec >= 2 * (int64_t)kTile * per_chunk;
    const int64_t whole = nvec / kTile;
    const int64_t lo = front ? whole * kTile : min((int64_t)part * per, nvec);
    const int64_t n = front ? (part == per_chunk - 1 ? nvec - lo : 0) : min(lo + per, nvec) - lo;
    const T* pv = p + head + lo * VE;
    uint8_t* qv = q + head + lo * VE;
    // first what is not a whole tile of real elements, then `full` whole tiles; the last tile stays in registers
    const int64_t full = front ? (whole - part + per_chunk - 1) / per_chunk : real == chunk ? n / kTile : 0;
    const int64_t rest = front ? n : n - full * kTile;
    const int64_t step = (int64_t)kTile * VE * (front ? per_chunk : 1);  // from one whole tile to the next
    const T* pf = front ? p + head + (int64_t)part * kTile * VE : pv + rest * VE;
    uint8_t* qf = front ? q + head + (int64_t)part * kTile * VE : qv + rest * VE;

    // pass 1
    float mn = FLT_MAX, mx = -FLT_MAX;
    RunningMinMax<T> run;
    Tile<T, kAligned> tile;
    for (int64_t v = 0; v < rest; v += kTile) {
      const int m = (int)min((int64_t)kTile, rest - v);
      tile.load(pv + v * VE, m);
      tile.minmax_all(m, real - head - (lo + v) * VE, run, mn, mx);
    }
    if (full > 0) {
      tile.load(pf, kTile);
      const T* next = pf + step;
      for (int64_t t = 1; t < full; ++t, next += step) {
        // a vector's successor is requested as soon as its registers are free: seven stay in flight
#pragma unroll
        for (int u = 0; u < kVecs; ++u) {
          run.add(tile.raw[u]);
          tile.raw[u] = load_elems<kAligned>(next + (tid + u * kThreads) * VE);
        }
      }
#pragma unroll
      for (int u = 0; u < kVecs; ++u) run.add(tile.raw[u]);
    }
    {
      float a, b;
      run.result(a, b);
      mn = fminf(mn, a);
      mx = fmaxf(mx, b);
    }
    if constexpr (!kAligned) {
      if (part == 0 && tid < head && tid < real) {
        const float f = to_f(p[tid]);
        mn = fminf(mn, f);
        mx = fmaxf(mx, f);
      }
      if (part == per_chunk - 1 && tail + tid < chunk && tail + tid < real) {
        const float f = to_f(p[tail + tid]);
        mn = fminf(mn, f);
        mx = fmaxf(mx, f);
      }
    }
    mmdev::block_minmax<kThreads>(mn, mx);
    if constexpr (kCluster) {
      agree_in_cluster(part, per_chunk, mn, mx);
      mmdev::block_minmax<kThreads>(mn, mx);
    } else if (per_chunk > 1 || sets > 1) {
      const bool all = agree(slots + (size_t)ci * (per_chunk + 1) * 2, part, per_chunk, tag, mn, mx);
      if (!__syncthreads_and(all)) {  // the answer is the same, only late
        for (int64_t i = tid; i < real; i += kThreads) {
          const float f = to_f(p[i]);
          mn = fminf(mn, f);
          mx = fmaxf(mx, f);
        }
      }
      mmdev::block_minmax<kThreads>(mn, mx);
    }
    if (mn > mx) mn = mx = 0.f;  // chunk without real elements
    if (part == 0 && tid == 0) mmdev::store_header<T>(base, mn, mx);
    // round through the storage dtype so both sides build the same grid
    const Quantiser g(mmdev::make_grid(to_f(from_f<T>(mn)), to_f(from_f<T>(mx))));

    // pass 2: the tile in registers first, then backwards over what L2 still holds
    if (full > 0) {
      const uint64_t policy = evict_first_policy();
      for (int64_t t = full - 1; t > 0; --t) {
        const T* prev = pf + (t - 1) * step;
#pragma unroll
        for (int u = 0; u < kVecs; ++u) {
          if (sets > 1) {
            tile.quantise_out(u, qf + t * step, g, policy);
            tile.raw[u] = load_elems_last<kAligned>(prev + (tid + u * kThreads) * VE, policy);
          } else {
            tile.quantise(u, qf + t * step, g);
            tile.raw[u] = load_elems<kAligned>(prev + (tid + u * kThreads) * VE);
          }
        }
      }
      tile.quantise_all(qf, kTile, g);
    }
    for (int64_t v = (rest - 1) / kTile * kTile; v >= 0 && rest > 0; v -= kTile) {
      const int m = (int)min((int64_t)kTile, rest - v);
      if (full > 0 || v + kTile < rest) tile.load(pv + v * VE, m);
      tile.quantise_all(qv + v * VE, m, g);
    }
    if constexpr (!kAligned) {
      if (part == 0 && tid < head) q[tid] = mmdev::quantise(to_f(p[tid]), g.g);
      if (part == per_chunk - 1 && tail + tid < chunk) q[tail + tid] = mmdev::quantise(to_f(p[tail + tid]), g.g);
    }
    if constexpr (kCluster) {
      cluster_wait();
      break;  // one chunk per cluster
    }
  }
}

// ---- two rounds of quantisation in place -----------------------------------------------------
// What ByteGrad over one rank does to a bucket: quantise, dequantise, and both again on the result.  The second
// round's range is that of the first round's values, which is known from the first range alone (rounding is
// monotonic), so every element goes through one table of 256 values: one read and one write where four kernels
// and a reduction moved 36 bytes per fp32 element (10 MB: 40 us of kernels in 9 launches).
template <typename T>
__device__ __forceinline__ void build_twice_lut(float* lut, const Quantiser& g) {
  const int q = (int)threadIdx.x;
  auto once = [&](int level) { return to_f(from_f<T>(mmdev::dequantise((uint8_t)level, g.g))); };
  const float mn = to_f(from_f<T>(g.mn)), mx = to_f(from_f<T>(g.mx));
  const float mn2 = once((int)mmdev::quantise(mn, g.g)), mx2 = once((int)mmdev::quantise(mx, g.g));
  const mmdev::Grid second = mmdev::make_grid(mn2, mx2);
  if (q < 256) lut[q] = to_f(from_f<T>(mmdev::dequantise(mmdev::quantise(once(q), second), second)));
}

// The buffers of a launch, which share its blocks by their sizes: all read, agree and write at the same time, so that several buffers pay
// for the latencies of one.
struct QuantiseBatch {
  QuantiseItem item[kMaxJoined];
  int end[kMaxJoined];  // blocks up to the buffer's last; its slots, one more than blocks, lie in the same order
  int count;
};

template <typename T>
__global__ void __launch_bounds__(kThreads, kBlocksPerSM)
    quantise_twice_kernel(const __grid_constant__ QuantiseBatch batch, unsigned long long* all_slots, uint32_t tag) {
  constexpr int VE = mmdev::Vec16<T>::VE;
  __shared__ float s_lut[256];
  const int tid = (int)threadIdx.x;
  int k = 0, first = 0;
  while ((int)blockIdx.x >= batch.end[k]) first = batch.end[k++];
  const int part = (int)blockIdx.x - first, parts = batch.end[k] - first;
  unsigned long long* slots = all_slots + 2 * (first + k);
  T* x = (T*)batch.item[k].x;
  const int64_t n = batch.item[k].n;
  wait_for_predecessor();
  const int64_t head = min(n, (int64_t)(((0 - reinterpret_cast<uintptr_t>(x)) & (uintptr_t)15) / sizeof(T)));
  const int64_t nvec = (n - head) / VE, tail = head + nvec * VE;
  const int64_t per = ((nvec + parts - 1) / parts + 31) & ~(int64_t)31;
  const int64_t lo = min((int64_t)part * per, nvec), m = min(lo + per, nvec) - lo;
  T* xv = x + head + lo * VE;
  float mn = FLT_MAX, mx = -FLT_MAX;
  RunningMinMax<T> run;
  Tile<T, true> tile;
  const int64_t tiles = (m + kTile - 1) / kTile;
  for (int64_t t = 0; t < tiles; ++t) {  // the last tile stays in registers
    const int many = (int)min((int64_t)kTile, m - t * kTile);
    tile.load(xv + t * kTile * VE, many);
    tile.minmax_all(many, (int64_t)many * VE, run, mn, mx);
  }
  {
    float a, b;
    run.result(a, b);
    mn = fminf(mn, a);
    mx = fmaxf(mx, b);
  }
  if (part == 0 && tid < head) {
    mn = fminf(mn, to_f(x[tid]));
    mx = fmaxf(mx, to_f(x[tid]));
  }
  if (part == parts - 1 && tail + tid < n) {
    mn = fminf(mn, to_f(x[tail + tid]));
    mx = fmaxf(mx, to_f(x[tail + tid]));
  }
  mmdev::block_minmax<kThreads>(mn, mx);
  if (parts > 1) {
    // a block that gave up could not read the chunk again, others write to it already: it passes NaN on instead
    // (it cannot happen under a cooperative launch)
    if (!__syncthreads_and(agree(slots, part, parts, tag, mn, mx))) mn = mx = nanf("");
    mmdev::block_minmax<kThreads>(mn, mx);
  }
  if (mn > mx) mn = mx = 0.f;
  Quantiser g(mmdev::make_grid(to_f(from_f<T>(mn)), to_f(from_f<T>(mx))));
  g.mn = mn;
  g.mx = mx;
  build_twice_lut<T>(s_lut, g);
  __syncthreads();
  for (int64_t t = tiles - 1; t >= 0; --t) {
    const int many = (int)min((int64_t)kTile, m - t * kTile);
    if (t != tiles - 1) tile.load(xv + t * kTile * VE, many);
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      if (tid + u * kThreads >= many) continue;
      float f[VE];
      widen(tile.raw[u], f, (const T*)nullptr);
      mmdev::lut_word(g.pack(f), f, s_lut);
      mmdev::store_vec(xv + t * kTile * VE, tid + u * kThreads, f);
    }
  }
  if (part == 0 && tid < head) x[tid] = from_f<T>(s_lut[mmdev::quantise(to_f(x[tid]), g.g)]);
  if (part == parts - 1 && tail + tid < n) x[tail + tid] = from_f<T>(s_lut[mmdev::quantise(to_f(x[tail + tid]), g.g)]);
}

// A launch's tag: not that of any of the last 2^32 - 2 launches of this process, of whatever type (they share
// slots), and not what a fresh slot holds.
uint32_t next_tag() {
  static std::atomic<uint32_t> launches{0};
  uint32_t t;
  do t = ++launches;
  while (t == 0);
  return t;
}

// The largest cluster that the stream's context can run: 16 blocks on the whole GPU, 8 in a green context of any size, fewer under other
// limits.  Asked once per stream, by an id that no other stream of the process gets.
int largest_cluster(cudaStream_t s) {
  // (never given back: engine threads may outlive static objects)
  static std::mutex& mu = *new std::mutex;
  static std::map<unsigned long long, int>& known = *new std::map<unsigned long long, int>;
  static thread_local unsigned long long last_id = 0;
  static thread_local int last = -1;
  unsigned long long id = 0;
  const bool has_id = cudaStreamGetId(s, &id) == cudaSuccess;
  if (has_id && last >= 0 && id == last_id) return last;
  if (!has_id) cudaGetLastError();
  std::lock_guard<std::mutex> g(mu);
  int largest = -1;
  if (auto it = known.find(id); has_id && it != known.end()) largest = it->second;
  if (largest < 0) {
    auto* kernel = compress_kernel<float, true, true>;
    BAGUA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (largest = 16; largest > 1; largest /= 2) {
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)largest;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)largest);
      cfg.blockDim = dim3(kThreads);
      cfg.stream = s;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int fit = 0;
      if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0) break;
      cudaGetLastError();
    }
    if (known.size() >= 256) known.clear();
    if (has_id) known[id] = largest;
  }
  if (has_id) {
    last_id = id;
    last = largest;
  }
  return largest;
}

template <typename T>
void compress_t(const void* in, int64_t num_real, int64_t chunk, int n_chunks, uint8_t* out, size_t out_bytes,
                int target, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  const size_t off = out_bytes / (size_t)n_chunks;
  const int first = target >= 0 ? target : 0;
  const int count = target >= 0 ? 1 : n_chunks;
  const bool aligned = ((uintptr_t)in % 16 == 0) && ((uintptr_t)out % 16 == 0) && (chunk % 16 == 0) && (off % 16 == 0);
  const int largest = chunk * (int64_t)sizeof(T) > kTileBytes ? largest_cluster(s) : 0;
  const int blocks = cluster_blocks(chunk * (int64_t)sizeof(T), count, aligned, largest);
  if (blocks == 1) {
    launch_overlapped(aligned ? compress_kernel<T, true, false> : compress_kernel<T, false, false>, dim3(count), dim3(kThreads), s,
                      (const T*)in, num_real, chunk, first, count, 1, count, 1, out, off, (unsigned long long*)nullptr, 0u);
    return;
  }
  if (blocks > 1) {
    auto* kernel = aligned ? compress_kernel<T, true, true> : compress_kernel<T, false, true>;
    static std::atomic<uint64_t> allowed[2] = {};  // by device; set twice does no harm
    int dev = 0;
    BAGUA_CUDA_CHECK(cudaGetDevice(&dev));
    if (!(allowed[aligned].load(std::memory_order_relaxed) >> (dev & 63) & 1)) {
      BAGUA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      allowed[aligned] |= 1ull << (dev & 63);
    }
    launch_clusters(kernel, count, blocks, dim3(kThreads), s, (const T*)in, num_real, chunk, first, count, 1, count, blocks, out, off,
                    (unsigned long long*)nullptr, 0u);
    return;
  }
  const Split d = split_chunks(count, chunk * (int64_t)sizeof(T), aligned, sm_count());
  auto* kernel = aligned ? compress_kernel<T, true, false> : compress_kernel<T, false, false>;
  BAGUA_CHECK(scratch != nullptr && scratch_bytes >= slot_bytes(count, d.per_chunk), MemPool,
              "compress: scratch buffer too small");
  const uint32_t tag = next_tag();
  launch_cooperative(kernel, dim3(d.grid()), dim3(kThreads), s, (const T*)in, num_real, chunk, first, count, d.sets,
                     d.per_group, d.per_chunk, out, off, (unsigned long long*)scratch, tag);
}

// ---- decompress ----------------------------------------------------------------------------
// kDqVecs quantised words per thread are in flight.  kAhead: the loads in front of the table, for blocks of many words (411 MB of
// fp32: 79 us, 95-97 with the loads behind the table of 1184 resident blocks; half as much fp16 47.8, 55).  Where those blocks have few
// words a thread the table comes first: up to four words four at a time (10 MB of fp32: 3.7 us, 4.2-4.6 with eight, of whose places most
// are empty), else eight (34 MB of fp32 7.0 us, 7.4 ahead, 7.7 by four in twice the blocks; 23 MB of unaligned fp16 8.9, 9.5, 8.5).
constexpr int kDqThreads = 256;
constexpr int kDqMany = 8, kDqFew = 4;

template <typename T, bool kAligned, int kDqVecs, bool kAhead>
__global__ void __launch_bounds__(kDqThreads)
    dequantise_kernel(const uint8_t* __restrict__ in, size_t chunk_offset, int64_t chunk, T* __restrict__ out) {
  constexpr int VE = mmdev::Vec16<T>::VE;
  __shared__ float s_lut[256];
  const int tid = (int)threadIdx.x;
  const int64_t c = blockIdx.y;
  const uint8_t* base = in + (size_t)c * chunk_offset;
  const uint8_t* q = base + kCompressHeaderBytes;
  T* o = out + c * chunk;
  const int64_t head =
      kAligned ? 0 : min(chunk, (int64_t)(((0 - reinterpret_cast<uintptr_t>(o)) & (uintptr_t)15) / sizeof(T)));
  const int64_t nvec = (chunk - head) / VE;
  const int64_t tail = head + nvec * VE;
  const int64_t per = ((nvec + gridDim.x - 1) / gridDim.x + 31) & ~(int64_t)31;
  const int64_t lo = min((int64_t)blockIdx.x * per, nvec), hi = min(lo + per, nvec);
  const uint64_t policy = evict_first_policy();
  typename mmdev::QWord<VE>::type w[kDqVecs];
  // all words before the first store: the compiler may not move a load over a store
  auto load = [&](int64_t v0) {
#pragma unroll
    for (int u = 0; u < kDqVecs; ++u)
      if (v0 + u * kDqThreads < hi) w[u] = load_bytes<kAligned, VE>(q + head, v0 + u * kDqThreads);
  };
  let_successor_start();
  wait_for_predecessor();
  if constexpr (kAhead) load(lo + tid);
  float mn, mx;
  mmdev::load_header<T>(base, mn, mx);
  const mmdev::Grid g = mmdev::make_grid(mn, mx);
  mmdev::build_dequant_lut<T>(s_lut, g);
  __syncthreads();
  for (int64_t v0 = lo + tid; v0 < hi;) {
    if constexpr (!kAhead) load(v0);
#pragma unroll
    for (int u = 0; u < kDqVecs; ++u) {
      if (v0 + u * kDqThreads >= hi) continue;
      float f[VE];
      mmdev::lut_word(w[u], f, s_lut);
      uint4 r;
      mmdev::store_vec(reinterpret_cast<T*>(&r), 0, f);
      store_first(reinterpret_cast<uint4*>(o + head) + v0 + u * kDqThreads, r, policy);
    }
    v0 += (int64_t)kDqVecs * kDqThreads;
    if constexpr (kAhead) load(v0);
  }
  if constexpr (!kAligned) {
    if (blockIdx.x == 0 && tid < head) o[tid] = from_f<T>(s_lut[q[tid]]);
    if (blockIdx.x == gridDim.x - 1 && tail + tid < chunk) o[tail + tid] = from_f<T>(s_lut[q[tail + tid]]);
  }
}

// Over one rank this runs beside a backward pass, as a cooperative launch that starts when all its blocks fit.  It takes
// all the blocks it can use all the same: unlike the exchange between ranks (fused_bytegrad.cu, 32 blocks) it waits for no
// peer, and is gone sooner than a smaller launch that occupies fewer SMs for longer.  Training steps with ByteGrad, us, with all
// (160 blocks for 10 MB) / 148 / 64 / 32 / 16: VGG-16, batch 32: 4771 / 4766 / 4756 / 4844 / 5276; 8 layers of BERT-large, 8 x 384
// tokens: 5000 / 5113-5540 / 5041 / 5162 / 5350.
QuantiseBatch quantise_batch(const QuantiseItem* items, int count, int64_t esize) {
  QuantiseBatch b;
  b.count = count;
  const int64_t all = (int64_t)sm_count() * kBlocksPerSM;
  int64_t wanted = 0, parts[kMaxJoined];
  for (int k = 0; k < count; ++k) {
    b.item[k] = items[k];
    wanted += parts[k] = split_chunks(1, items[k].n * esize, true, sm_count()).per_chunk;
  }
  int blocks = 0;
  for (int k = 0; k < count; ++k) {
    // more than there is room for: each buffer's share, rounded so that the sum fits
    if (wanted > all) parts[k] = std::max<int64_t>(1, parts[k] * (all - count) / wanted);
    b.end[k] = blocks += (int)parts[k];
  }
  return b;
}
size_t batch_slot_bytes(const QuantiseBatch& b) {
  const int blocks = b.end[b.count - 1];
  return blocks == b.count ? 0 : (size_t)(blocks + b.count) * kSlotBytes;  // a block alone waits for nobody
}

template <typename T>
void quantise_twice_t(const QuantiseItem* items, int count, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  const QuantiseBatch b = quantise_batch(items, count, (int64_t)sizeof(T));
  const dim3 grid(b.end[b.count - 1]);
  if (batch_slot_bytes(b) == 0) {  // nobody waits for anybody
    launch_overlapped(quantise_twice_kernel<T>, grid, dim3(kThreads), s, b, (unsigned long long*)nullptr, 0u);
    return;
  }
  BAGUA_CHECK(scratch != nullptr && scratch_bytes >= batch_slot_bytes(b), MemPool, "quantise_twice: scratch too small");
  launch_cooperative(quantise_twice_kernel<T>, grid, dim3(kThreads), s, b, (unsigned long long*)scratch, next_tag());
}

template <typename T>
void decompress_t(const uint8_t* in, size_t in_bytes, int64_t chunk, int n_chunks, void* out, cudaStream_t s) {
  const size_t off = in_bytes / (size_t)n_chunks;
  const bool aligned = ((uintptr_t)in % 16 == 0) && ((uintptr_t)out % 16 == 0) && (chunk % 16 == 0) && (off % 16 == 0);
  // a block takes at least two words per thread, up to 8 blocks per SM; where those would have more than kDqMany, as many as that takes
  constexpr int VE = mmdev::Vec16<T>::VE;
  const int64_t words = chunk / VE, cap = std::max<int64_t>(1, (int64_t)sm_count() * 8 / n_chunks);
  const int64_t want = std::max<int64_t>(1, (words + kDqThreads * 2 - 1) / (kDqThreads * 2)), each = kDqThreads * kDqMany;
  const dim3 grid((unsigned)std::min(want, std::max(cap, (words + each - 1) / each)), (unsigned)n_chunks);
  auto* kernel = aligned ? dequantise_kernel<T, true, kDqFew, false> : dequantise_kernel<T, false, kDqFew, false>;
  if (words > cap * each)
    kernel = aligned ? dequantise_kernel<T, true, kDqMany, true> : dequantise_kernel<T, false, kDqMany, true>;
  else if (words > cap * kDqThreads * kDqFew)
    kernel = aligned ? dequantise_kernel<T, true, kDqMany, false> : dequantise_kernel<T, false, kDqMany, false>;
  launch_overlapped(kernel, grid, dim3(kDqThreads), s, in, off, chunk, (T*)out);
}

}  // namespace

size_t compress_scratch_bytes(int n_chunks, int64_t bytes, cudaStream_t s) {
  return bytes <= kTileBytes ? 0 : scratch_bytes(n_chunks, bytes, sm_count(), largest_cluster(s));
}

void compress_minmax_u8(const void* in, DType dt, int64_t num_real, int64_t chunk, int n_chunks, uint8_t* out,
                        size_t out_bytes, int target, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  switch (dt) {
    case DType::F32:
      compress_t<float>(in, num_real, chunk, n_chunks, out, out_bytes, target, scratch, scratch_bytes, s);
      return;
    case DType::F16:
      compress_t<__half>(in, num_real, chunk, n_chunks, out, out_bytes, target, scratch, scratch_bytes, s);
      return;
    case DType::BF16:
      compress_t<__nv_bfloat16>(in, num_real, chunk, n_chunks, out, out_bytes, target, scratch, scratch_bytes, s);
      return;
    default: throw BaguaError(ErrorKind::Tensor, std::string("compress: unsupported dtype ") + dtype_name(dt));
  }
}

size_t quantise_twice_scratch_bytes(const QuantiseItem* items, int count, DType dt) {
  return batch_slot_bytes(quantise_batch(items, count, (int64_t)dtype_bytes(dt)));
}
void quantise_twice_minmax_u8(const QuantiseItem* items, int count, DType dt, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  BAGUA_CHECK(count > 0 && count <= kMaxJoined, Tensor, "quantise_twice: " << count << " buffers");
  switch (dt) {
    case DType::F32: quantise_twice_t<float>(items, count, scratch, scratch_bytes, s); return;
    case DType::F16: quantise_twice_t<__half>(items, count, scratch, scratch_bytes, s); return;
    case DType::BF16: quantise_twice_t<__nv_bfloat16>(items, count, scratch, scratch_bytes, s); return;
    default: throw BaguaError(ErrorKind::Tensor, std::string("compress: unsupported dtype ") + dtype_name(dt));
  }
}

void decompress_minmax_u8(const uint8_t* in, size_t in_bytes, int64_t chunk, int n_chunks, void* out, DType dt,
                          cudaStream_t s) {
  switch (dt) {
    case DType::F32: decompress_t<float>(in, in_bytes, chunk, n_chunks, out, s); return;
    case DType::F16: decompress_t<__half>(in, in_bytes, chunk, n_chunks, out, s); return;
    case DType::BF16: decompress_t<__nv_bfloat16>(in, in_bytes, chunk, n_chunks, out, s); return;
    default: throw BaguaError(ErrorKind::Tensor, std::string("decompress: unsupported dtype ") + dtype_name(dt));
  }
}

}  // namespace cuda
}  // namespace kernels
}  // namespace bagua
