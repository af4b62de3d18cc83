// Weight gradient of a 3 x 3 convolution (stride and padding 1) on channels-last bf16 activations, on the 5th-generation
// tensor cores; see model_ops.h.
//
// dw[co, r, s, ci] = sum over pixels p of dz[p, co] * x[p + (r - 1, s - 1), ci] is a product whose long dimension (up to 1.6
// million pixels) is the outer one of both operands.  Both therefore go to shared memory as they lie: TMA brings a
// rectangle of pixels, 64 channels (128 bytes) per row in the 128-byte swizzle, with zeros where it reaches over the edge
// of the image, and the product takes both operands "MN-major", eight pixels to a group.  The nine taps are nine views of
// one rectangle: a view that is one pixel or one image row further on starts 128 bytes or one pitch further on, and the
// distance between the 64-channel blocks of an operand (the descriptor's leading offset) may be such a shift as well,
// so that several taps are one instruction.  The two ways of using that:
//
//  * wide (both channel counts multiples of 128): M = 128 input channels; N = 192 = the views {left, here, right} of 64
//    output channels, twice for 128 of them; a block's job is one such tile of one kernel row.
//  * narrow (multiples of 64): M = 128 = two views of the 64 input channels, N = views of the 64 output channels.  With
//    views {here, a row down} of x against {left, here, right} of dz, and {here, right} of x against {here, right} a row
//    down of dz, ten products of which nine are the taps; the tenth is not used.
//
// What bounds it: shared memory, 128 bytes a cycle for the operands (a product of N = 192 takes 96 cycles and reads 10 KB) and
// for what TMA writes: 224 cycles per 16 pixels where the products alone take 192 (wide), 185 for 160 (narrow).
//
// The pixels are dealt to as many blocks per job as there are SMs for; each leaves its sums in fp32 and a second kernel adds
// them in order (no atomics: the result repeats its bits) and rounds the sum to bf16.
//
// One thread issues the loads, one the products, and all read the accumulators (320 or 384 of the 512 columns of
// tensor memory) at the end.  Every wait has a limit; if one ran out, the block's sums are NaN and the next call throws.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "../common.h"
#include "launch.cuh"
#include "model_ops.h"

namespace bagua {
namespace model_ops {

namespace {

using kernels::launch_overlapped;
using kernels::launch_overlapped_shared;
using kernels::let_successor_start;
using kernels::sm_count;
using kernels::wait_for_predecessor;

constexpr int kThreads = 256;
constexpr int kFoldX = 32, kFoldThreads = 256;
constexpr int kStages = 3;
constexpr int kRowBytes = 128;                 // 64 channels of a pixel
constexpr int kShared = 227 * 1024;            // what a block may use
constexpr int kSharedHead = 1024;              // for aligning the stages to the swizzle's period
constexpr int kTmemColumns = 512;
constexpr int kMaxSteps = 32;                  // products of sixteen pixels in a stage

struct Product {
  int a_start, a_step;  // bytes: the view's start in its plane, and from one 64-channel block of the operand to the next
  int b_start, b_step;
  int n, column;
};

// How a call is cut up.
struct Plan {
  bool wide;
  int W, H;
  int bw, bh;              // pixels of a rectangle: a multiple of 8 columns, bw / 8 * bh even
  int tiles_w, tiles_h;    // rectangles of an image
  int tiles;               // of all images
  int a_planes, b_planes;  // 64-channel planes in a stage (the same for both)
  int a_pitch, b_pitch;    // pixels from one image row of a plane to the next
  int a_plane, b_plane;    // bytes, multiples of 1024
  int a_bytes, b_bytes;    // of them, brought by TMA
  int ja, jb, jr;          // jobs by A's channels, B's channels and kernel rows
  int splits;
  int columns;             // of the accumulators
  Product product[2];
  int steps;
  uint4 step[kMaxSteps];   // what a product of sixteen pixels adds to the operands' descriptions

  __host__ __device__ int jobs() const { return ja * jb * jr; }
  __host__ __device__ int stage_bytes() const { return a_planes * a_plane + b_planes * b_plane; }
};

// An operand that lies pixel by pixel in the 128-byte swizzle is described by its address and `step`, the bytes between its
// 64-channel blocks, in the lower word, and by `group`, the bytes between its groups of eight pixels, in the upper.
__host__ __device__ constexpr uint32_t operand_low(uint32_t address, int step) { return (address >> 4) | (uint32_t)(step >> 4) << 16; }
__host__ __device__ constexpr uint32_t operand_high(int group) { return (uint32_t)(group >> 4) | 1u << 14 | 2u << 29; }
__device__ __forceinline__ uint64_t operand(uint32_t low, uint32_t high) { return (uint64_t)high << 32 | low; }

int round_up(int v, int to) { return (v + to - 1) / to * to; }
int ceil_div(int a, int b) { return (a + b - 1) / b; }

// The largest rectangle of which kStages fit in shared memory: whole image rows where they are short enough.
bool cut(Plan& p, int N, int H, int W, int Co, int Ci) {
  p.wide = Co % 128 == 0 && Ci % 128 == 0;
  p.W = W;
  p.H = H;
  // strips of equal width; an odd number of groups in a row takes rows in pairs, for which the widest may be too large
  const int widest = p.wide ? 128 : 64;
  int strips = ceil_div(W, widest);
  if (round_up(ceil_div(W, strips), 8) / 8 % 2 != 0 && round_up(ceil_div(W, strips), 8) > 72) strips = ceil_div(W, 72);
  p.bw = round_up(ceil_div(W, strips), 8);
  p.bh = 0;
  for (int bh = 1; bh <= std::max(2, H); ++bh) {
    if (p.bw / 8 * bh % 2 != 0) continue;
    Plan q = p;
    q.bh = bh;
    q.a_pitch = p.wide ? p.bw : p.bw + 1;
    q.b_pitch = p.bw + 2;
    const int rows = p.wide ? bh : bh + 1;
    q.a_planes = q.b_planes = p.wide ? 2 : 1;
    q.a_bytes = q.a_pitch * rows * kRowBytes;
    q.b_bytes = q.b_pitch * rows * kRowBytes;
    q.a_plane = round_up(q.a_bytes, 1024);
    q.b_plane = round_up(q.b_bytes, 1024);
    if (q.stage_bytes() * kStages > kShared - kSharedHead - 1024 || p.bw / 8 * bh / 2 > kMaxSteps) break;
    // more rows only where they leave no more of the last rectangle empty
    if (p.bh && ceil_div(H, bh) * bh > ceil_div(H, p.bh) * p.bh) continue;
    p = q;
  }
  if (!p.bh) return false;
  p.tiles_w = ceil_div(W, p.bw);
  p.tiles_h = ceil_div(H, p.bh);
  p.tiles = N * p.tiles_w * p.tiles_h;
  if (p.wide) {
    p.ja = Ci / 128;
    p.jb = Co / 128;
    p.jr = 3;
    p.columns = 384;
    for (int k = 0; k < 2; ++k) p.product[k] = Product{0, p.a_plane, k * p.b_plane, kRowBytes, 192, k * 192};
  } else {
    p.ja = Ci / 64;
    p.jb = Co / 64;
    p.jr = 1;
    p.columns = 320;
    p.product[0] = Product{0, p.a_pitch * kRowBytes, 0, kRowBytes, 192, 0};
    p.product[1] = Product{0, kRowBytes, (p.b_pitch + 1) * kRowBytes, kRowBytes, 128, 192};
  }
  p.splits = std::max(1, std::min(p.tiles, sm_count() / p.jobs()));
  // sixteen pixels are two groups of eight, the second of which may begin the next image row
  const int per_row = p.bw / 8;
  p.steps = per_row * p.bh / 2;
  for (int k = 0; k < p.steps; ++k) {
    const int i0 = 2 * k / per_row, j0 = 2 * k % per_row, i1 = (2 * k + 1) / per_row, j1 = (2 * k + 1) % per_row;
    const int a0 = (i0 * p.a_pitch + j0 * 8) * kRowBytes, a1 = (i1 * p.a_pitch + j1 * 8) * kRowBytes;
    const int b0 = (i0 * p.b_pitch + j0 * 8) * kRowBytes, b1 = (i1 * p.b_pitch + j1 * 8) * kRowBytes;
    p.step[k] = make_uint4((uint32_t)a0 >> 4, operand_high(a1 - a0), (uint32_t)b0 >> 4, operand_high(b1 - b0));
  }
  return true;
}

// ---- tensor memory, barriers, copies ---------------------------------------------------------------
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void barrier_init(uint32_t bar, int arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void barrier_expect(uint32_t bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool barrier_passed(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// False when the phase did not end within kWaitNanoseconds (or that many tries).
constexpr uint64_t kWaitNanoseconds = 4000000000ull;
__device__ __forceinline__ uint64_t nanoseconds() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool barrier_wait(uint32_t bar, uint32_t parity) {
  if (barrier_passed(bar, parity)) return true;
  const uint64_t start = nanoseconds();
  for (int tries = 0; tries < (1 << 26); ++tries) {
    if (barrier_passed(bar, parity)) return true;
    if (nanoseconds() - start > kWaitNanoseconds) return false;
  }
  return false;
}
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c, int w, int h, int n) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
      "l"(map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n)
      : "memory");
}
// bf16 operands, both with the pixels as their outer dimension; fp32 sums; M = 128.
__device__ __forceinline__ uint32_t product_kind(int n) {
  return 1u << 4 | 1u << 7 | 1u << 10 | 1u << 15 | 1u << 16 | (uint32_t)(n >> 3) << 17 | (uint32_t)(128 >> 4) << 24;
}
__device__ __forceinline__ void multiply(uint32_t d, uint64_t a, uint64_t b, uint32_t kind, uint32_t add) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a),
               "l"(b), "r"(kind), "r"(add));
}
// One lane of the (whole) warp.
__device__ __forceinline__ bool elected() {
  uint32_t yes;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(yes));
  return yes != 0;
}
// The barrier is arrived at when all products issued so far have been made.
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// (with its wait in one statement: nothing may look at the registers in between)
__device__ __forceinline__ void read_columns(uint32_t address, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
      "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(address)
      : "memory");
}

// A block's rectangles: those of split `split` of its job.
struct Range {
  int lo, hi;
};
__device__ __forceinline__ Range rectangles(const Plan& p, int split) {
  const int per = p.tiles / p.splits, more = p.tiles % p.splits;
  const int lo = split * per + min(split, more);
  return {lo, lo + per + (split < more ? 1 : 0)};
}

// map_a: x, map_b: dz.  partial, by split and job: [columns: view of dz, output channel][128 input channels, or two views of 64].
__global__ void __launch_bounds__(kThreads, 1)
    conv_wgrad_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Plan p,
                      float* __restrict__ partial, unsigned int* status) {
  extern __shared__ unsigned char s_raw[];
  __shared__ __align__(8) uint64_t s_full[kStages], s_empty[kStages], s_done;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_failed;
  const int tid = (int)threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t stages = (shared_address(s_raw) + kSharedHead - 1) & ~(uint32_t)(kSharedHead - 1);
  const int job = (int)blockIdx.x % p.jobs(), split = (int)blockIdx.x / p.jobs();
  const int kr = job % p.jr, jb = job / p.jr % p.jb, ja = job / p.jr / p.jb;
  const Range range = rectangles(p, split);

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      barrier_init(shared_address(&s_full[s]), 1);
      barrier_init(shared_address(&s_empty[s]), 1);
    }
    barrier_init(shared_address(&s_done), 1);
    s_failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Before tensor memory is taken: a predecessor that let this kernel start early may have blocks that have yet to take theirs, and this one
  // waits for them.
  wait_for_predecessor();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(shared_address(&s_tmem)), "r"(kTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;

  if (tid == 0) {  // loads
    const int stage_tx = p.a_planes * p.a_bytes + p.b_planes * p.b_bytes;
    int stage = 0, issued = 0;
    uint32_t parity = 1;  // the first round finds the stages empty
    int tw = range.lo % p.tiles_w, th = range.lo / p.tiles_w % p.tiles_h, n = range.lo / p.tiles_w / p.tiles_h;
    for (int t = range.lo; t < range.hi; ++t) {
      if (!barrier_wait(shared_address(&s_empty[stage]), parity) || s_failed) {
        s_failed = 1;
        break;
      }
      const uint32_t bar = shared_address(&s_full[stage]);
      const uint32_t a = stages + stage * p.stage_bytes(), b = a + p.a_planes * p.a_plane;
      barrier_expect(bar, stage_tx);
      const int w = tw * p.bw, h = th * p.bh;
      if (p.wide) {
        for (int k = 0; k < 2; ++k) {
          load_box(a + k * p.a_plane, &map_a, bar, ja * 128 + k * 64, w, h, n);
          load_box(b + k * p.b_plane, &map_b, bar, jb * 128 + k * 64, w - 1, h + 1 - kr, n);
        }
      } else {
        load_box(a, &map_a, bar, ja * 64, w, h, n);
        load_box(b, &map_b, bar, jb * 64, w - 1, h, n);
      }
      ++issued;
      if (++tw == p.tiles_w) {
        tw = 0;
        if (++th == p.tiles_h) {
          th = 0;
          ++n;
        }
      }
      if (++stage == kStages) {
        stage = 0;
        parity ^= 1;
      }
    }
    if (s_failed)  // no copy may be in flight when the block leaves
      for (int k = max(0, issued - kStages); k < issued; ++k)
        barrier_wait(shared_address(&s_full[k % kStages]), (uint32_t)(k / kStages) & 1);
  } else if (warp == 1) {
    // products: the whole warp walks along, so that the descriptions stay in uniform registers, and one lane issues
    int stage = 0;
    uint32_t parity = 0, add = 0;
    const uint32_t kind0 = product_kind(p.product[0].n), kind1 = product_kind(p.product[1].n);
    const uint32_t d0 = tmem + p.product[0].column, d1 = tmem + p.product[1].column;
    const bool issues = elected();
    for (int t = range.lo; t < range.hi; ++t) {
      if (!__all_sync(0xffffffffu, barrier_wait(shared_address(&s_full[stage]), parity) && !s_failed)) {
        s_failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a = stages + stage * p.stage_bytes(), b = a + p.a_planes * p.a_plane;
      const uint32_t a0 = operand_low(a + p.product[0].a_start, p.product[0].a_step);
      const uint32_t b0 = operand_low(b + p.product[0].b_start, p.product[0].b_step);
      const uint32_t a1 = operand_low(a + p.product[1].a_start, p.product[1].a_step);
      const uint32_t b1 = operand_low(b + p.product[1].b_start, p.product[1].b_step);
      if (issues) {
#pragma unroll 2
        for (int k = 0; k < p.steps; ++k) {
          const uint4 v = p.step[k];
          multiply(d0, operand(a0 + v.x, v.y), operand(b0 + v.z, v.w), kind0, add);
          multiply(d1, operand(a1 + v.x, v.y), operand(b1 + v.z, v.w), kind1, add);
          add = 1;
        }
        commit(shared_address(&s_empty[stage]));
      }
      __syncwarp();
      if (++stage == kStages) {
        stage = 0;
        parity ^= 1;
      }
    }
    if (issues) commit(shared_address(&s_done));
  }
  __syncwarp();
  if (!barrier_wait(shared_address(&s_done), 0)) s_failed = 1;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  let_successor_start();

  // four warps cover the 128 rows; the two halves of the block take every other 32 columns
  const bool failed = s_failed != 0;
  if (failed && tid == 0) {
    *(volatile unsigned int*)status = 1u;
    __threadfence_system();
  }
  float* out = partial + (size_t)blockIdx.x * 128 * p.columns;
  const int row = (warp & 3) * 32 + lane;
  for (int c = (warp >> 2) * 32; c < p.columns; c += 64) {
    uint32_t r[32];
    read_columns(tmem + ((uint32_t)(warp & 3) << 21) + c, r);
    if (failed) {
#pragma unroll
      for (int k = 0; k < 32; ++k) r[k] = 0x7fffffffu;
    }
    // (a thread's own 128 bytes at a time would be 32 lines per instruction: 8 us instead of 2 for the whole block)
#pragma unroll
    for (int k = 0; k < 32; ++k) out[(size_t)(c + k) * 128 + row] = __uint_as_float(r[k]);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
}

// ---- the splits' sums added up ------------------------------------------------------------------------
// A thread of the block's first dimension takes four input channels of one (output channel, tap); the second dimension takes
// the splits in turn, and its sums are added in order.
__global__ void __launch_bounds__(kFoldThreads)
    conv_wgrad_fold_kernel(const float4* __restrict__ partial, const Plan p, int Co, int Ci, __nv_bfloat16* __restrict__ dw,
                           int64_t stride_co, int64_t stride_r, int64_t stride_s, int64_t stride_ci) {
  __shared__ float4 s_sum[kFoldThreads];
  const int per_tap = Ci / 4;
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);  // [co][tap][ci / 4]
  const bool mine = i < Co * 9 * per_tap;
  const int ci = (mine ? i % per_tap : 0) * 4, tap = mine ? i / per_tap % 9 : 0, co = mine ? i / per_tap / 9 : 0;
  const int r = tap / 3, s = tap % 3;
  // (see the top of the file) of dz the column block, of x the row
  int job, block, row;
  if (p.wide) {
    job = ((ci / 128) * p.jb + co / 128) * 3 + r;
    block = co % 128 / 64 * 3 + 2 - s;
    row = ci % 128;
  } else {
    job = (ci / 64) * p.jb + co / 64;
    block = r > 0 ? 2 - s : s == 0 ? 4 : 3;
    row = (r > 0 ? r - 1 : s == 2) * 64 + ci % 64;
  }
  const int64_t at = (int64_t)job * 128 * p.columns + (int64_t)(block * 64 + co % 64) * 128 + row;
  const float4* from = partial + at / 4;
  const int64_t step = (int64_t)p.jobs() * 128 * p.columns / 4;
  wait_for_predecessor();
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  if (mine) {
#pragma unroll 4
    for (int k = (int)threadIdx.y; k < p.splits; k += (int)blockDim.y) {
      const float4 v = __ldcs(from + k * step);
      sum.x += v.x;
      sum.y += v.y;
      sum.z += v.z;
      sum.w += v.w;
    }
  }
  if (blockDim.y > 1) {
    s_sum[threadIdx.y * blockDim.x + threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.y != 0) return;
    for (int k = 1; k < (int)blockDim.y; ++k) {
      const float4 v = s_sum[k * blockDim.x + threadIdx.x];
      sum.x += v.x;
      sum.y += v.y;
      sum.z += v.z;
      sum.w += v.w;
    }
  }
  if (!mine) return;
  const float v[4] = {sum.x, sum.y, sum.z, sum.w};
  __nv_bfloat16* to = dw + co * stride_co + r * stride_r + s * stride_s + ci * stride_ci;
#pragma unroll
  for (int k = 0; k < 4; ++k) to[k * stride_ci] = __float2bfloat16_rn(v[k]);
}

// ---- host -------------------------------------------------------------------------------------------
// One word per device in host memory: a kernel that waited in vain sets it.  Never given back: a captured graph keeps its
// address.
unsigned int* status_word() {
  static std::atomic<unsigned int*> words[64] = {};
  static std::mutex mu;
  int dev = 0;
  BAGUA_CUDA_CHECK(cudaGetDevice(&dev));
  BAGUA_CHECK(dev >= 0 && dev < 64, Tensor, "device index " << dev << " out of range");
  if (unsigned int* w = words[dev].load(std::memory_order_acquire)) return w;
  std::lock_guard<std::mutex> g(mu);
  if (!words[dev].load()) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // nothing is enqueued
    BAGUA_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
    unsigned int* w = nullptr;
    const cudaError_t e = cudaHostAlloc((void**)&w, sizeof(unsigned int), cudaHostAllocMapped);
    BAGUA_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
    BAGUA_CUDA_CHECK(e);
    *w = 0;
    words[dev].store(w, std::memory_order_release);
  }
  return words[dev].load();
}

using EncodeTiled = decltype(&cuTensorMapEncodeTiled);
EncodeTiled encode_tiled() {
  static EncodeTiled f = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult st;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &st) != cudaSuccess ||
        st != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return (EncodeTiled)p;
  }();
  return f;
}

// Rectangles of `w` by `h` pixels and 64 channels of t [N, H, W, C].
CUtensorMap rectangle_map(const void* t, int N, int H, int W, int C, int w, int h) {
  CUtensorMap map;
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
  const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)C * 2 * W, (cuuint64_t)C * 2 * W * H};
  const cuuint32_t box[4] = {64, (cuuint32_t)w, (cuuint32_t)h, 1}, each[4] = {1, 1, 1, 1};
  const CUresult e = encode_tiled()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(t), dims, strides, box, each,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  BAGUA_CHECK(e == CUDA_SUCCESS, Tensor, "convolution weight gradient: tensor map refused (" << (int)e << ")");
  return map;
}

}  // namespace

bool conv_wgrad_supported(int64_t N, int64_t H, int64_t W, int64_t Co, int64_t Ci) {
  if (N < 1 || H < 1 || W < 1 || Co < 64 || Ci < 64 || Co % 64 || Ci % 64 || Co > 4096 || Ci > 4096) return false;
  if (H > (1 << 15) || W > (1 << 15) || N >= (1 << 30) || N * H * W >= (1ll << 30) || !encode_tiled()) return false;
  Plan p;
  return cut(p, (int)N, (int)H, (int)W, (int)Co, (int)Ci);
}

// Two launches and the meeting of the splits take 9 us however little there is to add up, and the sums that the second one
// reads grow with the product of the channel counts; the library's best kernel, which pairs SMs, is the faster one from 512 by 512
// channels on, but for fewer it uses others.  Measured here / by the library, us, by batch (back to back in a graph):
//   64 -> 64 at 224:    1: 20.6/24.9  8: 38.3/63.7  32: 104.6/206.7      at 56:  1: 9.4/10.1  32: 23.9/29.0
//   64 -> 128 at 112:   1: 12.5/19.7  8: 24.6/37.2  32: 53.2/108.9       at 56:  1: 9.6/10.1   2: 10.5/13.7
//   128 -> 128 at 112:  1: 14.4/20.1  8: 29.6/62.1  32: 87.4/125.1       at 28:  4: 11.3/10.2  8: 12.8/16.7
//   128 -> 256 at 56:   1: 12.5/9.7   2: 14.0/24.7  32: 46.7/95.4
//   256 -> 256 at 56:   2: 16.4/16.0  8: 29.0/53.1  32: 82.9/163.5       at 28:  8: 17.0/16.0  12: 19.3/19.9
//   256 -> 512 at 28:  16: 31.1/26.3  24: 40.1/34.9 32: 49.1/56.6        at 56:  4: 29.2/26.3   8: 45.5/56.1
//   512 -> 512 at 28:  32: 89.8/79.9  64: 167.6/151.0                    at 14: 32: 33.1/27.0
// Where rectangles leave much of themselves empty (7 x 7 images: 8 x 8) the library is as fast at any batch.
bool conv_wgrad_preferred(int64_t N, int64_t H, int64_t W, int64_t Co, int64_t Ci) {
  if (!conv_wgrad_supported(N, H, W, Co, Ci) || Co * Ci > (1 << 17) || N * H * W < std::max<int64_t>(6000, Co * Ci * 3 / 16)) return false;
  Plan p;
  cut(p, (int)N, (int)H, (int)W, (int)Co, (int)Ci);
  return (int64_t)p.tiles * p.bw * p.bh * 4 <= N * H * W * 5;
}

size_t conv_wgrad_scratch_bytes(int64_t N, int64_t H, int64_t W, int64_t Co, int64_t Ci) {
  Plan p;
  if (!conv_wgrad_supported(N, H, W, Co, Ci) || !cut(p, (int)N, (int)H, (int)W, (int)Co, (int)Ci)) return 0;
  return (size_t)p.splits * p.jobs() * 128 * p.columns * sizeof(float);
}

void conv_wgrad(const void* dz, const void* x, void* dw, const int64_t (&strides)[4], int64_t N, int64_t H, int64_t W,
                int64_t Co, int64_t Ci, void* scratch, cudaStream_t stream) {
  BAGUA_CHECK(conv_wgrad_supported(N, H, W, Co, Ci) && (uintptr_t)dz % 16 == 0 && (uintptr_t)x % 16 == 0 && scratch != nullptr &&
                  (uintptr_t)scratch % 16 == 0,
              Tensor, "convolution weight gradient: unsupported shape or unaligned buffers");
  unsigned int* status = status_word();
  if (*(volatile unsigned int*)status) {
    *(volatile unsigned int*)status = 0;
    throw BaguaError(ErrorKind::Tensor, "convolution weight gradient: a wait on the device ran out");
  }
  Plan p;
  cut(p, (int)N, (int)H, (int)W, (int)Co, (int)Ci);
  const int rows = p.wide ? p.bh : p.bh + 1;
  const CUtensorMap map_dz = rectangle_map(dz, (int)N, (int)H, (int)W, (int)Co, p.b_pitch, rows);
  const CUtensorMap map_x = rectangle_map(x, (int)N, (int)H, (int)W, (int)Ci, p.a_pitch, rows);
  const size_t shared = (size_t)p.stage_bytes() * kStages + kSharedHead;
  static std::once_flag once[64];
  int dev = 0;
  BAGUA_CUDA_CHECK(cudaGetDevice(&dev));
  std::call_once(once[dev & 63], [] {
    BAGUA_CUDA_CHECK(cudaFuncSetAttribute(conv_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kShared - 1024));
  });
  launch_overlapped_shared(conv_wgrad_kernel, dim3(p.jobs() * p.splits), dim3(kThreads), shared, stream, map_x, map_dz, p,
                           (float*)scratch, status);
  // enough threads for the memory: few results of many splits are shared out
  const int64_t quads = Co * 9 * Ci / 4;
  int sharers = 1;
  while (sharers < kFoldThreads / kFoldX && sharers * 4 <= p.splits && quads * sharers < (int64_t)sm_count() * 1024) sharers *= 2;
  const int across = kFoldThreads / sharers;
  const dim3 grid((unsigned)((quads + across - 1) / across)), block(across, sharers);
  launch_overlapped(conv_wgrad_fold_kernel, grid, block, stream, (const float4*)scratch, p, (int)Co, (int)Ci, (__nv_bfloat16*)dw,
                    strides[0], strides[1], strides[2], strides[3]);
}

}  // namespace model_ops
}  // namespace bagua
