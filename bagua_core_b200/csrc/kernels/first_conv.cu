// Backward of a network's first convolution block: the gradients of weight and bias straight from the gradient of
// the ReLU's output; see model_ops.h.
//
// Nobody wants the gradient of the network's input, so the convolution's output gradient dz is needed for these two
// sums alone, and is never written.  The weight gradient is the product [C x pixels] [pixels x 9 Ci], the bias gradient
// one more column of it (ones): a block walks tiles of 64 pixels, masks dy with the activation into shared memory,
// gathers the pixels' 3 x 3 patches (at most 27 values and the one, 32 with zeros) next to it, and adds tile by tile
// with m16n8k16 products in fp32 registers.  The two reads of [pixels, C] bound it from below: with 32 columns per 64
// channels the product needs a hundredth of the matrix rate, so mma.sync, which takes its operands from registers,
// is enough and leaves no accumulator to move.  The loads of the next tile are in flight during the products of this
// one; three blocks per SM, because four leave 64 registers per thread and spill.
//
// 32 x 224 x 224, 3 -> 64 channels (411 MB, 63 us at the copy rate): mask and bias sums 96 us, padding of the
// channels and the library's product 165 us, fold, cast, fills and gaps 20 us before; 83 us and 5 us for the fold
// now (98 us with a division per pixel and the bias sums in registers).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../common.h"
#include "launch.cuh"
#include "model_ops.h"

namespace bagua {
namespace model_ops {

namespace {

using kernels::launch_overlapped;
using kernels::sm_count;
using kernels::wait_for_predecessor;

constexpr int kTileThreads = 256;
constexpr int kPixels = 64;    // per tile: four products deep
constexpr int kChannels = 64;  // per block
constexpr int kPatch = 32;
constexpr int kPerSM = 3;
// Row pitches in shared memory: odd numbers of 16 bytes, so that the eight rows of an ldmatrix meet different banks.
constexpr int kDzPitch = kChannels * 2 + 16, kPatchPitch = kPatch * 2 + 16;

__device__ __forceinline__ void load_transposed(uint32_t (&r)[4], const void* shared) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(shared);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void multiply_add(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// dy where y is positive
__device__ __forceinline__ uint32_t masked(uint32_t dy, uint32_t y) {
  return dy & __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&y), __nv_bfloat162{});
}

// Values k0 .. k0 + 7 of a pixel's patch, in the order (row, column, channel), then a one, whose column of the product
// is the bias gradient; zeros beyond the image.
template <int CI>
__device__ __forceinline__ uint4 gather8(const uint16_t* __restrict__ x, unsigned p, unsigned rows, int h, int w, int H, int W,
                                         int k0) {
  uint32_t v[4];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int k = k0 + j, r = k / (3 * CI), s = (k - r * 3 * CI) / CI, ci = k % CI;
    const int hh = h + r - 1, ww = w + s - 1;
    uint32_t e = k == 9 * CI ? 0x3f80u : 0u;
    if (k < 9 * CI && p < rows && hh >= 0 && hh < H && ww >= 0 && ww < W)
      e = x[((int64_t)p + (int64_t)(r - 1) * W + (s - 1)) * CI + ci];
    v[j / 2] = (j & 1) ? v[j / 2] | (e << 16) : e;
  }
  return make_uint4(v[0], v[1], v[2], v[3]);
}

// partial: a row of C * 9 * CI weight sums and C bias sums per blockIdx.x; blockIdx.y takes 64 of the C channels.
template <int CI>
__global__ void __launch_bounds__(kTileThreads, kPerSM)
    first_conv_backward_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ y, const uint16_t* __restrict__ x,
                               float* __restrict__ partial, unsigned rows, int H, int W, int C) {
  __shared__ __align__(16) unsigned char s_dz[kPixels * kDzPitch];
  __shared__ __align__(16) unsigned char s_patch[kPixels * kPatchPitch];
  wait_for_predecessor();
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cg = tid & 7, pr = tid >> 3;           // masking: 8 channels of pixels pr and pr + 32
  const int pp = tid & 63, k0 = (tid >> 6) * 8;    // gathering: 8 values of pixel pp (k0 is the same over a warp)
  const int depth = warp & 3, half = warp >> 2;    // multiplying: 16 pixels, 32 of the 64 channels
  const unsigned tiles = (rows + kPixels - 1) / kPixels;
  const int64_t vecs = C / 8;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;
  const unsigned first = blockIdx.x * kPixels + pp, step = gridDim.x * kPixels;
  int w = (int)(first % (unsigned)W), h = (int)(first / (unsigned)W % (unsigned)H);
  const int step_w = (int)(step % (unsigned)W), step_h = (int)(step / (unsigned)W % (unsigned)H);
  uint4 a[2], b[2], patch;
  auto load = [&](unsigned tile) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned p = tile * kPixels + pr + 32 * i;
      a[i] = b[i] = make_uint4(0, 0, 0, 0);
      if (p < rows) {
        const int64_t v = (int64_t)p * vecs + blockIdx.y * 8 + cg;
        a[i] = dy[v];
        b[i] = y[v];
      }
    }
    const unsigned p = tile * kPixels + pp;
    switch (k0) {  // compile-time positions in the patch
      case 0: patch = gather8<CI>(x, p, rows, h, w, H, W, 0); break;
      case 8: patch = gather8<CI>(x, p, rows, h, w, H, W, 8); break;
      case 16: patch = gather8<CI>(x, p, rows, h, w, H, W, 16); break;
      default: patch = gather8<CI>(x, p, rows, h, w, H, W, 24); break;
    }
    w += step_w;  // the position of the next tile's pixel, without a division
    if (w >= W) {
      w -= W;
      ++h;
    }
    h += step_h;
    if (h >= H) h -= H;
  };

  unsigned tile = blockIdx.x;
  if (tile < tiles) load(tile);
  while (tile < tiles) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      *reinterpret_cast<uint4*>(s_dz + (pr + 32 * i) * kDzPitch + cg * 16) = make_uint4(masked(a[i].x, b[i].x), masked(a[i].y, b[i].y), masked(a[i].z, b[i].z), masked(a[i].w, b[i].w));
    *reinterpret_cast<uint4*>(s_patch + pp * kPatchPitch + k0 * 2) = patch;
    __syncthreads();
    tile += gridDim.x;
    if (tile < tiles) load(tile);
    // both operands lie with the pixels as rows and are turned on the way to the registers
    uint32_t q[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
      load_transposed(q[n], s_patch + (depth * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * kPatchPitch + n * 32 + (lane >> 4) * 16);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      uint32_t f[4];
      load_transposed(f, s_dz + (depth * 16 + (lane & 7) + (lane >> 4) * 8) * kDzPitch + (half * 32 + m * 16 + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        multiply_add(acc[m][2 * n], f, q[n][0], q[n][1]);
        multiply_add(acc[m][2 * n + 1], f, q[n][2], q[n][3]);
      }
    }
    __syncthreads();
  }

  // the four depths of a channel are added in order
  float* s_sum = reinterpret_cast<float*>(s_dz);
  float* row = partial + (size_t)blockIdx.x * C * (9 * CI + 1);
  for (int d = 0; d < 4; ++d) {
    if (depth == d) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float* at = s_sum + (half * 32 + m * 16 + (lane >> 2) + (k >> 1) * 8) * kPatch + n * 8 + (lane & 3) * 2 + (k & 1);
            *at = d == 0 ? acc[m][n][k] : *at + acc[m][n][k];
          }
    }
    __syncthreads();
  }
  for (int i = tid; i < kChannels * 9 * CI; i += kTileThreads)
    row[(size_t)blockIdx.y * kChannels * 9 * CI + i] = s_sum[i / (9 * CI) * kPatch + i % (9 * CI)];
  if (tid < kChannels) row[(size_t)C * 9 * CI + blockIdx.y * kChannels + tid] = s_sum[tid * kPatch + 9 * CI];
}
static_assert(kChannels * kPatch * sizeof(float) <= kPixels * kDzPitch, "the sums meet in the tile's memory");

// Column sums of the partial rows: nw columns to dw, the nb behind them to db (which may be null).  The weight gradient
// is rounded to bf16 on the way, as every other layer's is by the library, which returns it in bf16.
constexpr int kCols = 32, kRows = 32;
__global__ void __launch_bounds__(kCols * kRows)
    first_conv_fold_kernel(const float* __restrict__ partial, int blocks, int nw, int nb, float* __restrict__ dw, bool add_w,
                           float* __restrict__ db, bool add_b) {
  __shared__ float s_acc[kRows][kCols];
  wait_for_predecessor();
  const int c = (int)(blockIdx.x * kCols + threadIdx.x), n = nw + nb;
  float s = 0.f;
  if (c < n) {
#pragma unroll 8
    for (int r = (int)threadIdx.y; r < blocks; r += kRows) s += partial[(size_t)r * n + c];
  }
  s_acc[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || c >= n) return;
  s = 0.f;
#pragma unroll
  for (int r = 0; r < kRows; ++r) s += s_acc[r][threadIdx.x];
  if (c < nw) {
    s = __bfloat162float(__float2bfloat16_rn(s));
    dw[c] = add_w ? dw[c] + s : s;
  } else if (db != nullptr) {
    db[c - nw] = add_b ? db[c - nw] + s : s;
  }
}

int first_conv_blocks(int64_t rows, int C) {
  const int64_t tiles = (rows + kPixels - 1) / kPixels;
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sm_count() * kPerSM / (C / kChannels)));
}

}  // namespace

size_t first_conv_backward_scratch_bytes(int64_t rows, int C, int Ci) {
  return (size_t)first_conv_blocks(rows, C) * C * (9 * Ci + 1) * sizeof(float);
}

void first_conv_backward(const void* dy, const void* y, const void* x, float* dw, bool add_w, float* db, bool add_b, int64_t N,
                         int64_t H, int64_t W, int C, int Ci, void* scratch, cudaStream_t s) {
  const int64_t rows = N * H * W;
  BAGUA_CHECK(first_conv_backward_supported(N, H, W, C, Ci) && (uintptr_t)dy % 16 == 0 && (uintptr_t)y % 16 == 0, Tensor,
              "first convolution's backward: unsupported shape or unaligned buffers");
  auto* kernel = Ci == 1   ? first_conv_backward_kernel<1>
                 : Ci == 2 ? first_conv_backward_kernel<2>
                           : first_conv_backward_kernel<3>;
  const int blocks = first_conv_blocks(rows, C);
  launch_overlapped(kernel, dim3(blocks, C / kChannels), dim3(kTileThreads), s, (const uint4*)dy, (const uint4*)y,
                    (const uint16_t*)x, (float*)scratch, (unsigned)rows, (int)H, (int)W, C);
  const int nw = C * 9 * Ci, n = nw + C;
  launch_overlapped(first_conv_fold_kernel, dim3((n + kCols - 1) / kCols), dim3(kCols, kRows), s, (const float*)scratch, blocks,
                    nw, C, dw, add_w, db, add_b);
}

}  // namespace model_ops
}  // namespace bagua
