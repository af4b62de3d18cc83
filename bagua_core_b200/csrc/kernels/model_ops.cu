// Fused bias + ReLU (forward, in place) and its backward with the bias-gradient reduction,
// on channels-last bf16 activations viewed as [rows, C]; see model_ops.h.
//
// Both kernels are pure streams over the activation: 16-byte vectors (8 channels), every
// warp reads whole contiguous rows, grids are a small multiple of the 148 SMs and loop with a
// grid stride.  The backward keeps one fp32 accumulator per channel of the thread's vector
// across all rows it visits, folds the block's accumulators through shared memory and writes
// one partial row per block; a second tiny kernel adds the partial rows in block order, so the
// bias gradient is bit-reproducible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../common.h"
#include "model_ops.h"
#include "launch.cuh"
#include "model_ops_bodies.cuh"

namespace bagua {
namespace model_ops {

namespace {

using namespace bodies;
using kernels::launch_overlapped;
using kernels::wait_for_predecessor;

template <bool kSigns>
__global__ void __launch_bounds__(kThreads)
    bias_relu_kernel(uint4* __restrict__ z, const __nv_bfloat16* __restrict__ bias, int64_t nvec, int cgroups,
                     uint8_t* __restrict__ signs) {
  wait_for_predecessor();
  bias_relu_body<kSigns>(z, bias, nvec, cgroups, signs);
}
template <bool kSigns>
__global__ void __launch_bounds__(kThreads)
    bias_relu_backward_kernel(const uint4* dy, const uint4* __restrict__ y, uint4* dz, float* __restrict__ partial,
                              int64_t rows, int cgroups, const uint8_t* __restrict__ signs) {
  __shared__ float s_acc[kThreads * 8];
  wait_for_predecessor();
  bias_relu_backward_body<kSigns>(dy, y, dz, partial, rows, cgroups, s_acc, signs);
}
constexpr int kFoldCols = 32, kFoldRows = 32;
__global__ void __launch_bounds__(kFoldCols * kFoldRows)
    bias_grad_finish_kernel(const float* __restrict__ partial, float* __restrict__ db, int blocks, int C, bool accumulate) {
  __shared__ float s_acc[kFoldCols * kFoldRows];
  wait_for_predecessor();
  bias_grad_finish_body(partial, db, blocks, C, s_acc, accumulate);
}
__global__ void __launch_bounds__(kThreads)
    column_sum_kernel(const uint4* __restrict__ x, float* __restrict__ partial, int64_t rows, int cgroups, bool accumulate) {
  __shared__ float s_acc[kThreads * 8];
  wait_for_predecessor();
  column_sum_body(x, partial, rows, cgroups, s_acc, accumulate);
}
__global__ void __launch_bounds__(kThreads)
    maxpool2x2_forward_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, int64_t nvec_out, int64_t Wo,
                              int64_t W, int cgroups) {
  wait_for_predecessor();
  maxpool2x2_forward_body(x, y, nvec_out, Wo, W, cgroups);
}
__global__ void __launch_bounds__(kThreads)
    maxpool2x2_backward_kernel(const uint4* __restrict__ x, const uint4* __restrict__ dy, uint4* __restrict__ dx,
                               int64_t nvec_out, int64_t Wo, int64_t W, int cgroups) {
  wait_for_predecessor();
  maxpool2x2_backward_body(x, dy, dx, nvec_out, Wo, W, cgroups);
}

__global__ void __launch_bounds__(kThreads)
    bias_relu_pool_kernel(uint4* __restrict__ y, uint4* __restrict__ p, const __nv_bfloat16* __restrict__ bias,
                          int64_t pooled_pixels, int64_t Wo, int64_t W, int cgroups) {
  wait_for_predecessor();
  bias_relu_pool_body(y, p, bias, pooled_pixels, Wo, W, cgroups);
}
template <bool kCodes>
__global__ void __launch_bounds__(kThreads)
    bias_relu_pool_only_kernel(const uint4* __restrict__ z, uint4* __restrict__ p, const __nv_bfloat16* __restrict__ bias,
                               int64_t pooled_pixels, int64_t Wo, int64_t W, int cgroups, uint32_t* __restrict__ codes) {
  wait_for_predecessor();
  bias_relu_pool_only_body<kCodes>(z, p, bias, pooled_pixels, Wo, W, cgroups, codes);
}
__global__ void __launch_bounds__(kThreads)
    bias_relu_pool_backward_codes_kernel(const uint4* __restrict__ dp, const uint32_t* __restrict__ codes, uint4* __restrict__ dz,
                                         float* __restrict__ partial, int64_t pooled_rows, int64_t Wo, int64_t W, int cgroups) {
  __shared__ float s_acc[kThreads * 8];
  wait_for_predecessor();
  bias_relu_pool_backward_codes_body(dp, codes, dz, partial, pooled_rows, Wo, W, cgroups, s_acc);
}
template <bool kFromZ>
__global__ void __launch_bounds__(kThreads)
    bias_relu_pool_backward_kernel(const uint4* __restrict__ dp, const uint4* __restrict__ y, uint4* __restrict__ dz,
                                   float* __restrict__ partial, int64_t pooled_rows, int64_t Wo, int64_t W, int cgroups,
                                   const __nv_bfloat16* __restrict__ bias) {
  __shared__ float s_acc[kThreads * 8];
  wait_for_predecessor();
  bias_relu_pool_backward_body<kFromZ>(dp, y, dz, partial, pooled_rows, Wo, W, cgroups, s_acc, bias);
}

void fold_partials(const float* partial, float* db, int blocks, int C, bool accumulate, cudaStream_t stream) {
  // few partial rows need few threads
  const int rows = blocks >= kFoldRows ? kFoldRows : blocks > 4 ? 8 : 4;
  launch_overlapped(bias_grad_finish_kernel, dim3((C + kFoldCols - 1) / kFoldCols), dim3(kFoldCols, rows), stream, partial, db, blocks, C, accumulate);
}

// A thread per vector and no more: blocks that come and go pass over the memory as one front, where those that stay walk apart
// (forward with pooling, 64 channels at 224 x 224, batch 32: 45.0 us through 1184 blocks, 42.6 so).
int pool_grid(int64_t nvec_out) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((nvec_out + kThreads - 1) / kThreads, 1 << 30));
}

int backward_blocks(int64_t rows, int C) {
  const int rows_per_iter = kThreads / (C / 8);
  const int64_t want = (rows + rows_per_iter - 1) / rows_per_iter;
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, kMaxBlocks));
}

}  // namespace

static_assert(kThreads == kBlockThreads, "bias_relu_supported() assumes the kernels' block size");

void bias_relu_inplace_bf16(void* z, const void* bias, int64_t rows, int C, cudaStream_t stream, void* signs) {
  BAGUA_CHECK(bias_relu_supported(rows, C) && (uintptr_t)z % 16 == 0, Tensor,
              "fused bias+ReLU: unsupported shape [" << rows << ", " << C << "] or unaligned activation");
  const int64_t nvec = rows * (C / 8);
  const int64_t want = (nvec + (int64_t)kThreads * 4 - 1) / ((int64_t)kThreads * 4);
  // four vectors per thread and no more, as in pool_grid() (64 channels at 224 x 224, batch 32: 74.5 us through 1184 blocks, 64.9 so, 86.6
  // with two vectors per thread, to which reading the bias is more)
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, 1 << 30));
  launch_overlapped(signs ? bias_relu_kernel<true> : bias_relu_kernel<false>, dim3(grid), dim3(kThreads), stream, (uint4*)z,
                    (const __nv_bfloat16*)bias, nvec, C / 8, (uint8_t*)signs);
}

size_t bias_relu_backward_scratch_bytes(int64_t rows, int C) {
  if (!bias_relu_supported(rows, C)) return 0;
  return (size_t)backward_blocks(rows, C) * (size_t)C * sizeof(float);
}

void bias_relu_backward_bf16(const void* dy, const void* y, void* dz, float* db, int64_t rows, int C, void* scratch,
                             cudaStream_t stream, bool accumulate, const void* signs) {
  BAGUA_CHECK(bias_relu_supported(rows, C) && (uintptr_t)dy % 16 == 0 && (uintptr_t)y % 16 == 0 &&
                  (uintptr_t)dz % 16 == 0 && scratch != nullptr,
              Tensor, "fused bias+ReLU backward: unsupported shape [" << rows << ", " << C << "] or unaligned buffers");
  const int blocks = backward_blocks(rows, C);
  launch_overlapped(signs ? bias_relu_backward_kernel<true> : bias_relu_backward_kernel<false>, dim3(blocks), dim3(kThreads), stream,
                    (const uint4*)dy, (const uint4*)y, (uint4*)dz, (float*)scratch, rows, C / 8, (const uint8_t*)signs);
  fold_partials((const float*)scratch, db, blocks, C, accumulate, stream);
}

namespace {
// Row slices of a column sum: enough blocks for every SM, at least 32 rows each.
int column_sum_splits(int64_t rows, int C) {
  const int col_blocks = (C / 8 + 31) / 32;
  return (int)std::max<int64_t>(1, std::min<int64_t>(rows / 32, 2 * 148 / col_blocks));
}
}  // namespace

size_t column_sum_scratch_bytes(int64_t rows, int C) {
  const int splits = column_sum_splits(rows, C);
  return splits == 1 ? 0 : (size_t)splits * (size_t)C * sizeof(float);
}

void column_sum_bf16(const void* x, float* out, int64_t rows, int C, void* scratch, cudaStream_t stream, bool accumulate) {
  BAGUA_CHECK(column_sum_supported(rows, C) && (uintptr_t)x % 16 == 0 &&
                  (scratch != nullptr || column_sum_scratch_bytes(rows, C) == 0),
              Tensor,
              "column sum: unsupported shape [" << rows << ", " << C << "] or unaligned buffer");
  const int splits = column_sum_splits(rows, C);
  const bool direct = splits == 1;  // few rows: the one slice's sums are the result
  launch_overlapped(column_sum_kernel, dim3((C / 8 + 31) / 32, splits), dim3(kThreads), stream, (const uint4*)x,
                    direct ? out : (float*)scratch, rows, C / 8, direct && accumulate);
  if (!direct) fold_partials((const float*)scratch, out, splits, C, accumulate, stream);
}

void maxpool2x2_forward_bf16(const void* x, void* y, int64_t N, int64_t H, int64_t W, int C, cudaStream_t stream) {
  BAGUA_CHECK(maxpool2x2_supported(N, H, W, C) && (uintptr_t)x % 16 == 0 && (uintptr_t)y % 16 == 0, Tensor,
              "fused max-pool: unsupported shape [" << N << ", " << H << ", " << W << ", " << C << "] or unaligned buffers");
  const int64_t nvec_out = N * (H / 2) * (W / 2) * (C / 8);
  launch_overlapped(maxpool2x2_forward_kernel, dim3(pool_grid(nvec_out)), dim3(kThreads), stream, (const uint4*)x, (uint4*)y, nvec_out, W / 2, W, C / 8);
}

void maxpool2x2_backward_bf16(const void* x, const void* dy, void* dx, int64_t N, int64_t H, int64_t W, int C,
                              cudaStream_t stream) {
  BAGUA_CHECK(maxpool2x2_supported(N, H, W, C) && (uintptr_t)x % 16 == 0 && (uintptr_t)dy % 16 == 0 &&
                  (uintptr_t)dx % 16 == 0,
              Tensor,
              "fused max-pool backward: unsupported shape [" << N << ", " << H << ", " << W << ", " << C
                                                             << "] or unaligned buffers");
  const int64_t nvec_out = N * (H / 2) * (W / 2) * (C / 8);
  launch_overlapped(maxpool2x2_backward_kernel, dim3(pool_grid(nvec_out)), dim3(kThreads), stream, (const uint4*)x, (const uint4*)dy, (uint4*)dx, nvec_out, W / 2, W, C / 8);
}

void bias_relu_pool_bf16(void* y, void* p, const void* bias, int64_t N, int64_t H, int64_t W, int C, cudaStream_t stream) {
  BAGUA_CHECK(bias_relu_supported(N * H * W, C) && maxpool2x2_supported(N, H, W, C) && (uintptr_t)y % 16 == 0 &&
                  (uintptr_t)p % 16 == 0,
              Tensor,
              "fused bias+ReLU+pool: unsupported shape [" << N << ", " << H << ", " << W << ", " << C
                                                          << "] or unaligned buffers");
  const int64_t pooled_pixels = N * (H / 2) * (W / 2);
  launch_overlapped(bias_relu_pool_kernel, dim3(pool_grid(pooled_pixels * (C / 8))), dim3(kThreads), stream, (uint4*)y, (uint4*)p, (const __nv_bfloat16*)bias, pooled_pixels, W / 2, W, C / 8);
}

void bias_relu_pool_only_bf16(const void* z, void* p, const void* bias, int64_t N, int64_t H, int64_t W, int C,
                              cudaStream_t stream, void* codes) {
  BAGUA_CHECK(bias_relu_supported(N * H * W, C) && maxpool2x2_supported(N, H, W, C) && (uintptr_t)z % 16 == 0 &&
                  (uintptr_t)p % 16 == 0,
              Tensor,
              "fused bias+ReLU+pool: unsupported shape [" << N << ", " << H << ", " << W << ", " << C
                                                          << "] or unaligned buffers");
  const int64_t pooled_pixels = N * (H / 2) * (W / 2);
  launch_overlapped(codes ? bias_relu_pool_only_kernel<true> : bias_relu_pool_only_kernel<false>, dim3(pool_grid(pooled_pixels * (C / 8))),
                    dim3(kThreads), stream, (const uint4*)z, (uint4*)p, (const __nv_bfloat16*)bias, pooled_pixels, W / 2, W, C / 8,
                    (uint32_t*)codes);
}

void bias_relu_pool_backward_bf16(const void* dp, const void* y, const void* bias, void* dz, float* db, int64_t N,
                                  int64_t H, int64_t W, int C, void* scratch, cudaStream_t stream, bool accumulate) {
  BAGUA_CHECK(bias_relu_supported(N * H * W, C) && maxpool2x2_supported(N, H, W, C) && (uintptr_t)dp % 16 == 0 &&
                  (uintptr_t)y % 16 == 0 && (uintptr_t)dz % 16 == 0 && scratch != nullptr,
              Tensor,
              "fused bias+ReLU+pool backward: unsupported shape [" << N << ", " << H << ", " << W << ", " << C
                                                                   << "] or unaligned buffers");
  const int64_t pooled_rows = N * (H / 2) * (W / 2);
  const int blocks = backward_blocks(pooled_rows, C);
  auto* kernel = bias ? bias_relu_pool_backward_kernel<true> : bias_relu_pool_backward_kernel<false>;
  launch_overlapped(kernel, dim3(blocks), dim3(kThreads), stream, (const uint4*)dp, (const uint4*)y, (uint4*)dz, (float*)scratch, pooled_rows, W / 2, W, C / 8, (const __nv_bfloat16*)bias);
  fold_partials((const float*)scratch, db, blocks, C, accumulate, stream);
}

void bias_relu_pool_backward_codes_bf16(const void* dp, const void* codes, void* dz, float* db, int64_t N, int64_t H, int64_t W, int C,
                                        void* scratch, cudaStream_t stream, bool accumulate) {
  BAGUA_CHECK(bias_relu_supported(N * H * W, C) && maxpool2x2_supported(N, H, W, C) && (uintptr_t)dp % 16 == 0 &&
                  (uintptr_t)codes % 4 == 0 && (uintptr_t)dz % 16 == 0 && scratch != nullptr,
              Tensor, "fused bias+ReLU+pool backward: unsupported shape [" << N << ", " << H << ", " << W << ", " << C
                                                                           << "] or unaligned buffers");
  const int64_t pooled_rows = N * (H / 2) * (W / 2);
  const int blocks = backward_blocks(pooled_rows, C);
  launch_overlapped(bias_relu_pool_backward_codes_kernel, dim3(blocks), dim3(kThreads), stream, (const uint4*)dp, (const uint32_t*)codes,
                    (uint4*)dz, (float*)scratch, pooled_rows, W / 2, W, C / 8);
  fold_partials((const float*)scratch, db, blocks, C, accumulate, stream);
}

}  // namespace model_ops
}  // namespace bagua
