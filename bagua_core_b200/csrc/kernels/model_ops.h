// Fused element-wise kernels for the benchmark models' convolution blocks (sm_100a).
//
// A VGG-style block is convolution → bias → ReLU.  The framework runs the bias/ReLU part as
// separate passes over the activation (forward: add, clamp; backward: ReLU mask, then a
// column reduction for the bias gradient, which alone took 12 % of a VGG-16 step on a B200).
// These kernels do each direction in one pass over a channels-last activation viewed as a
// row-major [rows = N·H·W, C] matrix of bf16:
//   forward   y = max(z + bias, 0), in place on the convolution's output;
//   backward  dz = dy · [y > 0] and db[c] = Σ_rows dz[row, c] (fp32 accumulation, fixed
//             summation order, no atomics), from one read of dy and y.
// The pooling layers between the blocks get the same treatment (see below).
// No counterpart in the reference, which has no model code.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>

namespace bagua {
namespace model_ops {

// Threads per block of the CUDA kernels.
constexpr int kBlockThreads = 256;

// C must be a multiple of 8, 8 <= C <= 2048, C / 8 a divisor of kBlockThreads; pointers 16-byte aligned.
bool bias_relu_supported(int64_t rows, int C);

// z: [rows, C] bf16 (in place), bias: [C] bf16.  signs (may be null): rows * C / 8 bytes, a bit for every value that is positive.
void bias_relu_inplace_bf16(void* z, const void* bias, int64_t rows, int C, cudaStream_t stream, void* signs = nullptr);

// Bytes of scratch (per-block partial sums) the backward needs for this shape.
size_t bias_relu_backward_scratch_bytes(int64_t rows, int C);

// dy, y, dz: [rows, C] bf16 (dz may alias dy); db: [C] fp32, written or added to; scratch as sized above.  With the forward's
// `signs` y is not read (the seven un-pooled blocks of VGG-16 at batch 32, us in all: backward 128.6 from y, 90.4 from the signs, forward
// 142.0 without and 147.9 with them).
void bias_relu_backward_bf16(const void* dy, const void* y, void* dz, float* db, int64_t rows, int C, void* scratch,
                             cudaStream_t stream, bool accumulate = false, const void* signs = nullptr);

// Backward of relu(conv3x3(x) + bias), stride and padding 1, where the gradient of x is not wanted (a network's first
// layer): with dz = dy where y > 0, dw [C, 3, 3, Ci] = sum over pixels of dz and the pixel's patch of x, db [C] = sum of
// dz, both fp32, written or added to (db may be null); dz itself is not written.  x [N, H, W, Ci], dy and y
// [N, H, W, C], bf16 and channels-last; dy and y 16-byte aligned.  More than 3 input channels (patches beyond 32
// values) are the library's.
inline bool first_conv_backward_supported(int64_t N, int64_t H, int64_t W, int64_t C, int64_t Ci) {
  return N > 0 && H > 0 && W > 0 && N * H * W < (1ll << 30) && C >= 64 && C % 64 == 0 && C <= 4096 && Ci >= 1 && Ci <= 3;
}
size_t first_conv_backward_scratch_bytes(int64_t rows, int C, int Ci);
void first_conv_backward(const void* dy, const void* y, const void* x, float* dw, bool add_w, float* db, bool add_b, int64_t N,
                         int64_t H, int64_t W, int C, int Ci, void* scratch, cudaStream_t s);

// dw[co, r, s, ci] = sum over pixels of dz and x shifted by (r - 1, s - 1): the weight gradient of a 3 x 3 convolution with stride
// and padding 1, summed in fp32 and rounded to bf16.  dz [N, H, W, Co], x [N, H, W, Ci], bf16, channels-last, 16-byte aligned;
// `strides` of dw by co, r, s, ci in elements.  Channel counts are multiples of 64.
bool conv_wgrad_supported(int64_t N, int64_t H, int64_t W, int64_t Co, int64_t Ci);
bool conv_wgrad_preferred(int64_t N, int64_t H, int64_t W, int64_t Co, int64_t Ci);  // supported, and faster than the library's
size_t conv_wgrad_scratch_bytes(int64_t N, int64_t H, int64_t W, int64_t Co, int64_t Ci);
void conv_wgrad(const void* dz, const void* x, void* dw, const int64_t (&strides)[4], int64_t N, int64_t H, int64_t W, int64_t Co,
                int64_t Ci, void* scratch, cudaStream_t stream);

// out[c] (+)= sum over rows of x [rows, C] in bf16, accumulated in fp32 in a fixed order: the bias gradient of a
// linear layer.  C a multiple of 8, x 16-byte aligned.  (3072 x 1024: 8 us; the library's reduction 13 us.)
inline bool column_sum_supported(int64_t rows, int C) { return rows > 0 && C >= 8 && C % 8 == 0; }
size_t column_sum_scratch_bytes(int64_t rows, int C);
void column_sum_bf16(const void* x, float* out, int64_t rows, int C, void* scratch, cudaStream_t stream, bool accumulate);

// ---- 2x2 / stride-2 max pooling on channels-last bf16 activations ---------------------
// x: [N, H, W, C] (H, W even, C a multiple of 8), y: [N, H/2, W/2, C].  The forward stores no
// index tensor; the backward recomputes each window's arg-max from x (first maximum in
// (h, w) scan order, like the framework's kernel) and writes every element of dx exactly
// once, so dx needs no zero-fill and no atomics.
bool maxpool2x2_supported(int64_t N, int64_t H, int64_t W, int C);
void maxpool2x2_forward_bf16(const void* x, void* y, int64_t N, int64_t H, int64_t W, int C, cudaStream_t stream);
void maxpool2x2_backward_bf16(const void* x, const void* dy, void* dx, int64_t N, int64_t H, int64_t W, int C,
                              cudaStream_t stream);

// ---- bias + ReLU followed by 2x2 pooling, as one forward and one backward pass ------------
// y: [N, H, W, C] convolution output, overwritten with max(y + bias, 0); p: [N, H/2, W/2, C].
// Needs both bias_relu_supported(N*H*W, C) and maxpool2x2_supported(N, H, W, C).
void bias_relu_pool_bf16(void* y, void* p, const void* bias, int64_t N, int64_t H, int64_t W, int C, cudaStream_t stream);
// The same p from z: [N, H, W, C] convolution output that is left as it is.  codes (may be null): N * (H/2) * (W/2) * C / 8 words,
// which position of its window every pooled value came from (model_ops_bodies.cuh).
void bias_relu_pool_only_bf16(const void* z, void* p, const void* bias, int64_t N, int64_t H, int64_t W, int C,
                              cudaStream_t stream, void* codes = nullptr);
// Without codes; blocks train through the codes, this is what they are compared with.
// dp: [N, H/2, W/2, C]; y as written by the in-place forward and bias null, or y = z and its bias;
// dz: [N, H, W, C] (every element written); db: [C] fp32; scratch of
// bias_relu_backward_scratch_bytes(N*(H/2)*(W/2), C) bytes.
void bias_relu_pool_backward_bf16(const void* dp, const void* y, const void* bias, void* dz, float* db, int64_t N,
                                  int64_t H, int64_t W, int C, void* scratch, cudaStream_t stream,
                                  bool accumulate = false);

// The same from the forward's codes.
void bias_relu_pool_backward_codes_bf16(const void* dp, const void* codes, void* dz, float* db, int64_t N, int64_t H, int64_t W, int C,
                                        void* scratch, cudaStream_t stream, bool accumulate = false);

// ---- host restatements (model_ops_cpu.cc): same arguments, host pointers, any C ----------
void bias_relu_inplace_bf16_host(void* z, const void* bias, int64_t rows, int C);
void bias_relu_backward_bf16_host(const void* dy, const void* y, void* dz, float* db, int64_t rows, int C);
void maxpool2x2_forward_bf16_host(const void* x, void* y, int64_t N, int64_t H, int64_t W, int C);
void maxpool2x2_backward_bf16_host(const void* x, const void* dy, void* dx, int64_t N, int64_t H, int64_t W, int C);
void bias_relu_pool_bf16_host(void* y, void* p, const void* bias, int64_t N, int64_t H, int64_t W, int C);
void bias_relu_pool_only_bf16_host(const void* z, void* p, const void* bias, int64_t N, int64_t H, int64_t W, int C);
// y: the activation (the caller makes it from z and the bias where it kept those)
void bias_relu_pool_backward_bf16_host(const void* dp, const void* y, void* dz, float* db, int64_t N, int64_t H,
                                       int64_t W, int C);

}  // namespace model_ops
}  // namespace bagua
