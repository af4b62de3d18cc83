// Fused kernels for transformer encoder layers in bf16 with fp32 parameters (sm_100a).
//
// Around its matrix products and attention an encoder layer is a chain of passes over [rows, H] activations
// of a few MB: residual sum, layer normalisation, GELU, and backward their gradients with column sums over all
// rows for the parameters.  As framework calls that is two to four launches and passes per site (sum, cast of
// the affine parameters, normalisation; backward two kernels and an accumulation).  Here each site is one
// kernel per direction, plus the fold of its partial column sums.
// No counterpart in the reference, which has no model code.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>

namespace bagua {
namespace encoder_ops {

// Hidden sizes of the row kernels: one warp per row, 8 columns per lane and step, everything in registers.
inline bool row_supported(int64_t rows, int64_t H) { return rows > 0 && H >= 8 && H % 8 == 0 && H <= 1024; }

// y = layer_norm(x + r) * gamma + beta; x, r (may be null), y in bf16, gamma and beta fp32 (at any 4-byte address).  The sum is
// rounded to bf16 and left in `sum` (null when r is).  Statistics fp32, one per row.
void add_layer_norm_forward(const void* x, const void* r, const float* gamma, const float* beta, float eps, void* sum, void* y,
                            float* mean, float* rstd, int64_t rows, int H, cudaStream_t s);
// ds (bf16) and the parameters' gradients, written or added to.  `sum`: what was normalised.
size_t layer_norm_backward_scratch_bytes(int64_t rows, int H);
void layer_norm_backward(const void* dy, const void* sum, const float* gamma, const float* mean, const float* rstd, void* ds,
                         float* dgamma, float* dbeta, bool add_gamma, bool add_beta, void* scratch, int64_t rows, int H,
                         cudaStream_t s);

// Input of an encoder: y = layer_norm(tok[ids] + pos[position] + typ[0]) in bf16 from fp32 tables, ids [batch, seq].  An id
// outside [0, vocab) gives a row of NaN and no gradient.
void embed_layer_norm_forward(const int64_t* ids, int64_t vocab, const float* tok, const float* pos, const float* typ, const float* gamma,
                              const float* beta, float eps, void* y, float* mean, float* rstd, int64_t batch, int64_t seq, int H,
                              cudaStream_t s);
// Gradients of all five tables ADDED to dtok [V, H], dpos [>= seq, H], dtyp [H], dgamma, dbeta.  ds: fp32 scratch [rows, H].  Rows of one
// token are summed in order up to kMaxOrdered occurrences; beyond that, slices of that length are added atomically.
constexpr int kMaxTokens = 4096, kMaxOrdered = 256;
size_t embed_backward_scratch_bytes(int64_t rows, int H);
void embed_layer_norm_backward(const void* dy, const int64_t* ids, int64_t vocab, const float* tok, const float* pos, const float* typ,
                               const float* gamma, const float* mean, const float* rstd, float* ds, float* dtok, float* dpos,
                               float* dtyp, float* dgamma, float* dbeta, void* scratch, int64_t batch, int64_t seq, int H,
                               cudaStream_t s);

// y = gelu(z) (exact); backward: dz = dy * gelu'(z) and its column sums, one pass.  [rows, C] bf16, C % 8 == 0.
void gelu_forward(const void* z, void* y, int64_t n, cudaStream_t s);
size_t gelu_backward_scratch_bytes(int64_t rows, int C);
void gelu_backward(const void* dy, const void* z, void* dz, float* db, bool accumulate, void* scratch, int64_t rows, int C,
                   cudaStream_t s);

// out [batch, seq, 3, heads, dim] from three gradients [batch, heads, seq, dim] whose last stride is 1; strides in
// elements (batch, head, seq) per tensor; dim a multiple of 8, all addresses and strides of 16 bytes.
struct HeadStrides {
  int64_t batch, head, seq;
};
void merge_heads(const void* const src[3], const HeadStrides stride[3], void* out, int64_t batch, int64_t seq, int heads,
                 int dim, cudaStream_t s);

}  // namespace encoder_ops
}  // namespace bagua
