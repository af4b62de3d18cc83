// Fused kernels for transformer encoders in bf16 with fp32 parameters (sm_100a).
//
// Around its matrix products, attention and layer normalisations (library kernels) an encoder is a chain of small
// passes: embedding lookups and sums, GELU, the bias gradients, the packing of the attention gradients, a span loss,
// and the dense gradient of the token table.  As framework calls that is two to sixteen launches per site; here it
// is one per direction, plus the fold of partial column sums.  Everything on the way from the input to the loss is
// computed with the roundings of the framework's operations: a bf16 network is chaotic enough that one rounding
// done differently in the first layer moves gradients behind sums over all tokens by their own size.
// No counterpart in the reference, which has no model code.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <cstdint>

namespace bagua {
namespace encoder_ops {

// Throws if a kernel on the current device has met a token id outside its table or a span target outside its sequence since
// the last look.  Such a call goes on with NaN in the index's place; the error comes with the next one whose host side
// looks after the kernel ran, as with any error that a device finds.
void check_indices();

// x = tok[ids] + pos[position] + typ[0] in fp32, ids [batch, seq].  An id outside [0, vocab) gives a row of NaN and no
// gradient.
void embed_sum(const int64_t* ids, int64_t vocab, const float* tok, const float* pos, const float* typ, float* x, int64_t batch,
               int64_t seq, int H, cudaStream_t s);
// The tables' gradients from dx [batch * seq, H], ADDED to dtok [vocab, H], dpos [>= seq, H] and dtyp [H], each of which
// may be null.  Rows of one token are summed in order up to kMaxOrdered occurrences; beyond that, slices of that length are
// added atomically.  Returns the number of kernels launched.
//
// kMaxTokens: every block looks over all ids, so the scatter grows with the square of the tokens and the dense path, which
// also writes the whole table, does not.  Embedding and normalisation in both directions, this / the framework's, us: 30522 rows
// of 1024: 4096 tokens 127 / 452, 8192 281 / 627, 16384 676 / 1022, 32768 1716 / 1660; rows of 256: 104 / 358, 182 / 367,
// 465 / 457, 1383 / 740; 1000 rows of 64: 102 / 350, 140 / 353, 217 / 353, 467 / 465.  The line is the last of these at which
// this path is well ahead at every width.
constexpr int kMaxTokens = 8192, kMaxOrdered = 256;
size_t embed_backward_scratch_bytes(int64_t rows, int H);
int embed_backward(const float* dx, const int64_t* ids, int64_t vocab, float* dtok, float* dpos, float* dtyp, void* scratch,
                   int64_t batch, int64_t seq, int H, cudaStream_t s);

// y = gelu(z) (exact).  Backward of an activation: dz = dy * gelu'(z), or dy where the ReLU's result `z` is positive, and
// its column sums, in one pass.  [rows, C] bf16, C % 8 == 0.
void gelu_forward(const void* z, void* y, int64_t n, cudaStream_t s);
size_t activation_backward_scratch_bytes(int64_t rows, int C);
void activation_backward(bool gelu, const void* dy, const void* z, void* dz, float* db, bool accumulate, void* scratch,
                         int64_t rows, int C, cudaStream_t s);

// loss = (cross_entropy(logits[..., 0], start) + cross_entropy(logits[..., 1], end)) / 2, logits [batch, seq, 2] bf16; stats:
// 2 * batch + 2 floats for the backward.
void span_loss_forward(const void* logits, const int64_t* start, const int64_t* end, float* loss, float* stats, int64_t batch,
                       int64_t seq, cudaStream_t s);
void span_loss_backward(const void* logits, const int64_t* start, const int64_t* end, const float* stats, const float* dloss,
                        void* dlogits, int64_t batch, int64_t seq, cudaStream_t s);

// out [batch, seq, 3, heads, dim] from three gradients [batch, heads, seq, dim] whose last stride is 1; strides in
// elements (batch, head, seq) per tensor; dim a multiple of 8, all addresses and strides of 16 bytes.
struct HeadStrides {
  int64_t batch, head, seq;
};
void merge_heads(const void* const src[3], const HeadStrides stride[3], void* out, int64_t batch, int64_t seq, int heads,
                 int dim, cudaStream_t s);

}  // namespace encoder_ops
}  // namespace bagua
