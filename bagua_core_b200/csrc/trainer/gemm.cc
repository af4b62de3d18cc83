#include "gemm.h"

#include <ATen/Context.h>
#include <ATen/cuda/CUDAContext.h>
#include <cublasLt.h>

#include <cstring>
#include <memory>
#include <unordered_map>

#include "../pool/resource_pool.h"

namespace bagua {
namespace trainer {
namespace gemm {

namespace {

// The forward product has the framework's own workspace (1 MB unless CUBLASLT_WORKSPACE_SIZE says otherwise) and counts its
// bias as an operand to be aligned, so that the library picks the algorithm that the framework's layer has: the activations,
// and with them the ReLU masks and everything behind, keep their bits.  (Without a bias the framework goes through another
// of the library's interfaces and may get another algorithm.)  Gradients have no such edges and may use more.
constexpr size_t kGradientWorkspace = 32u << 20;

// How partial sums over parts of k may be added up: torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction.
uint32_t reduction_schemes(at::CuBLASReductionOption option) {
  switch (option) {
    case at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK: return CUBLASLT_REDUCTION_SCHEME_MASK;
    case at::CuBLASReductionOption::DisallowReducedPrecisionAllowSplitK: return CUBLASLT_REDUCTION_SCHEME_COMPUTE_TYPE;
    default: return CUBLASLT_REDUCTION_SCHEME_NONE;
  }
}

constexpr size_t kMaxPlans = 512;  // per thread; a program with more shapes than that starts over

struct Key {
  int kind, device;
  int64_t m, n, k;
  // whether there is a bias or an addition, how the operands are aligned (in powers of two up to 256) and how partial sums
  // may be added
  uint32_t flags;
  bool operator==(const Key& o) const { return std::memcmp(this, &o, sizeof(Key)) == 0; }
};
struct Hash {
  size_t operator()(const Key& k) const {
    uint64_t h = (uint64_t)k.kind * 0x9e3779b97f4a7c15ull + (uint64_t)k.device;
    for (uint64_t v : {(uint64_t)k.m, (uint64_t)k.n, (uint64_t)k.k, (uint64_t)k.flags}) h = (h ^ v) * 0xff51afd7ed558ccdull, h ^= h >> 29;
    return (size_t)h;
  }
};

struct Plan {
  cublasLtMatmulDesc_t desc = nullptr;
  cublasLtMatrixLayout_t a = nullptr, b = nullptr, d = nullptr;
  cublasLtMatmulAlgo_t algo;
  size_t workspace = 0;
  bool usable = false;
  Plan() = default;
  Plan(const Plan&) = delete;
  ~Plan() {
    if (a) cublasLtMatrixLayoutDestroy(a);
    if (b) cublasLtMatrixLayoutDestroy(b);
    if (d) cublasLtMatrixLayoutDestroy(d);
    if (desc) cublasLtMatmulDescDestroy(desc);
  }
};

uint32_t alignment_log(const void* p) {
  uint32_t l = 0;
  while (l < 8 && ((uintptr_t)p & (1u << l)) == 0) ++l;
  return l;
}

// One product in the library's column-major terms: D [rows x cols] = op(A) op(B) (+ D).
struct Problem {
  cublasOperation_t opa, opb;
  int64_t a_rows, a_cols, b_rows, b_cols, d_rows, d_cols;
  bool d_fp32, bias, forward, relu;
};

bool build(Plan& p, cublasLtHandle_t lt, const Problem& q, const void* A, const void* B, const void* D, const void* bias,
           at::CuBLASReductionOption reductions) {
  auto ok = [](cublasStatus_t s) { return s == CUBLAS_STATUS_SUCCESS; };
  if (!ok(cublasLtMatmulDescCreate(&p.desc, CUBLAS_COMPUTE_32F, CUDA_R_32F))) return false;
  auto set = [&](cublasLtMatmulDescAttributes_t at, const void* v, size_t n) {
    return ok(cublasLtMatmulDescSetAttribute(p.desc, at, v, n));
  };
  if (!set(CUBLASLT_MATMUL_DESC_TRANSA, &q.opa, sizeof(q.opa)) || !set(CUBLASLT_MATMUL_DESC_TRANSB, &q.opb, sizeof(q.opb)))
    return false;
  if (q.bias || q.relu) {
    const cublasLtEpilogue_t e = q.bias ? (q.relu ? CUBLASLT_EPILOGUE_RELU_BIAS : CUBLASLT_EPILOGUE_BIAS) : CUBLASLT_EPILOGUE_RELU;
    if (!set(CUBLASLT_MATMUL_DESC_EPILOGUE, &e, sizeof(e))) return false;
  }
  if (q.bias) {
    const cudaDataType_t t = CUDA_R_16BF;
    if (!set(CUBLASLT_MATMUL_DESC_BIAS_DATA_TYPE, &t, sizeof(t)) ||
        !set(CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof(bias)))
      return false;
  }
  const cudaDataType_t dt = q.d_fp32 ? CUDA_R_32F : CUDA_R_16BF;
  if (!ok(cublasLtMatrixLayoutCreate(&p.a, CUDA_R_16BF, (uint64_t)q.a_rows, (uint64_t)q.a_cols, q.a_rows)) ||
      !ok(cublasLtMatrixLayoutCreate(&p.b, CUDA_R_16BF, (uint64_t)q.b_rows, (uint64_t)q.b_cols, q.b_rows)) ||
      !ok(cublasLtMatrixLayoutCreate(&p.d, dt, (uint64_t)q.d_rows, (uint64_t)q.d_cols, q.d_rows)))
    return false;
  cublasLtMatmulPreference_t pref = nullptr;
  if (!ok(cublasLtMatmulPreferenceCreate(&pref))) return false;
  // (the framework's is read from the environment at each call, which takes longer than the rest of a launch)
  p.workspace = q.forward ? at::cuda::getCUDABlasLtWorkspaceSize() : kGradientWorkspace;
  const uint32_t schemes = reduction_schemes(reductions);
  const uint32_t al[4] = {1u << alignment_log(A), 1u << alignment_log(B), 1u << alignment_log(D),
                          1u << alignment_log(q.bias ? bias : D)};
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &p.workspace, sizeof(p.workspace));
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, &al[0], 4);
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES, &al[1], 4);
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES, &al[2], 4);
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES, &al[3], 4);
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_REDUCTION_SCHEME_MASK, &schemes, sizeof(schemes));
  cublasLtMatmulHeuristicResult_t best;
  int found = 0;
  const cublasStatus_t s = cublasLtMatmulAlgoGetHeuristic(lt, p.desc, p.a, p.b, p.d, p.d, pref, 1, &best, &found);
  cublasLtMatmulPreferenceDestroy(pref);
  if (!ok(s) || found < 1) return false;
  p.algo = best.algo;
  return true;
}

bool run(int kind, const Problem& q, int64_t m, int64_t n, int64_t k, const at::Tensor& A, const at::Tensor& B, at::Tensor& D,
         const void* bias, bool add) {
  const int device = (int)A.device().index();
  if (device != (int)c10::cuda::current_device()) return false;  // the handle is that of the current device
  Key key;
  std::memset(&key, 0, sizeof(key));
  key.kind = kind;
  key.device = device;
  key.m = m;
  key.n = n;
  key.k = k;
  const at::CuBLASReductionOption reductions = at::globalContext().allowBF16ReductionCuBLAS();
  key.flags = ((uint32_t)reductions << 20) | (q.bias ? 1u : 0u) | (add ? 2u : 0u) | (q.relu ? 4u : 0u) | (alignment_log(A.data_ptr()) << 4) | (alignment_log(B.data_ptr()) << 8) |
              (alignment_log(D.data_ptr()) << 12) | (q.bias ? alignment_log(bias) << 16 : 0u);
  // per thread: a plan's descriptor carries the bias pointer of the call
  using Plans = std::unordered_map<Key, std::unique_ptr<Plan>, Hash>;
  static thread_local Plans* plans = new Plans();  // library objects: not destroyed with the thread
  cublasLtHandle_t lt = at::cuda::getCurrentCUDABlasLtHandle();
  auto it = plans->find(key);
  if (it == plans->end()) {
    if (plans->size() >= kMaxPlans) plans->clear();
    auto p = std::make_unique<Plan>();
    p->usable = build(*p, lt, q, A.data_ptr(), B.data_ptr(), D.data_ptr(), bias, reductions);
    it = plans->emplace(key, std::move(p)).first;
  }
  Plan& p = *it->second;
  if (!p.usable) return false;
  if (q.bias &&
      cublasLtMatmulDescSetAttribute(p.desc, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof(bias)) != CUBLAS_STATUS_SUCCESS)
    return false;
  cudaStream_t s = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
  auto ws = MemoryPool::for_device(device).pull(p.workspace, (uint64_t)(uintptr_t)s);
  const float one = 1.f, beta = add ? 1.f : 0.f;
  if (cublasLtMatmul(lt, p.desc, &one, A.data_ptr(), p.a, B.data_ptr(), p.b, &beta, D.data_ptr(), p.d, D.data_ptr(), p.d,
                     &p.algo, ws->ptr(), p.workspace, s) == CUBLAS_STATUS_SUCCESS)
    return true;
  p.usable = false;
  return false;
}

bool plain(const at::Tensor& t) {
  return t.is_cuda() && t.dim() == 2 && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.numel() > 0;
}
// The library is given addresses and sizes only: what does not fit together is refused here, and the framework's
// product says why.
bool sized(const at::Tensor& t, int64_t rows, int64_t cols, const at::Tensor& like) {
  return t.size(0) == rows && t.size(1) == cols && t.device() == like.device();
}

}  // namespace

bool linear(const at::Tensor& x, const at::Tensor& w, const at::Tensor& b, bool relu, at::Tensor& y) {
  if (!plain(x) || !plain(w) || !plain(y)) return false;
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  if (!sized(w, N, K, x) || !sized(y, M, N, x)) return false;
  if (b.defined() && (b.scalar_type() != at::kBFloat16 || !b.is_contiguous() || b.dim() != 1 || b.size(0) != N || b.device() != x.device()))
    return false;
  const Problem q{CUBLAS_OP_T, CUBLAS_OP_N, K, N, K, M, N, M, false, b.defined(), true, relu};
  return run(0, q, M, N, K, w, x, y, b.defined() ? b.data_ptr() : nullptr, false);
}

bool input_grad(const at::Tensor& dy, const at::Tensor& w, at::Tensor& dx) {
  if (!plain(dy) || !plain(w) || !plain(dx)) return false;
  const int64_t M = dy.size(0), N = dy.size(1), K = w.size(1);
  if (!sized(w, N, K, dy) || !sized(dx, M, K, dy)) return false;
  const Problem q{CUBLAS_OP_N, CUBLAS_OP_N, K, N, N, M, K, M, false, false, false, false};
  return run(1, q, M, N, K, w, dy, dx, nullptr, false);
}

bool weight_grad(const at::Tensor& dy, const at::Tensor& x, at::Tensor& g, bool accumulate) {
  if (!plain(dy) || !plain(x) || g.scalar_type() != at::kFloat || !g.is_contiguous() || g.dim() != 2) return false;
  const int64_t M = dy.size(0), N = dy.size(1), K = x.size(1);
  if (!sized(x, M, K, dy) || !sized(g, N, K, dy)) return false;
  const Problem q{CUBLAS_OP_N, CUBLAS_OP_T, K, M, N, M, K, N, true, false, false, false};
  return run(2, q, M, N, K, x, dy, g, nullptr, accumulate);
}

}  // namespace gemm
}  // namespace trainer
}  // namespace bagua
