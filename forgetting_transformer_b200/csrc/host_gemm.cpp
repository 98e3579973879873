// torch.mm costs the host 9 us a call (dispatch, checks, heuristics, a result tensor), which is what bounded a block's
// step on short sequences; the same library call on remembered descriptors costs 3.
#include "host_gemm.h"

#include <cublasLt.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <unordered_map>

namespace foxh {

namespace {
struct Key {
  int64_t v[8];   // m, n, k, lda, ldb, ldc, ldd, flags
  bool operator==(const Key& o) const { return std::equal(v, v + 8, o.v); }
};
struct KeyHash {
  size_t operator()(const Key& k) const {
    uint64_t h = 1469598103934665603ull;
    for (int64_t x : k.v) h = (h ^ static_cast<uint64_t>(x)) * 1099511628211ull, h ^= h >> 29;
    return static_cast<size_t>(h);
  }
};

void lt(cublasStatus_t s, const char* what) {
  if (s != CUBLAS_STATUS_SUCCESS) raise_fox(std::string(what) + " failed: cublasLt status " + std::to_string(static_cast<int>(s)));
}

// Descriptors and the algorithm the library proposes for one product shape.
struct Plan {
  cublasLtMatmulDesc_t op = nullptr;
  cublasLtMatrixLayout_t a = nullptr, b = nullptr, c = nullptr, d = nullptr;
  cublasLtMatmulAlgo_t algo;
  ~Plan() {
    if (a) cublasLtMatrixLayoutDestroy(a);
    if (b) cublasLtMatrixLayoutDestroy(b);
    if (c) cublasLtMatrixLayoutDestroy(c);
    if (d) cublasLtMatrixLayoutDestroy(d);
    if (op) cublasLtMatmulDescDestroy(op);
  }
};

cublasLtHandle_t handle(int device) {
  static std::mutex mu;
  static cublasLtHandle_t handles[64] = {};
  if (device < 0 || device >= 64) raise_fox("device ordinal out of range");
  std::lock_guard<std::mutex> g(mu);
  if (!handles[device]) lt(cublasLtCreate(&handles[device]), "cublasLtCreate");
  return handles[device];
}

constexpr size_t kMostPlans = 4096;
std::mutex g_plans_mu;
std::unordered_map<Key, std::shared_ptr<const Plan>, KeyHash> g_plans;

// (of an operation descriptor) the library's matrices are column-major: D^T = op(B)^T op(A)^T, so B is its first operand
void describe(cublasLtMatmulDesc_t op, bool ta, bool tb, const void* bias) {
  const cublasOperation_t opb = tb ? CUBLAS_OP_T : CUBLAS_OP_N, opa = ta ? CUBLAS_OP_T : CUBLAS_OP_N;
  lt(cublasLtMatmulDescSetAttribute(op, CUBLASLT_MATMUL_DESC_TRANSA, &opb, sizeof(opb)), "cublasLtMatmulDescSetAttribute");
  lt(cublasLtMatmulDescSetAttribute(op, CUBLASLT_MATMUL_DESC_TRANSB, &opa, sizeof(opa)), "cublasLtMatmulDescSetAttribute");
  if (!bias) return;
  const cublasLtEpilogue_t add = CUBLASLT_EPILOGUE_BIAS;
  lt(cublasLtMatmulDescSetAttribute(op, CUBLASLT_MATMUL_DESC_EPILOGUE, &add, sizeof(add)), "cublasLtMatmulDescSetAttribute");
  lt(cublasLtMatmulDescSetAttribute(op, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &bias, sizeof(bias)), "cublasLtMatmulDescSetAttribute");
}

std::shared_ptr<const Plan> make_plan(cublasLtHandle_t h, const Key& key, bool ta, bool tb, bool bf16, uint32_t align, const void* bias) {
  const int64_t m = key.v[0], n = key.v[1], k = key.v[2];
  auto p = std::make_shared<Plan>();
  const cudaDataType_t dt = bf16 ? CUDA_R_16BF : CUDA_R_16F;
  lt(cublasLtMatmulDescCreate(&p->op, CUBLAS_COMPUTE_32F, CUDA_R_32F), "cublasLtMatmulDescCreate");
  describe(p->op, ta, tb, bias);
  lt(cublasLtMatrixLayoutCreate(&p->b, dt, tb ? k : n, tb ? n : k, key.v[4]), "cublasLtMatrixLayoutCreate");
  lt(cublasLtMatrixLayoutCreate(&p->a, dt, ta ? m : k, ta ? k : m, key.v[3]), "cublasLtMatrixLayoutCreate");
  lt(cublasLtMatrixLayoutCreate(&p->c, dt, n, m, key.v[5]), "cublasLtMatrixLayoutCreate");
  lt(cublasLtMatrixLayoutCreate(&p->d, dt, n, m, key.v[6]), "cublasLtMatrixLayoutCreate");
  cublasLtMatmulPreference_t pref;
  lt(cublasLtMatmulPreferenceCreate(&pref), "cublasLtMatmulPreferenceCreate");
  const size_t ws = kGemmWorkspace;
  // split reductions only in fp32 (the in-place scheme adds partial sums in the output's 16 bits)
  const uint32_t reductions = CUBLASLT_REDUCTION_SCHEME_NONE | CUBLASLT_REDUCTION_SCHEME_COMPUTE_TYPE;
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &ws, sizeof(ws));
  cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_REDUCTION_SCHEME_MASK, &reductions, sizeof(reductions));
  for (auto attr : {CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES,
                    CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES})
    cublasLtMatmulPreferenceSetAttribute(pref, attr, &align, sizeof(align));
  cublasLtMatmulHeuristicResult_t res;
  int found = 0;
  const cublasStatus_t s = cublasLtMatmulAlgoGetHeuristic(h, p->op, p->b, p->a, p->c, p->d, pref, 1, &res, &found);
  cublasLtMatmulPreferenceDestroy(pref);
  lt(s, "cublasLtMatmulAlgoGetHeuristic");
  if (found < 1) raise_fox("cublasLt has no algorithm for this product");
  p->algo = res.algo;
  return p;
}
}  // namespace

void gemm(const Gemm& g, int64_t m, int64_t n, int64_t k, const void* A, int64_t lda, bool ta, const void* B, int64_t ldb, bool tb,
          const void* C, int64_t ldc, void* D, int64_t ldd, const void* bias) {
  const bool bf16 = g.code == FOX_DTYPE_BF16;
  if (!C) {
    C = D;
    ldc = ldd;
    // (with beta = 0 the operand is not read)
  }
  const float alpha = 1.f, beta = C == D && ldc == ldd ? 0.f : 1.f;
  const uintptr_t bits = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
                         reinterpret_cast<uintptr_t>(D) | 256;
  const uint32_t align = static_cast<uint32_t>(bits & (~bits + 1));
  const Key key{{m, n, k, lda, ldb, ldc, ldd,
                 static_cast<int64_t>(g.device) | (ta ? 64 : 0) | (tb ? 128 : 0) | (bf16 ? 256 : 0) | (beta != 0.f ? 512 : 0) | (bias ? 1024 : 0) |
                     (static_cast<int64_t>(align) << 16)}};
  const cublasLtHandle_t h = handle(g.device);
  std::shared_ptr<const Plan> p;
  {
    std::lock_guard<std::mutex> lock(g_plans_mu);
    auto it = g_plans.find(key);
    if (it != g_plans.end()) p = it->second;
  }
  if (!p) {
    p = make_plan(h, key, ta, tb, bf16, align, bias);
    std::lock_guard<std::mutex> lock(g_plans_mu);
    if (g_plans.size() >= kMostPlans) g_plans.clear();
    g_plans.emplace(key, p);
  }
  // (the remembered descriptor is shared and holds another call's bias pointer: a bias takes one of its own)
  cublasLtMatmulDescOpaque_t own;
  cublasLtMatmulDesc_t op = p->op;
  if (bias) {
    lt(cublasLtMatmulDescInit(&own, CUBLAS_COMPUTE_32F, CUDA_R_32F), "cublasLtMatmulDescInit");
    op = &own;
    describe(op, ta, tb, bias);
  }
  lt(cublasLtMatmul(h, op, &alpha, B, p->b, A, p->a, &beta, C, p->c, D, p->d, &p->algo, g.work, kGemmWorkspace, g.st),
     "cublasLtMatmul");
}

}  // namespace foxh
