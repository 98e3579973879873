// Plain 16-bit matrix products through cublasLt, on raw row-major pointers.
#pragma once
#include "host_common.h"

namespace foxh {

struct Gemm {
  int device = 0, code = 0;          // FOX_DTYPE_BF16 / FP16
  cudaStream_t st = nullptr;
  void* work = nullptr;              // kGemmWorkspace bytes, this stream's for the products queued one after another
};
constexpr size_t kGemmWorkspace = size_t{32} << 20;

// D (m, n) = op(A) op(B) [+ C] [+ bias], fp32 accumulation, row-major with row strides: A is (m, k), or (k, m) when ta; B is
// (k, n), or (n, k) when tb.  C may be null (nothing is added) and is another matrix than D.  bias: n values of D's type on a
// 16-byte boundary, added to every row before D is rounded, or null.
void gemm(const Gemm& g, int64_t m, int64_t n, int64_t k, const void* A, int64_t lda, bool ta, const void* B, int64_t ldb, bool tb,
          const void* C, int64_t ldc, void* D, int64_t ldd, const void* bias = nullptr);

}  // namespace foxh
