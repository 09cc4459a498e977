// FP32 operands as BF16 term planes (adjoint.cu), for the term products (gemm_f32_tc.cu) and the adjoint.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace gb {

// The R x K operand whose element (r, k) is X[r rs + k ks], to planes [term][r][pitch] and, with
// planes_t, from the same read, [term][k][pitch_t] (rows contiguous only).
struct SplitOperand {
  const float* X;
  int64_t R, K, rs, ks;
  __nv_bfloat16* planes;
  int64_t pitch;
  __nv_bfloat16* planes_t;
  int64_t pitch_t;
};
constexpr int SPLIT_MAX_OPERANDS = 3;

// Splits up to SPLIT_MAX_OPERANDS operands into nterms = 2 or 3 terms each in one launch, counted as
// `kind`, which also writes zeros to zero[0 .. nzero - 1].
int split_bf16_terms(const SplitOperand* ops, int count, int nterms, unsigned int* zero, int nzero, int kind,
                     cudaStream_t s);

}  // namespace gb
