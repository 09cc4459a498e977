// Semiring GEMM, float elements: one-warp tiles on k pairs (semiring4_tile.cuh) or 128x128
// CTA tiles, 8x8 per thread (semiring.cuh).
#include "semiring.cuh"

namespace gb {

int semiring_gemm_f32(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
                      const float* B, int64_t ldb, int accumulate, float* C, int64_t ldc, int sms, cudaStream_t s) {
  return semiring4_gemm<float, 8>(sr, ta, tb, M, N, K, A, lda, B, ldb, accumulate, C, ldc, sms, s);
}

}  // namespace gb
