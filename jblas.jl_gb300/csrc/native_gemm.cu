// Native FP64 GEMM on the CUDA cores (GB_MODE_NATIVE), on the element-dealt tiles of f64_tile.cuh,
// and C = beta C for both types (FP32: native_f32.cu).
//
// Per element the arithmetic is exactly jmul!'s: d = a1*x1, then d = fma(ak, xk, d) for
// k = 2..K in order (src/gemm.jl:76-89, 154-168).  The accumulator starts at -0.0 so
// that the first step fma(a1, x1, -0.0) equals the rounded product a1*x1 bit for bit,
// signed zeros included; the K tail is handled with an exact trip count (no zero
// padding, which would turn -0 into +0 and Inf*0 into NaN).
#include <cstring>

#include "f64_gemm.cuh"
#include "gb_common.cuh"
#include "native_gemm.cuh"
#include "profile.cuh"

namespace gb {

// C = beta * C (alpha == 0 or K == 0); beta == 0 writes zeros without reading C.
template <typename T>
__global__ void scale_c_kernel(int64_t M, int64_t N, T beta, T* __restrict__ C, int64_t ldc) {
  const int64_t total = M * N;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t m = t % M, n = t / M;
    T* c = &C[m + n * ldc];
    *c = (beta == T(0)) ? T(0) : beta * *c;
  }
}

template <typename T>
static int launch_scale(int64_t M, int64_t N, T beta, T* C, int64_t ldc, cudaStream_t s) {
  const int64_t total = M * N;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  if (blocks < 1) blocks = 1;
  GB_LAUNCH(GB_KERNEL_SCALE_C, s,
            scale_c_kernel<T><<<static_cast<unsigned>(blocks), 256, 0, s>>>(M, N, beta, C, ldc));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

int native_scale_f32(int64_t M, int64_t N, float beta, float* C, int64_t ldc, cudaStream_t s) {
  return launch_scale<float>(M, N, beta, C, ldc, s);
}

int native_kernel_onto_f64(int64_t M, int64_t N, int64_t K, const double* A, int64_t lda, const double* B,
                           int64_t ldb, double* C, int64_t ldc, int sms, cudaStream_t s) {
  if (M == 0 || N == 0 || K == 0) return GB_OK;   // an empty chain leaves D as it is
  return launch_f64_gemm(GB_KERNEL_NATIVE_GEMM, F64Chain<true>{1.0, 0.0, F64_CHAIN}, M, N, K, A, 1, lda, B, 1, ldb, C, ldc,
                         sms, s);
}

int native_gemm_f64(int ta, int tb, int64_t M, int64_t N, int64_t K, double alpha, const double* A,
                    int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc, int sms,
                    cudaStream_t s) {
  if (M == 0 || N == 0) return GB_OK;
  if (alpha == 0.0 || K == 0) return launch_scale<double>(M, N, beta, C, ldc, s);
  long long ab[2];
  std::memcpy(&ab[0], &alpha, 8);
  std::memcpy(&ab[1], &beta, 8);
  return launch_f64_gemm(GB_KERNEL_NATIVE_GEMM, F64Chain<false>{alpha, beta, f64_out(ab[0], ab[1])}, M, N, K, A,
                         ta ? lda : 1, ta ? 1 : lda, B, tb ? ldb : 1, tb ? 1 : ldb, C, ldc, sms, s);
}

}  // namespace gb
