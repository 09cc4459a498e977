// Semiring GEMM on the CUDA cores: C = [C (+)] (+)_k op(A)[i,k] (x) op(B)[k,j].
//
// jBLAS keeps a tuple-SIMD Vec type (src/simd.jl) out of its module with the note that it
// could serve "custom number types ... so it works with min-plus algebra" (src/jBLAS.jl:10).
// Here the custom arithmetic is a policy of the tiles (semiring4_tile.cuh and simt_gemm.cuh for 4-byte
// elements, semiring_f64.cu for doubles): the accumulator starts at the identity of (+), each k
// folds in one (x) product, and the epilogue folds in C when accumulating.
//
// (+) is min or max.  For floating point it ignores a NaN operand (fminf / fmaxf) and a
// zero result is stored as +0.0: min and max are then associative and commutative on every
// input, including the sign of zero, so the result does not depend on the K order.  int32
// + and * wrap modulo 2^32 (computed on uint32_t).
//
// Because (+) is exact and associative, two consecutive k can be folded in by one
// three-input min / max (min.f32 / max.f32 with three sources; __vimin3_s32 / __vimax3_s32):
// 1.5 instructions per element instead of 2 where that is faster (float: every semiring;
// int32: (max, min) and (min, max)).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <type_traits>

#include "gb_common.cuh"
#include "profile.cuh"
#include "semiring4_tile.cuh"
#include "simt_gemm.cuh"

namespace gb {

template <typename T>
struct SrArith;

template <>
struct SrArith<float> {
  static __device__ __forceinline__ float lo() { return __int_as_float(0xff800000); }   // -Inf
  static __device__ __forceinline__ float hi() { return __int_as_float(0x7f800000); }   // +Inf
  static __device__ __forceinline__ float min(float a, float b) { return fminf(a, b); }
  static __device__ __forceinline__ float max(float a, float b) { return fmaxf(a, b); }
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float canon(float v) { return v == 0.0f ? 0.0f : v; }
  static __device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
  }
  static __device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
  }
};

template <>
struct SrArith<double> {   // (identities and the steps of a chain: semiring_f64.cu)
  static __device__ __forceinline__ double min(double a, double b) { return fmin(a, b); }
  static __device__ __forceinline__ double max(double a, double b) { return fmax(a, b); }
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double canon(double v) { return v == 0.0 ? 0.0 : v; }
};

template <>
struct SrArith<int32_t> {
  static __device__ __forceinline__ int32_t lo() { return INT32_MIN; }
  static __device__ __forceinline__ int32_t hi() { return INT32_MAX; }
  static __device__ __forceinline__ int32_t min(int32_t a, int32_t b) { return a < b ? a : b; }
  static __device__ __forceinline__ int32_t max(int32_t a, int32_t b) { return a > b ? a : b; }
  static __device__ __forceinline__ int32_t add(int32_t a, int32_t b) {
    return static_cast<int32_t>(static_cast<uint32_t>(a) + static_cast<uint32_t>(b));
  }
  static __device__ __forceinline__ int32_t mul(int32_t a, int32_t b) {
    return static_cast<int32_t>(static_cast<uint32_t>(a) * static_cast<uint32_t>(b));
  }
  static __device__ __forceinline__ int32_t canon(int32_t v) { return v; }
  static __device__ __forceinline__ int32_t min3(int32_t a, int32_t b, int32_t c) { return __vimin3_s32(a, b, c); }
  static __device__ __forceinline__ int32_t max3(int32_t a, int32_t b, int32_t c) { return __vimax3_s32(a, b, c); }
};

template <typename T, int SR>
struct SemiringOp {
  using Ar = SrArith<T>;
  static constexpr bool kMinPlus = SR == GB_SEMIRING_MIN_PLUS || SR == GB_SEMIRING_MIN_MAX;
  static constexpr bool kPairs =
      std::is_floating_point<T>::value || SR == GB_SEMIRING_MAX_MIN || SR == GB_SEMIRING_MIN_MAX;
  int accumulate;

  static __device__ __forceinline__ T oplus(T x, T y) { return kMinPlus ? Ar::min(x, y) : Ar::max(x, y); }
  static __device__ __forceinline__ T otimes(T a, T b) {
    if (SR == GB_SEMIRING_MIN_PLUS || SR == GB_SEMIRING_MAX_PLUS) return Ar::add(a, b);
    if (SR == GB_SEMIRING_MAX_MIN) return Ar::min(a, b);
    if (SR == GB_SEMIRING_MIN_MAX) return Ar::max(a, b);
    return Ar::mul(a, b);
  }
  static __device__ __forceinline__ T init() { return kMinPlus ? Ar::hi() : Ar::lo(); }
  static __device__ __forceinline__ T step(T acc, T a, T b) { return oplus(acc, otimes(a, b)); }
  static __device__ __forceinline__ T step2(T acc, T a0, T b0, T a1, T b1) {
    const T p0 = otimes(a0, b0), p1 = otimes(a1, b1);
    return kMinPlus ? Ar::min3(acc, p0, p1) : Ar::max3(acc, p0, p1);
  }
  __device__ __forceinline__ void store(T* c, T acc) const { *c = Ar::canon(accumulate ? oplus(*c, acc) : acc); }
};

template <typename T, int SR, int BM, int BN, int BK, int TM, int TN>
static int launch_semiring(int ta, int tb, int64_t M, int64_t N, int64_t K, const T* A, int64_t lda,
                           const T* B, int64_t ldb, int accumulate, T* C, int64_t ldc, cudaStream_t s) {
  dim3 grid;
  if (!simt_grid<BM, BN>(M, N, &grid)) return GB_ERR_UNSUPPORTED;
  constexpr int NT = (BM / TM) * (BN / TN);
  const SemiringOp<T, SR> op{accumulate};
#define GB_SR_CASE(TA_, TB_)                                                                        \
  GB_LAUNCH(GB_KERNEL_SEMIRING_GEMM, s,                                                             \
            (simt_gemm_kernel<T, SemiringOp<T, SR>, BM, BN, BK, TM, TN, TA_, TB_><<<grid, NT, 0, s>>>( \
                M, N, K, op, A, lda, B, ldb, C, ldc)))
  if (!ta && !tb) GB_SR_CASE(false, false);
  else if (!ta && tb) GB_SR_CASE(false, true);
  else if (ta && !tb) GB_SR_CASE(true, false);
  else GB_SR_CASE(true, true);
#undef GB_SR_CASE
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

// All semirings for one element type and tile configuration (M, N > 0; arguments checked).
template <typename T, int BM, int BN, int BK, int TM, int TN>
static int semiring_gemm(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const T* A, int64_t lda,
                         const T* B, int64_t ldb, int accumulate, T* C, int64_t ldc, cudaStream_t s) {
  switch (sr) {
#define GB_SR(SR_)                                                                                 \
  case SR_:                                                                                        \
    return launch_semiring<T, SR_, BM, BN, BK, TM, TN>(ta, tb, M, N, K, A, lda, B, ldb, accumulate, C, \
                                                       ldc, s);
    GB_SR(GB_SEMIRING_MIN_PLUS)
    GB_SR(GB_SEMIRING_MAX_PLUS)
    GB_SR(GB_SEMIRING_MAX_MIN)
    GB_SR(GB_SEMIRING_MIN_MAX)
    GB_SR(GB_SEMIRING_MAX_TIMES)
#undef GB_SR
    default:
      return GB_ERR_INVALID_VALUE;
  }
}

// ------------------------------------------------------------------ 4-byte elements
__device__ __forceinline__ pair4 add_f32x2(pair4 a, pair4 b) {
  pair4 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ pair4 mul_f32x2(pair4 a, pair4 b) {
  pair4 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
template <typename T>
__device__ __forceinline__ T as4(uint32_t v);
template <>
__device__ __forceinline__ float as4<float>(uint32_t v) { return __uint_as_float(v); }
template <>
__device__ __forceinline__ int32_t as4<int32_t>(uint32_t v) { return static_cast<int32_t>(v); }
__device__ __forceinline__ uint32_t bits4(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t bits4(int32_t v) { return static_cast<uint32_t>(v); }

// SemiringOp on the bits of 4-byte elements, as semiring4_tile takes them.
template <typename T, int SR>
struct Semiring4Op {
  using Op = SemiringOp<T, SR>;
  int accumulate;
  static __device__ __forceinline__ uint32_t init() { return bits4(Op::init()); }
  static __device__ __forceinline__ uint32_t step(uint32_t acc, uint32_t a, uint32_t b) {
    return bits4(Op::step(as4<T>(acc), as4<T>(a), as4<T>(b)));
  }
  static __device__ __forceinline__ uint32_t step2(uint32_t acc, pair4 a, pair4 b) {
    if constexpr (std::is_same<T, float>::value && (SR == GB_SEMIRING_MIN_PLUS || SR == GB_SEMIRING_MAX_PLUS ||
                                                    SR == GB_SEMIRING_MAX_TIMES)) {
      const pair4 p = SR == GB_SEMIRING_MAX_TIMES ? mul_f32x2(a, b) : add_f32x2(a, b);
      const float x = as4<T>(lo4(p)), y = as4<T>(hi4(p)), c = as4<T>(acc);
      return bits4(Op::kMinPlus ? SrArith<T>::min3(c, x, y) : SrArith<T>::max3(c, x, y));
    } else if constexpr (Op::kPairs) {
      return bits4(Op::step2(as4<T>(acc), as4<T>(lo4(a)), as4<T>(lo4(b)), as4<T>(hi4(a)), as4<T>(hi4(b))));
    } else {
      return step(step(acc, lo4(a), lo4(b)), hi4(a), hi4(b));
    }
  }
  __device__ __forceinline__ bool reads_c() const { return accumulate != 0; }
  __device__ __forceinline__ uint32_t value(uint32_t acc) const { return bits4(SrArith<T>::canon(as4<T>(acc))); }
  __device__ __forceinline__ uint32_t value(uint32_t c, uint32_t acc) const {
    return bits4(SrArith<T>::canon(Op::oplus(as4<T>(c), as4<T>(acc))));
  }
};

// One CTA per SM of WARPS independent warps, as native FP32 (native_f32.cu) deals its tiles.
template <class S, int WARPS, class Op>
__global__ void __launch_bounds__(32 * WARPS, 1)
    semiring4_kernel(int64_t M, int64_t N, int64_t K, const Op op, const uint32_t* __restrict__ A, int64_t ars,
                     int64_t aks, const uint32_t* __restrict__ B, int64_t bks, int64_t bcs, uint32_t* __restrict__ C,
                     int64_t ldc, unsigned tiles_m, unsigned tiles) {
  extern __shared__ __align__(16) uint32_t sr_smem[];
  const unsigned warp = threadIdx.x >> 5;
  uint32_t* smem = sr_smem + warp * (S::SMEM_BYTES / 4);
  for (unsigned t = blockIdx.x + gridDim.x * warp; t < tiles; t += gridDim.x * WARPS) {
    const unsigned tn = t / tiles_m, tm = t - tn * tiles_m;
    const int64_t m0 = static_cast<int64_t>(tm) * S::BM, n0 = static_cast<int64_t>(tn) * S::BN;
    const int r = static_cast<int>(M - m0 < S::BM ? M - m0 : S::BM), c = static_cast<int>(N - n0 < S::BN ? N - n0 : S::BN);
    semiring4_tile<S>(r, c, K, op, A + m0 * ars, ars, aks, B + n0 * bcs, bks, bcs, C + m0 + n0 * ldc, ldc, smem);
  }
}

template <class S, int WARPS, class Op>
static int launch_semiring4(const Op& op, int64_t M, int64_t N, int64_t K, const uint32_t* A, int64_t ars, int64_t aks,
                            const uint32_t* B, int64_t bks, int64_t bcs, uint32_t* C, int64_t ldc, int sms,
                            cudaStream_t s) {
  constexpr int SMEM = WARPS * S::SMEM_BYTES;
  static_assert(SMEM <= 232448, "shared memory per CTA");
  const int64_t tiles_m = (M + S::BM - 1) / S::BM, tiles = tiles_m * ((N + S::BN - 1) / S::BN);
  if (tiles > 0x7FFFFFFF) return GB_ERR_UNSUPPORTED;
  auto kernel = semiring4_kernel<S, WARPS, Op>;
  static std::atomic<unsigned long long> opted{0};
  const int rc = opt_in_dynamic_smem(kernel, SMEM, opted);
  if (rc) return rc;
  GB_LAUNCH(GB_KERNEL_SEMIRING_GEMM, s,
            (kernel<<<static_cast<unsigned>(tiles < sms ? tiles : sms), 32 * WARPS, SMEM, s>>>(
                M, N, K, op, A, ars, aks, B, bks, bcs, C, ldc, static_cast<unsigned>(tiles_m),
                static_cast<unsigned>(tiles))));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

// All semirings of a 4-byte element type (M, N > 0; arguments checked).  One-warp 32 x 32 tiles, or the
// 128 x 128 tiles of simt_gemm.cuh, whichever are done sooner on the fullest SM: a k of n tiles takes
// max(110, 19.2 n (1 + 2.2 / (n + 1))) cycles on the former and max(340, 300 n) on the latter (the
// large tiles read a quarter of the operands, the small ones leave no SM idle).  (min, +) in float:
// 512^3 93 -> 33 us, 1024^3 175 -> 94, 2048^3 618 -> 567; at 4096^3 the large tiles are ahead.
template <typename T, int BK>
static int semiring4_gemm(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const T* A, int64_t lda,
                          const T* B, int64_t ldb, int accumulate, T* C, int64_t ldc, int sms, cudaStream_t s) {
  if ((M + 127) / 128 > 0x7FFFFFFF || (N + 127) / 128 > 65535) return GB_ERR_UNSUPPORTED;
  auto fullest = [&](int64_t d) {
    return static_cast<double>((((M + d - 1) / d) * ((N + d - 1) / d) + sms - 1) / sms);
  };
  const double n = fullest(32), small = n * 19.2 * (1.0 + 2.2 / (n + 1.0)), large = 300.0 * fullest(128);
  if ((large < 340.0 ? 340.0 : large) < (small < 110.0 ? 110.0 : small))
    return semiring_gemm<T, 128, 128, BK, 8, 8>(sr, ta, tb, M, N, K, A, lda, B, ldb, accumulate, C, ldc, s);
  const uint32_t *a = reinterpret_cast<const uint32_t*>(A), *b = reinterpret_cast<const uint32_t*>(B);
  uint32_t* c = reinterpret_cast<uint32_t*>(C);
  const int64_t ars = ta ? lda : 1, aks = ta ? 1 : lda, bks = tb ? ldb : 1, bcs = tb ? 1 : ldb;
  switch (sr) {
#define GB_SR(SR_)                                                                                            \
  case SR_:                                                                                                   \
    return launch_semiring4<SrShape<8, 4>, 16>(Semiring4Op<T, SR_>{accumulate}, M, N, K, a, ars, aks, b, bks, bcs, \
                                               c, ldc, sms, s);
    GB_SR(GB_SEMIRING_MIN_PLUS)
    GB_SR(GB_SEMIRING_MAX_PLUS)
    GB_SR(GB_SEMIRING_MAX_MIN)
    GB_SR(GB_SEMIRING_MIN_MAX)
    GB_SR(GB_SEMIRING_MAX_TIMES)
#undef GB_SR
    default:
      return GB_ERR_INVALID_VALUE;
  }
}

int semiring_gemm_f64(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const double* A, int64_t lda,
                      const double* B, int64_t ldb, int accumulate, double* C, int64_t ldc, int sms, cudaStream_t s);
int semiring_gemm_f32(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
                      const float* B, int64_t ldb, int accumulate, float* C, int64_t ldc, int sms, cudaStream_t s);
int semiring_gemm_i32(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const int32_t* A,
                      int64_t lda, const int32_t* B, int64_t ldb, int accumulate, int32_t* C, int64_t ldc, int sms,
                      cudaStream_t s);

}  // namespace gb
