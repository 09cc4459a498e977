// Semiring GEMM, double elements, on the element-dealt tiles of f64_tile.cuh.
//
// What bounds it: an FP64 instruction holds an SM partition for 64 cycles, and fmin and fmax on doubles
// compare on that pipe (a (min, +) step of add and fmin measured 152 cycles).  Here min and max run on
// the integer ALUs, on order-preserving 64-bit keys, which leaves (min, +), (max, +) and (max, x) their
// one add or multiply and (max, min) and (min, max) no FP64 instruction at all.
//
// With key(x) = the bits of x, magnitude bits flipped when the sign is set, signed 64-bit order is
// the order of doubles (-0.0 just below 0.0), NaNs beyond the infinities on both sides.  As unsigned
//   (+) = min   code(x) = key(x) - key(-Inf)      (+) = max   code(x) = key(Inf) - key(x)
// every number gets a code up to TOP = 0xFFE0000000000001, smaller is the one (+) keeps, (+)'s
// identity is TOP, and every NaN is above TOP: unsigned min from TOP on is (+) with NaNs ignored.
// For (max, min) and (min, max) the panels are rewritten in shared memory as code + 1, 0 for a NaN:
// there (x) is the unsigned max, which ignores a NaN beside a number, and its result minus one, which
// sends a pair of NaNs to the top, goes into the unsigned min.
//
// Measured against fmin / fmax on register tiles of 4 x 4 a thread: (min, +) 64^3 161 -> 13 us a call,
// 300^3 730 -> 74 us, 1024^3 4.85 -> 2.13 ms (1.74 at the pipe's rate; (max, x) the same);
// (max, min) 1539 x 390 x 382 1.82 -> 0.21 ms, 1024^3 0.94 ms, bound by the integer instructions.
#include "f64_gemm.cuh"
#include "semiring.cuh"

namespace gb {

template <int SR>
struct F64Semiring {
  using Word = unsigned long long;
  using Acc = Word;
  static constexpr bool MIN = SemiringOp<double, SR>::kMinPlus;
  static constexpr bool ENCODE = SR == GB_SEMIRING_MAX_MIN || SR == GB_SEMIRING_MIN_MAX;
  static constexpr int AHEAD = 1;   // (4: the k loops of (max, min) and (min, max) spill, 1024^3 0.92 -> 0.95 ms)
  using Elem = typename std::conditional<ENCODE, Word, double>::type;
  static constexpr Word TOP = 0xFFE0000000000001ull, KEY_INF = 0x7FF0000000000000ull;   // key(-Inf) = ~KEY_INF
  int accumulate;

  static __device__ __forceinline__ Word flip(Word w) {   // bits <-> key
    return w ^ (static_cast<Word>(static_cast<long long>(w) >> 63) >> 1);
  }
  static __device__ __forceinline__ Word code(Word bits) {
    return MIN ? flip(bits) - ~KEY_INF : KEY_INF - flip(bits);
  }
  static __device__ __forceinline__ Word code(double x) {
    return code(static_cast<Word>(__double_as_longlong(x)));
  }
  static __device__ __forceinline__ Word lesser(Word a, Word b) { return a < b ? a : b; }
  static __device__ __forceinline__ Word encode(Word bits) {
    const Word w = code(bits);
    return w > TOP ? 0 : w + 1;
  }
  static __device__ __forceinline__ Word step(Word acc, Elem a, Elem b) {
    if constexpr (ENCODE) return lesser(acc, (a > b ? a : b) - 1);
    else return lesser(acc, code(SemiringOp<double, SR>::otimes(a, b)));
  }
  __device__ __forceinline__ Word init(const double*, bool) const { return TOP; }
  __device__ __forceinline__ bool reads_c() const { return accumulate != 0; }
  __device__ __forceinline__ double value(double c, Word acc) const { return value(lesser(code(c), acc)); }
  __device__ __forceinline__ bool plain() const { return false; }
  static __device__ __forceinline__ double raw(Word acc) { return value(acc); }
  static __device__ __forceinline__ double value(Word acc) {
    const Word bits = flip(MIN ? acc + ~KEY_INF : KEY_INF - acc);
    return SrArith<double>::canon(__longlong_as_double(static_cast<long long>(bits)));
  }
};

int semiring_gemm_f64(int sr, int ta, int tb, int64_t M, int64_t N, int64_t K, const double* A, int64_t lda,
                      const double* B, int64_t ldb, int accumulate, double* C, int64_t ldc, int sms, cudaStream_t s) {
  switch (sr) {
#define GB_SR(SR_)                                                                                                  \
  case SR_:                                                                                                         \
    return launch_f64_gemm(GB_KERNEL_SEMIRING_GEMM, F64Semiring<SR_>{accumulate}, M, N, K, A, ta ? lda : 1,         \
                           ta ? 1 : lda, B, tb ? ldb : 1, tb ? 1 : ldb, C, ldc, sms, s);
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

}  // namespace gb
