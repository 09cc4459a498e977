// Native FP64 GEMM on the CUDA cores (GB_MODE_NATIVE), on the element-dealt tiles of f64_tile.cuh,
// and C = beta C for both types (FP32: native_f32.cu).
//
// Per element the arithmetic is exactly jmul!'s: d = a1*x1, then d = fma(ak, xk, d) for
// k = 2..K in order (src/gemm.jl:76-89, 154-168).  The accumulator starts at -0.0 so
// that the first step fma(a1, x1, -0.0) equals the rounded product a1*x1 bit for bit,
// signed zeros included; the K tail is handled with an exact trip count (no zero
// padding, which would turn -0 into +0 and Inf*0 into NaN).
#include "f64_tile.cuh"
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

// FP64: a persistent grid of CTAs strides over the tiles (f64_tile.cuh), tiles down the columns
// of C first.  CTA b runs on SM b mod SMs (CTAs are placed one per SM in turn), so every SM gets
// the same number of tiles, or one fewer; with one CTA per tile the SMs that finished a round
// first took several tiles of the next at once (1024^3 on 32 x 32 tiles: 5 to 10 tiles an SM).
template <bool ONTO>
__global__ void __launch_bounds__(F64_THREADS, F64_CTAS)
    f64_gemm_kernel(int64_t M, int64_t N, int64_t K, double alpha, double beta, const double* __restrict__ A,
                    int64_t ars, int64_t aks, const double* __restrict__ B, int64_t bks, int64_t bcs,
                    double* __restrict__ C, int64_t ldc, int bm, int bn, unsigned tiles_m, unsigned tiles) {
  __shared__ __align__(16) double smem[F64_SMEM_ELEMS];
  const bool unit = alpha == 1.0 && beta == 0.0;
  for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned tn = t / tiles_m, tm = t - tn * tiles_m;
    const int64_t m0 = static_cast<int64_t>(tm) * bm, n0 = static_cast<int64_t>(tn) * bn;
    const int r = static_cast<int>(M - m0 < bm ? M - m0 : bm), c = static_cast<int>(N - n0 < bn ? N - n0 : bn);
    f64_tile_any<ONTO>(r, c, K, A + m0 * ars, ars, aks, B + n0 * bcs, bks, bcs, alpha, beta, unit, C + m0 + n0 * ldc,
                       ldc, static_cast<int>(t ^ (t >> 2)), smem);
    __syncthreads();   // the next tile reuses the shared panels
  }
}

// Tile extents of an FP64 product: the ones whose busiest SM has the least to do, in DFMA units
// (32 elements) of one of its four partitions:
//   ceil(tiles / SMs) * (ceil(units per tile / 4) + 0.05 + 8 / K)
// where the constants are a tile's barriers, first loads and stores (about 8 k of one unit).  One
// tile per SM leaves a partition with one warp, whose operand reads nothing hides: measured 1.42x
// the pipe time at 256^3 (47.6 us), against 1.06x with two tiles (35.7 us) and more.  Candidates:
// 32 x 32, 32 x 16, 16 x 16, 16 x 8 and 8 x 8, and 64 x 16 and 64 x 8, each fitted to the matrix
// (bm = ceil(M / ceil(M / 32)), ...); the first on a tie.
static void native_f64_tile(int64_t M, int64_t N, int64_t K, int sms, int* bm, int* bn) {
  static const int shapes[][2] = {{32, 32}, {32, 16}, {16, 16}, {64, 16}, {64, 8}, {16, 8}, {8, 8}};
  const double per_tile = 0.05 + 8.0 / static_cast<double>(K);
  double best = 0.0;
  *bm = 0;
  for (const auto& sh : shapes) {
    const int64_t tm = (M + sh[0] - 1) / sh[0], tn = (N + sh[1] - 1) / sh[1];
    const int fm = static_cast<int>((M + tm - 1) / tm), fn = static_cast<int>((N + tn - 1) / tn);
    const int64_t waves = (tm * tn + sms - 1) / sms;
    const double cost = static_cast<double>(waves) * (static_cast<double>((fm * fn + 127) / 128) + per_tile) *
                        (waves == 1 ? 1.42 : waves == 2 ? 1.06 : 1.0);
    if (*bm == 0 || cost < best) {
      best = cost;
      *bm = fm;
      *bn = fn;
    }
  }
}

template <bool ONTO>
static int launch_f64(int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t ars, int64_t aks,
                      const double* B, int64_t bks, int64_t bcs, double beta, double* C, int64_t ldc, int sms,
                      cudaStream_t s) {
  if ((M + 63) / 64 > 0x7FFFFFFF || (N + 63) / 64 > 65535) return GB_ERR_UNSUPPORTED;
  int bm, bn;
  native_f64_tile(M, N, K, sms, &bm, &bn);
  const int64_t tiles_m = (M + bm - 1) / bm, tiles = tiles_m * ((N + bn - 1) / bn);
  if (tiles > 0x7FFFFFFF) return GB_ERR_UNSUPPORTED;
  const int64_t cap = static_cast<int64_t>(F64_CTAS) * sms;
  GB_LAUNCH(GB_KERNEL_NATIVE_GEMM, s,
            (f64_gemm_kernel<ONTO><<<static_cast<unsigned>(tiles < cap ? tiles : cap), F64_THREADS, 0, s>>>(
                M, N, K, alpha, beta, A, ars, aks, B, bks, bcs, C, ldc, bm, bn, static_cast<unsigned>(tiles_m),
                static_cast<unsigned>(tiles))));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

int native_kernel_onto_f64(int64_t M, int64_t N, int64_t K, const double* A, int64_t lda, const double* B,
                           int64_t ldb, double* C, int64_t ldc, int sms, cudaStream_t s) {
  if (M == 0 || N == 0 || K == 0) return GB_OK;   // an empty chain leaves D as it is
  return launch_f64<true>(M, N, K, 1.0, A, 1, lda, B, 1, ldb, 0.0, C, ldc, sms, s);
}

int native_gemm_f64(int ta, int tb, int64_t M, int64_t N, int64_t K, double alpha, const double* A,
                    int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc, int sms,
                    cudaStream_t s) {
  if (M == 0 || N == 0) return GB_OK;
  if (alpha == 0.0 || K == 0) return launch_scale<double>(M, N, beta, C, ldc, s);
  return launch_f64<false>(M, N, K, alpha, A, ta ? lda : 1, ta ? 1 : lda, B, tb ? ldb : 1, tb ? 1 : ldb, beta, C,
                           ldc, sms, s);
}

}  // namespace gb
