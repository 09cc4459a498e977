// An FP64 product over the tiles of f64_tile.cuh: native GEMM (native_gemm.cu) and the FP64 semirings
// (semiring_f64.cu).
#pragma once
#include "f64_tile.cuh"
#include "gb_common.cuh"
#include "profile.cuh"

namespace gb {

// A persistent grid of CTAs strides over the tiles (f64_tile.cuh), tiles down the columns
// of C first; with one CTA per tile the SMs that finished a round first took several tiles of the next
// at once (1024^3 on 32 x 32 tiles: 5 to 10 tiles an SM).  The tiles left after whole rounds go to the
// CTAs from the second quarter of the grid on: a full grid's later quarters have one CTA on every SM
// but four, while its first 160 CTAs put three on each of those (CTAs 0, 72, 136 and 208 ran on one
// SM).  With the remainder on the first CTAs 1000 x 1000 x 100 (1024 tiles: 8 on the fullest SM, now
// 7) took 204.6 us, now 180.2; 500^3 253 -> 223, 2048 x 2048 x 256 1787 -> 1726, (min, +) 1024^3
// 2.13 -> 2.06 ms.
template <class Op>
__global__ void __launch_bounds__(F64_THREADS, F64_CTAS)
    f64_gemm_kernel(int64_t M, int64_t N, int64_t K, const Op op, const double* __restrict__ A, int64_t ars,
                    int64_t aks, const double* __restrict__ B, int64_t bks, int64_t bcs, double* __restrict__ C,
                    int64_t ldc, int bm, int bn, unsigned tiles_m, unsigned tiles) {
  __shared__ __align__(16) double smem[F64_SMEM_ELEMS];
  const unsigned skip = tiles > gridDim.x ? gridDim.x / F64_CTAS : 0;
  for (unsigned t = blockIdx.x + (blockIdx.x < skip ? gridDim.x : 0) - skip; t < tiles; t += gridDim.x) {
    const unsigned tn = t / tiles_m, tm = t - tn * tiles_m;
    const int64_t m0 = static_cast<int64_t>(tm) * bm, n0 = static_cast<int64_t>(tn) * bn;
    const int r = static_cast<int>(M - m0 < bm ? M - m0 : bm), c = static_cast<int>(N - n0 < bn ? N - n0 : bn);
    f64_tile_any(r, c, K, A + m0 * ars, ars, aks, B + n0 * bcs, bks, bcs, op, C + m0 + n0 * ldc, ldc,
                 static_cast<int>(t ^ (t >> 2)), smem);
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
inline void f64_tile_extents(int64_t M, int64_t N, int64_t K, int sms, int* bm, int* bn) {
  static const int shapes[][2] = {{32, 32}, {32, 16}, {16, 16}, {64, 16}, {64, 8}, {16, 8}, {8, 8}};
  const double per_tile = 0.05 + 8.0 / static_cast<double>(K > 0 ? K : 1);
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

// Enqueues the product; `which` names it for the profile.  M, N > 0.
template <class Op>
int launch_f64_gemm(int which, const Op& op, int64_t M, int64_t N, int64_t K, const double* A, int64_t ars, int64_t aks,
                    const double* B, int64_t bks, int64_t bcs, double* C, int64_t ldc, int sms, cudaStream_t s) {
  if ((M + 63) / 64 > 0x7FFFFFFF || (N + 63) / 64 > 65535) return GB_ERR_UNSUPPORTED;
  int bm, bn;
  f64_tile_extents(M, N, K, sms, &bm, &bn);
  const int64_t tiles_m = (M + bm - 1) / bm, tiles = tiles_m * ((N + bn - 1) / bn);
  if (tiles > 0x7FFFFFFF) return GB_ERR_UNSUPPORTED;
  const int64_t cap = static_cast<int64_t>(F64_CTAS) * sms;
  GB_LAUNCH(which, s,
            (f64_gemm_kernel<Op><<<static_cast<unsigned>(tiles < cap ? tiles : cap), F64_THREADS, 0, s>>>(
                M, N, K, op, A, ars, aks, B, bks, bcs, C, ldc, bm, bn, static_cast<unsigned>(tiles_m),
                static_cast<unsigned>(tiles))));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

}  // namespace gb
