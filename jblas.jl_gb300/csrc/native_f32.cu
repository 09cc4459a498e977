// Native FP32 GEMM and kernel! on the CUDA cores: jmul!'s per-element FMA chain
// (src/gemm.jl:76-89, 154-168) on the packed tiles of simt4_tile.cuh.
//
// The accumulator starts at -0.0, so the first step fma(a1, x1, -0.0) equals the rounded product
// a1*x1 bit for bit; every tile shape, operand layout and packing runs the same chain.
//
// Measured in alternation with 128 x 128 / 64 x 64 scalar register tiles (FFMA peak 78 TFLOP/s):
// 256^3 16.6 -> 13 us a call, 1536^3 217 -> 172 us, 2048^3 404 -> 336 us, 4096^3 2.70 -> 2.31 ms,
// 4097 x 4095 x 4001 2.67 -> 2.30, 8192 x 8192 x 4096 10.4 -> 8.66 (63 TFLOP/s), 16384 x 64 x 16384
// 1.11 -> 0.88; kernel! at 2048^3 519 -> 369 us.
#include <algorithm>

#include "gb_common.cuh"
#include "native_gemm.cuh"
#include "profile.cuh"
#include "simt4_tile.cuh"

namespace gb {

// jBLAS's kernel! (src/kernels.jl:212-238): the chain starts from D's value and is stored as is.
struct F32Onto {
  static constexpr bool kInitFromC = true;
  static __device__ __forceinline__ uint32_t init() { return 0u; }
  static __device__ __forceinline__ pair4 step(pair4 acc, pair4 a, pair4 b) { return fma_f32x2(a, b, acc); }
  __device__ __forceinline__ bool reads_c() const { return false; }
  __device__ __forceinline__ uint32_t value(uint32_t acc) const { return acc; }
  __device__ __forceinline__ uint32_t value(uint32_t, uint32_t acc) const { return acc; }
};

// One product as the kernels take it: element (i, k) of A at a + i * ars + k * aks, (k, j) of B at
// b + k * bks + j * bcs, (i, j) of C at c + i * crs + j * ccs; pad_a / pad_b: the operand's buffer
// reaches whole tiles.
struct F32Args {
  int64_t M, N, K;
  const uint32_t* a;
  int64_t ars, aks;
  const uint32_t* b;
  int64_t bks, bcs;
  uint32_t* c;
  int64_t crs, ccs;
  int pad_a, pad_b;
};

// One CTA per SM of WARPS independent warps, each taking tiles of its own: with many small CTAs the
// hardware's placement decides which SMs get the last tiles (4097 x 4096 x 4096 on four-CTA SMs: 16
// tiles on some and 12 on others instead of 13 or 14, 2.77 ms instead of 2.43).  Warp w of CTA b
// takes tiles b + grid w, + grid WARPS, ..., rows of tiles first.
template <class S, bool ANY, int WARPS, class Op>
__global__ void __launch_bounds__(32 * WARPS, 1) f32_gemm_kernel(const F32Args g, const Op op, unsigned tiles_m,
                                                                 unsigned tiles) {
  extern __shared__ __align__(16) uint32_t s4_smem[];
  const unsigned warp = threadIdx.x >> 5;
  uint32_t* smem = s4_smem + warp * (S::SMEM_BYTES / 4);
  for (unsigned t = blockIdx.x + gridDim.x * warp; t < tiles; t += gridDim.x * WARPS) {
    const unsigned tn = t / tiles_m, tm = t - tn * tiles_m;
    const int64_t m0 = static_cast<int64_t>(tm) * S::BM, n0 = static_cast<int64_t>(tn) * S::BN;
    const int r = static_cast<int>(g.M - m0 < S::BM ? g.M - m0 : S::BM);
    const int c = static_cast<int>(g.N - n0 < S::BN ? g.N - n0 : S::BN);
    simt4_tile<S, ANY>(r, c, g.pad_a ? S::BM : r, g.pad_b ? S::BN : c, g.K, op, g.a + m0 * g.ars, g.ars, g.aks,
                       g.b + n0 * g.bcs, g.bks, g.bcs, g.c + m0 * g.crs + n0 * g.ccs, g.crs, g.ccs, smem);
  }
}

// The tile shapes, with what a rule on them needs: the cycles one k of a tile takes on an SM filled
// with such tiles, the least it takes alone, how slowly few tiles reach the full rate, and what an
// operand that is not x-contiguous and aligned costs (measured at 2 GHz on 256^3 to 4096^3).
enum F32Tile { T64X64, T32X32, T32X16 };
struct F32TileInfo {
  int bm, bn;
  double full, alone, few;
  double unpacked;   // share by which one operand in 4-byte copies slows the product
};
static const F32TileInfo kF32Tile[] = {
    {64, 64, 41.5, 196.0, 1.0, 0.06}, {32, 32, 12.6, 79.0, 1.5, 0.16}, {32, 16, 8.2, 60.0, 1.5, 0.16}};

// Time model (cycles) of an M x N x K product on one shape: n tiles on the busiest SM take
// max(alone, n full (1 + few / (n + 1))) cycles a k, and each some 600 for its first loads and stores.
static double f32_cost(F32Tile t, int64_t M, int64_t N, int64_t K, int sms) {
  const F32TileInfo& i = kF32Tile[t];
  const int64_t tiles = ((M + i.bm - 1) / i.bm) * ((N + i.bn - 1) / i.bn);
  const double n = static_cast<double>((tiles + sms - 1) / sms);
  const double per_k = std::max(i.alone, n * i.full * (1.0 + i.few / (n + 1.0)));
  return static_cast<double>(K) * per_k + 600.0 * n;
}

template <class S, bool ANY, int WARPS, class Op>
static int launch_shape(const F32Args& g, const Op& op, int sms, cudaStream_t s) {
  constexpr int SMEM = WARPS * S::SMEM_BYTES;
  static_assert(SMEM <= 232448, "shared memory per CTA");
  const int64_t tiles_m = (g.M + S::BM - 1) / S::BM, tiles = tiles_m * ((g.N + S::BN - 1) / S::BN);
  if (tiles > 0x7FFFFFFF) return GB_ERR_UNSUPPORTED;
  auto kernel = f32_gemm_kernel<S, ANY, WARPS, Op>;
  static std::atomic<unsigned long long> opted{0};
  const int rc = opt_in_dynamic_smem(kernel, SMEM, opted);
  if (rc) return rc;
  const unsigned grid = static_cast<unsigned>(tiles < sms ? tiles : sms);
  GB_LAUNCH(GB_KERNEL_NATIVE_GEMM, s, (kernel<<<grid, 32 * WARPS, SMEM, s>>>(g, op, static_cast<unsigned>(tiles_m),
                                                                            static_cast<unsigned>(tiles))));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

template <bool ANY, class Op>
static int launch_tile(F32Tile t, const F32Args& g, const Op& op, int sms, cudaStream_t s) {
  switch (t) {
    case T64X64: return launch_shape<S4Shape<16, 8>, ANY, 8>(g, op, sms, s);
    case T32X32: return launch_shape<S4Shape<8, 4>, ANY, 16>(g, op, sms, s);
    default: return launch_shape<S4Shape<8, 2>, true, 16>(g, op, sms, s);
  }
}

// Packing: copies of one or both operands with x contiguous, rows padded to whole tiles, as jBLAS's
// packing buffers were meant (src/memory_management.jl:78-177).  64 x 64 elements a CTA; a
// k-contiguous source is transposed through shared memory, an x-contiguous (unaligned) one is copied.
// Bound by memory: 27 us for a 4096 x 4096 operand (64 MiB read, 64 MiB written).
constexpr int PACK = 64;
struct PackJob {
  const uint32_t* src;   // element (x, k) at src + x * xs + k * ks; xs or ks is 1
  int64_t xs, ks, X;
  uint32_t* dst;         // element (x, k) at dst + k * ld + x
  int64_t ld;
};
__global__ void __launch_bounds__(256) f32_pack_kernel(const PackJob j0, const PackJob j1, int64_t K) {
  __shared__ uint32_t tile[PACK][PACK + 1];
  const PackJob& j = blockIdx.z ? j1 : j0;
  const int64_t x0 = static_cast<int64_t>(blockIdx.x) * PACK, k0 = static_cast<int64_t>(blockIdx.y) * PACK;
  if (x0 >= j.X) return;
  const int lane = threadIdx.x % PACK, row = threadIdx.x / PACK;   // 4 rows of 64 a step
  if (j.ks == 1) {
#pragma unroll
    for (int i = 0; i < PACK; i += 4)
      if (x0 + row + i < j.X && k0 + lane < K) tile[row + i][lane] = j.src[(x0 + row + i) * j.xs + k0 + lane];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PACK; i += 4)
      if (x0 + lane < j.X && k0 + row + i < K) j.dst[(k0 + row + i) * j.ld + x0 + lane] = tile[lane][row + i];
  } else {
#pragma unroll
    for (int i = 0; i < PACK; i += 4)
      if (x0 + lane < j.X && k0 + row + i < K)
        j.dst[(k0 + row + i) * j.ld + x0 + lane] = j.src[x0 + lane + (k0 + row + i) * j.ks];
  }
}

static bool x_aligned(const void* p, int64_t xs, int64_t ks) {
  return xs == 1 && (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ks & 3) == 0;
}

// Estimated cost in cycles of packing `x` rows of K elements: read and write at about 4 TB/s.
static double pack_cost(int64_t x, int64_t K) { return 8.0 * static_cast<double>(x) * static_cast<double>(K) / 4e12 * 2e9; }
// One more launch and the buffer's allocation, as much on the host as on the device.
constexpr double PACK_LAUNCH = 9e-6 * 2e9;

template <class Op>
static int f32_run(F32Args g, const Op& op, int sms, cudaMemPool_t pool, cudaStream_t s) {
  const int64_t M = g.M, N = g.N, K = g.K;
  // The 32 x 16 tile is taller than wide: a product of few rows runs with the operands' roles
  // exchanged, C^T = B^T A^T (the same chain; fma commutes), where that is cheaper.
  auto best_of = [&](int64_t m, int64_t n, F32Tile* t) {
    double best = 1e300;
    for (F32Tile c : {T64X64, T32X32, T32X16}) {
      const double cost = f32_cost(c, m, n, K, sms);
      if (cost < best) best = cost, *t = c;
    }
    return best;
  };
  F32Tile tile = T32X32, tile_x = T32X32;
  double direct = best_of(M, N, &tile);
  const double exchanged = best_of(N, M, &tile_x);
  if (exchanged < 0.97 * direct) {
    std::swap(g.M, g.N);
    std::swap(g.a, g.b);
    std::swap(g.ars, g.bcs);
    std::swap(g.aks, g.bks);
    std::swap(g.crs, g.ccs);
    direct = exchanged;
    tile = tile_x;
  }
  // Direct, on 4-byte copies of an operand that needs them, or packed, whichever the model finds
  // cheaper: packing costs two passes over an operand and a launch, and pays from about 800 rows and
  // columns up (4097 x 4095 x 4001 2.77 -> 2.40 ms; 1024^3 with both k-contiguous 77 -> 69 us).
  const bool va = x_aligned(g.a, g.ars, g.aks), vb = x_aligned(g.b, g.bcs, g.bks);
  const double penalty = kF32Tile[tile].unpacked * ((va ? 0 : 1) + (vb ? 0 : 1));
  if (tile != T32X16 &&
      (va && vb ? 0.0 : PACK_LAUNCH + pack_cost((va ? 0 : g.M) + (vb ? 0 : g.N), K)) <= penalty * direct) {
    uint32_t* ws = nullptr;
    const int64_t la = va ? 0 : (g.M + 127) / 128 * 128, lb = vb ? 0 : (g.N + 127) / 128 * 128;
    bool ready = va && vb;
    if (!ready && pool && (K + PACK - 1) / PACK <= 65535) {
      // under capture the call keeps to the direct path (no allocation in the graph); so it does when
      // the workspace cannot be had
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone &&
          cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ws), static_cast<size_t>(la + lb) * K * 4, pool, s) ==
              cudaSuccess) {
        PackJob jobs[2];
        int n = 0;
        int64_t most = 0;
        auto pack = [&](const uint32_t*& p, int64_t& xs, int64_t& ks, int64_t X, uint32_t* dst, int64_t ld, int& pad) {
          jobs[n++] = PackJob{p, xs, ks, X, dst, ld};
          most = std::max(most, X);
          p = dst;
          xs = 1;
          ks = ld;
          pad = 1;
        };
        if (!va) pack(g.a, g.ars, g.aks, g.M, ws, la, g.pad_a);
        if (!vb) pack(g.b, g.bcs, g.bks, g.N, ws + la * K, lb, g.pad_b);
        const dim3 grid(static_cast<unsigned>((most + PACK - 1) / PACK), static_cast<unsigned>((K + PACK - 1) / PACK),
                        static_cast<unsigned>(n));
        GB_LAUNCH(GB_KERNEL_NATIVE_GEMM, s, (f32_pack_kernel<<<grid, 256, 0, s>>>(jobs[0], jobs[n - 1], K)));
        ready = true;
      } else {
        cudaGetLastError();
      }
    }
    if (ready) {
      const int rc = launch_tile<false>(tile, g, op, sms, s);
      if (ws) cudaFreeAsync(ws, s);
      return rc;
    }
  }
  return launch_tile<true>(tile, g, op, sms, s);
}

int native_gemm_f32(int ta, int tb, int64_t M, int64_t N, int64_t K, float alpha, const float* A, int64_t lda,
                    const float* B, int64_t ldb, float beta, float* C, int64_t ldc, int sms, cudaMemPool_t pool,
                    cudaStream_t s) {
  if (M == 0 || N == 0) return GB_OK;
  if (alpha == 0.0f || K == 0) return native_scale_f32(M, N, beta, C, ldc, s);
  if ((M + 127) / 128 > 0x7FFFFFFF || (N + 127) / 128 > 65535) return GB_ERR_UNSUPPORTED;
  const F32Args g{M, N, K, reinterpret_cast<const uint32_t*>(A), ta ? lda : 1, ta ? 1 : lda,
                  reinterpret_cast<const uint32_t*>(B), tb ? ldb : 1, tb ? 1 : ldb, reinterpret_cast<uint32_t*>(C), 1,
                  ldc, 0, 0};
  return f32_run(g, F32Chain{alpha, beta}, sms, pool, s);
}

int native_kernel_onto_f32(int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B, int64_t ldb,
                           float* C, int64_t ldc, int sms, cudaMemPool_t pool, cudaStream_t s) {
  if (M == 0 || N == 0 || K == 0) return GB_OK;   // an empty chain leaves D as it is
  if ((M + 63) / 64 > 0x7FFFFFFF || (N + 63) / 64 > 65535) return GB_ERR_UNSUPPORTED;
  const F32Args g{M, N, K, reinterpret_cast<const uint32_t*>(A), 1, lda, reinterpret_cast<const uint32_t*>(B), 1, ldb,
                  reinterpret_cast<uint32_t*>(C), 1, ldc, 0, 0};
  return f32_run(g, F32Onto{}, sms, pool, s);
}

}  // namespace gb
