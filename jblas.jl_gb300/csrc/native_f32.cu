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

// How an operand's panels are copied: 16 bytes at a time, 4 bytes along x (unaligned), or 4 along k.
enum F32Copy { COPY_16, COPY_4_X, COPY_4_K };
static F32Copy copy_of(const void* p, int64_t xs, int64_t ks) {
  if (xs != 1) return COPY_4_K;
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ks & 3) == 0 ? COPY_16 : COPY_4_X;
}

// The tile shapes and a time model of a product on each (cycles at 2 GHz), with n tiles on the fullest SM
// and so ceil(n / 4) warps on its fullest partition:
//   a k    max(alone, warp0 + warp ceil(n / 4)) and, with operands in 4-byte copies, their sum of copy n and
//          COPY_LATENCY more
//   once   fixed + tile n, where a tile's stores depend on whether C's rows are contiguous for the tile
//          (not with the operands' roles exchanged) and C is read
// Fitted to the times of 860 products on every shape, both ways round, packed and not (up to 4e10
// multiply-adds, an eighth of them in vectors of 8 to 128): the choice is within 2% of the best one on
// average, 5% faster than that of a model of full tiles and one cost per tile, whose misses were short K
// (256 x 4672 x 32 12.4 us on 64 x 64 tiles, 8.4 on 32 x 32) and long products with both operands in
// 4-byte copies (112 x 9081 x 3103 276 us, packed 230).  On 660 other products: 254 faster by more than 2%,
// 34 slower (at most 16%), 4.7% faster on average; 11 slower than on the register tiles of 4 x 4 to 8 x 8
// elements a thread that came before (at most 9%; 31, at most 19%, under that model).
enum F32Tile { T64X64, T32X32, T32X16 };
struct F32TileInfo {
  int bm, bn;
  double alone, warp0, warp;
  double copy[3];       // by F32Copy
  double fixed, tile[2][2];   // [roles exchanged][C read]
};
static const F32TileInfo kF32Tile[] = {
    {64, 64, 172, 0, 113, {0.0, 5.3, 10}, 6900, {{5500, 1100}, {5000, 9000}}},
    {32, 32, 93, 21, 39.7, {0.0, 1.5, 3.1}, 740, {{1100, 760}, {480, 4000}}},
    {32, 16, 52.6, 15.6, 26.5, {0.0, 1, 1.6}, 545, {{400, 760}, {210, 1470}}}};
constexpr double COPY_LATENCY = 13.4;
// The 32 x 16 tile with the longer side of C along its 16 columns reads that side's operand in half the
// width (36 x 8672 x 10813 520 us, the other way round 415).
constexpr double SHORT_ROWS = 1.107;
// Packing copies of `x` rows of K elements: read and write, and one more launch and the buffer's
// allocation, as much on the host as on the device.
constexpr double PACK_BYTES_PER_CYCLE = 1950, PACK_LAUNCH = 16500;

// The cost of a choice; of the tile's own time alone with packed operands.
static double f32_cost(F32Tile t, bool exchanged, int64_t M, int64_t N, int64_t K, F32Copy a, F32Copy b, bool reads_c,
                       int sms) {
  const F32TileInfo& i = kF32Tile[t];
  const int64_t tiles = ((M + i.bm - 1) / i.bm) * ((N + i.bn - 1) / i.bn);
  const int64_t n = (tiles + sms - 1) / sms;
  const double copies = i.copy[a] + i.copy[b], nd = static_cast<double>(n);
  const double per_k = std::max(i.alone, i.warp0 + i.warp * static_cast<double>((n + 3) / 4)) *
                           (t == T32X16 && M < N ? SHORT_ROWS : 1.0) +
                       (copies > 0.0 ? copies * nd + COPY_LATENCY : 0.0);
  return static_cast<double>(K) * per_k + i.fixed + i.tile[exchanged][reads_c] * nd;
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

// C^T = B^T A^T: the same chain (fma commutes), with the tile's rows along the columns of C.
static void exchange_roles(F32Args* g) {
  std::swap(g->M, g->N);
  std::swap(g->a, g->b);
  std::swap(g->ars, g->bcs);
  std::swap(g->aks, g->bks);
  std::swap(g->crs, g->ccs);
}

// Direct, on 4-byte copies of the operands that need them, or packed; either way round; on the shape that the
// model finds soonest.  Packing needs a buffer: under capture (no allocation in the graph), or when it
// cannot be had, the call takes the best direct choice.
template <class Op>
static int f32_run(F32Args g, const Op& op, bool reads_c, int sms, cudaMemPool_t pool, cudaStream_t s) {
  const int64_t K = g.K;
  struct Choice {
    double cost = 1e300;
    F32Tile tile = T32X32;
    bool exchanged = false;
  } direct, packed;
  const F32Copy ca = copy_of(g.a, g.ars, g.aks), cb = copy_of(g.b, g.bcs, g.bks);
  const double pack = PACK_LAUNCH + 8.0 / PACK_BYTES_PER_CYCLE * static_cast<double>(K) *
                                        static_cast<double>((ca != COPY_16 ? g.M : 0) + (cb != COPY_16 ? g.N : 0));
  for (int x = 0; x < 2; ++x) {
    for (F32Tile t : {T64X64, T32X32, T32X16}) {
      auto offer = [&](Choice* c, F32Copy a, F32Copy b, double more) {
        const double cost = (f32_cost(t, x, x ? g.N : g.M, x ? g.M : g.N, K, x ? b : a, x ? a : b, reads_c, sms) + more) *
                            (x ? 1.01 : 1.0);
        if (cost < c->cost) *c = Choice{cost, t, x != 0};
      };
      offer(&direct, ca, cb, 0.0);
      if (ca != COPY_16 || cb != COPY_16) offer(&packed, COPY_16, COPY_16, pack);
    }
  }
  if (packed.cost < direct.cost && pool && (K + PACK - 1) / PACK <= 65535) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    F32Args p = g;
    if (packed.exchanged) exchange_roles(&p);
    const bool pa = copy_of(p.a, p.ars, p.aks) != COPY_16, pb = copy_of(p.b, p.bcs, p.bks) != COPY_16;
    const int64_t la = pa ? (p.M + 127) / 128 * 128 : 0, lb = pb ? (p.N + 127) / 128 * 128 : 0;
    uint32_t* ws = nullptr;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone &&
        cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ws), static_cast<size_t>(la + lb) * K * 4, pool, s) ==
            cudaSuccess) {
      PackJob jobs[2];
      int n = 0;
      int64_t most = 0;
      auto job = [&](const uint32_t*& src, int64_t& xs, int64_t& ks, int64_t X, uint32_t* dst, int64_t ld, int& pad) {
        jobs[n++] = PackJob{src, xs, ks, X, dst, ld};
        most = std::max(most, X);
        src = dst;
        xs = 1;
        ks = ld;
        pad = 1;
      };
      if (pa) job(p.a, p.ars, p.aks, p.M, ws, la, p.pad_a);
      if (pb) job(p.b, p.bcs, p.bks, p.N, ws + la * K, lb, p.pad_b);
      const dim3 grid(static_cast<unsigned>((most + PACK - 1) / PACK), static_cast<unsigned>((K + PACK - 1) / PACK),
                      static_cast<unsigned>(n));
      GB_LAUNCH(GB_KERNEL_NATIVE_GEMM, s, (f32_pack_kernel<<<grid, 256, 0, s>>>(jobs[0], jobs[n - 1], K)));
      const int rc = launch_tile<false>(packed.tile, p, op, sms, s);
      cudaFreeAsync(ws, s);
      return rc;
    }
    cudaGetLastError();
  }
  if (direct.exchanged) exchange_roles(&g);
  return ca == COPY_16 && cb == COPY_16 ? launch_tile<false>(direct.tile, g, op, sms, s)
                                        : launch_tile<true>(direct.tile, g, op, sms, s);
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
  return f32_run(g, F32Chain{alpha, beta}, beta != 0.0f, sms, pool, s);
}

int native_kernel_onto_f32(int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B, int64_t ldb,
                           float* C, int64_t ldc, int sms, cudaMemPool_t pool, cudaStream_t s) {
  if (M == 0 || N == 0 || K == 0) return GB_OK;   // an empty chain leaves D as it is
  if ((M + 63) / 64 > 0x7FFFFFFF || (N + 63) / 64 > 65535) return GB_ERR_UNSUPPORTED;
  const F32Args g{M, N, K, reinterpret_cast<const uint32_t*>(A), 1, lda, reinterpret_cast<const uint32_t*>(B), 1, ldb,
                  reinterpret_cast<uint32_t*>(C), 1, ldc, 0, 0};
  return f32_run(g, F32Onto{}, true, sms, pool, s);
}

}  // namespace gb
