// Adjoint of gemm!: dA = dC * B^T and dB = A^T * dC in ONE tcgen05 launch (FP32 in/out).
//
// No reference counterpart: this is the pullback a ChainRulesCore rrule for jBLAS's
// jmul!/gemm! (src/gemm.jl:244) returns.  Products use the 3xBF16 split: every FP32 value
// x is held as hi = bf16(x), lo = bf16(x - hi), and
//   x*y ~= hi_x*hi_y + hi_x*lo_y + lo_x*hi_y      (lo_x*lo_y, below 2^-16 |xy|, is dropped)
// accumulated in FP32 in TMEM: three plane pairs of one group of the slice-product engine.
//
// Operand planes (K-major BF16, two planes each: hi, lo):
//   dA = dC * B^T   left  dC as [p][i][j]   (transposed from column-major dC)
//                   right B  as [p][k][j]   (transposed from column-major B)
//   dB = A^T * dC   left  A  as [p][k][i]   (A's columns are already contiguous in i)
//                   right dC as [p][j][i]   (dC's columns are already contiguous in i)
// dC is read from memory once: one kernel writes both of its plane layouts.
#include <cuda_bf16.h>

#include <cstring>

#include "gb_common.cuh"
#include "profile.cuh"
#include "split_terms.cuh"
#include "tc_gemm.cuh"

namespace gb {

// x = t_0 + t_1 (+ t_2) in BF16 terms: t_0 = bf16(x), t_1 = bf16(x - t_0), t_2 = bf16(x - t_0 - t_1).
// Each difference is exact in FP32 (it keeps the lower bits of x), so with three terms the sum is
// x exactly (24 = 3 x 8 significand bits, barring underflow); with two, |x - t_0 - t_1| <= 2^-17 |x|.
template <int NT>
__device__ __forceinline__ void split_terms(float x, uint32_t (&t)[NT]) {
  float r = x;
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const __nv_bfloat16 b = __float2bfloat16_rn(r);
    t[i] = static_cast<uint32_t>(__bfloat16_as_ushort(b));
    r -= __bfloat162float(b);
  }
}

// The term planes of up to three operands in one launch, each operand's blocks in turn.  Bound by memory:
// 4 bytes read and 2 NT written an element.  An operand alone is 8 to 15 us of a mid-size product, much
// of it the launch and the last wave.
//   chunks   (element (r, k) at X[r rs + k ks], any strides): a thread takes 8 consecutive k of a
//            row, a 16-byte store per plane, or 16 where k is contiguous and every row aligned (four
//            16-byte loads; 8 there: 190 us instead of 185 for a product whose split is 40); tpr =
//            2^log_tpr threads along k (as many as a row has chunks, at most 256), the other
//            256 / tpr along rows.  An unaligned row costs a warp 8 lines per load, 16 with 16 k a
//            thread, and a row to a block left half the threads of 2047 k idle.
//   tile     (rows contiguous): a 64 x 64 tile through shared memory.  Warp w loads columns
//            8w..8w+7 (lanes along r: 128-byte loads); a thread then splits 16 k of one row and
//            stores 32 bytes of every plane, and for the transposed planes 16 rows of one k (whole
//            lines in both layouts).  The terms stay in registers; keeping them in shared memory
//            for both layouts cost 48 conflicting 2-byte stores a thread.
// 3001 x 2047 and 2047 x 2503, three terms: 16 + 15.5 us in two launches, 22 us in one.
struct SplitPart {
  SplitOperand op;
  uint32_t first;   // first block
  uint32_t gx;      // chunks: blocks along k; tile: blocks along the rows
  int32_t log_tpr, tile;
  int32_t wide;     // chunks of 16
};
struct SplitParts {
  SplitPart part[SPLIT_MAX_OPERANDS];
  unsigned int* zero;   // written by block 0
  int32_t nzero;
};

// N consecutive values -> 2 N bytes of each of NT planes at dst + i plane (the first nvalid of them).
template <int NT, int N>
__device__ __forceinline__ void store_terms(const float (&x)[N], __nv_bfloat16* dst, int64_t plane, int nvalid) {
  uint32_t packed[NT][N / 2];
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    uint32_t t0[NT], t1[NT];
    split_terms<NT>(x[j], t0);
    split_terms<NT>(x[j + 1], t1);
#pragma unroll
    for (int i = 0; i < NT; ++i) packed[i][j / 2] = t0[i] | (t1[i] << 16);
  }
  if (nvalid == N) {
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      uint4* d4 = reinterpret_cast<uint4*>(dst + i * plane);
#pragma unroll
      for (int q = 0; q < N / 8; ++q)
        d4[q] = make_uint4(packed[i][4 * q], packed[i][4 * q + 1], packed[i][4 * q + 2], packed[i][4 * q + 3]);
    }
  } else {   // unrolled with a predicate: the packed terms stay in registers
    unsigned short* d2 = reinterpret_cast<unsigned short*>(dst);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (j < nvalid) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
          d2[i * plane + j] = static_cast<unsigned short>(packed[i][j / 2] >> (16 * (j & 1)));
      }
    }
  }
}

template <int NT, int N>
__device__ __forceinline__ void split_chunks(const SplitPart& p, uint32_t block) {
  const SplitOperand& o = p.op;
  const uint32_t by = block / p.gx, bx = block - by * p.gx;
  const int lt = p.log_tpr;
  const int64_t r = (static_cast<int64_t>(by) << (8 - lt)) + (threadIdx.x >> lt);
  const int64_t k0 = ((static_cast<int64_t>(bx) << lt) + (threadIdx.x & ((1 << lt) - 1))) * N;
  if (r >= o.R || k0 >= o.K) return;
  const int nvalid = static_cast<int>(o.K - k0 < N ? o.K - k0 : N);
  const float* __restrict__ src = o.X + r * o.rs + k0 * o.ks;
  float x[N];
  if (o.ks == 1 && nvalid == N && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
      const float4 v = reinterpret_cast<const float4*>(src)[q];
      x[4 * q] = v.x;
      x[4 * q + 1] = v.y;
      x[4 * q + 2] = v.z;
      x[4 * q + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = (j < nvalid) ? src[j * o.ks] : 0.0f;
  }
  store_terms<NT>(x, o.planes + r * o.pitch + k0, o.R * o.pitch, nvalid);
}

template <int NT>
__device__ __forceinline__ void split_tile(const SplitPart& p, uint32_t block, float (&tile)[64][65]) {
  const SplitOperand& o = p.op;
  const uint32_t by = block / p.gx, bx = block - by * p.gx;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t r0 = static_cast<int64_t>(bx) * 64, k0 = static_cast<int64_t>(by) * 64;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int kk = w * 8 + c;
    const int64_t k = k0 + kk;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int rr = lane + 32 * h;
      const int64_t r = r0 + rr;
      tile[kk][rr] = (r < o.R && k < o.K) ? o.X[r + k * o.ks] : 0.0f;
    }
  }
  __syncthreads();
  const int line = tid >> 2, at = (tid & 3) * 16;   // this thread's row (k row) and 16-wide chunk
  float x[16];
  if (r0 + line < o.R && k0 + at < o.K) {   // planes [r][k]
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = tile[at + j][line];
    const int64_t left = o.K - k0 - at;
    store_terms<NT>(x, o.planes + (r0 + line) * o.pitch + k0 + at, o.R * o.pitch, static_cast<int>(left < 16 ? left : 16));
  }
  if (o.planes_t && k0 + line < o.K && r0 + at < o.R) {   // planes [k][r]
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = tile[line][at + j];
    const int64_t left = o.R - r0 - at;
    store_terms<NT>(x, o.planes_t + (k0 + line) * o.pitch_t + r0 + at, o.K * o.pitch_t,
                    static_cast<int>(left < 16 ? left : 16));
  }
}

template <int NT>
__global__ void __launch_bounds__(256) split_terms_kernel(const __grid_constant__ SplitParts parts) {
  __shared__ float tile[64][65];   // [k][r]
  if (blockIdx.x == 0)
    for (int z = threadIdx.x; z < parts.nzero; z += 256) parts.zero[z] = 0;
  int i = 0;
#pragma unroll
  for (int q = 1; q < SPLIT_MAX_OPERANDS; ++q)
    if (blockIdx.x >= parts.part[q].first) i = q;
  const SplitPart& p = parts.part[i];
  const uint32_t block = blockIdx.x - p.first;
  if (p.tile) split_tile<NT>(p, block, tile);
  else if (p.wide) split_chunks<NT, 16>(p, block);
  else split_chunks<NT, 8>(p, block);
}

int split_bf16_terms(const SplitOperand* ops, int count, int nterms, unsigned int* zero, int nzero, int kind,
                     cudaStream_t s) {
  if ((nterms != 2 && nterms != 3) || count < 0 || count > SPLIT_MAX_OPERANDS) return GB_ERR_INVALID_VALUE;
  SplitParts parts;
  std::memset(&parts, 0, sizeof(parts));
  parts.zero = zero;
  parts.nzero = nzero;
  int64_t blocks = 0;
  for (int i = 0; i < SPLIT_MAX_OPERANDS; ++i) {
    SplitPart& p = parts.part[i];
    p.first = static_cast<uint32_t>(blocks);
    p.gx = 1;
    if (i >= count || ops[i].R <= 0 || ops[i].K <= 0) {
      // no blocks; one past the last is never reached, and an empty operand before a full one
      // starts where that one does
      continue;
    }
    const SplitOperand& o = ops[i];
    p.op = o;
    if (o.planes_t && o.rs != 1) return GB_ERR_UNSUPPORTED;   // the transposed layout is written from row-contiguous X
    int64_t n;
    if (o.rs == 1) {
      const int64_t ktiles = (o.K + 63) / 64, rtiles = (o.R + 63) / 64;
      if (ktiles > 65535 || rtiles > 0x7FFFFFFF) return GB_ERR_UNSUPPORTED;
      p.tile = 1;
      p.gx = static_cast<uint32_t>(rtiles);
      n = rtiles * ktiles;
    } else {
      p.wide = o.ks == 1 && (o.rs & 3) == 0 && (reinterpret_cast<uintptr_t>(o.X) & 15) == 0;
      const int64_t each = p.wide ? 16 : 8, chunks = (o.K + each - 1) / each;
      while (p.log_tpr < 8 && (1 << p.log_tpr) < chunks) ++p.log_tpr;
      const int64_t gx = (chunks + (1 << p.log_tpr) - 1) >> p.log_tpr, rows = 256 >> p.log_tpr;
      p.gx = static_cast<uint32_t>(gx);
      n = gx * ((o.R + rows - 1) / rows);
    }
    blocks += n;
    if (blocks > 0x7FFFFFFF) return GB_ERR_UNSUPPORTED;
  }
  if (blocks == 0) return GB_OK;
  const unsigned grid = static_cast<unsigned>(blocks);
  if (nterms == 2)
    GB_LAUNCH(kind, s, split_terms_kernel<2><<<grid, 256, 0, s>>>(parts));
  else
    GB_LAUNCH(kind, s, split_terms_kernel<3><<<grid, 256, 0, s>>>(parts));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

static inline int64_t pitch64(int64_t k) { return ((k + 63) / 64) * 64; }
static inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Schedule of the 3xBF16 product: one group, pairs (hi,hi), (hi,lo), (lo,hi).
static void split3_schedule(SliceSchedule& S, int kb_chunk) {
  std::memset(&S, 0, sizeof(S));
  S.ngroups = 1;
  S.kb_chunk = kb_chunk;
  S.bits = 0;
  S.level[0] = 0;
  S.npairs[0] = 3;
  S.pair_off[0] = 0;
  S.pp[0] = 0; S.pq[0] = 0;
  S.pp[1] = 0; S.pq[1] = 1;
  S.pp[2] = 1; S.pq[2] = 0;
}

// Workspace layout for an adjoint of A (M x K), B (K x N), dC (M x N).
static TcSplit adjoint_split(int64_t M, int64_t N, int64_t K, int sms) {
  auto t = [](int64_t x) { return (x + 255) / 256; };
  return tc_split_plan({t(M) * t(K), t(K) * t(N)}, {(N + TC_BK - 1) / TC_BK, (M + TC_BK - 1) / TC_BK}, 3, sms / 2);
}

size_t adjoint_workspace_bytes(int64_t M, int64_t N, int64_t K, int sms, bool split) {
  const int64_t pN = pitch64(N), pM = pitch64(M);
  const TcSplit sp = split ? adjoint_split(M, N, K, sms) : TcSplit();
  return al256(2 * static_cast<size_t>(M) * pN * 2) + al256(2 * static_cast<size_t>(K) * pN * 2) +
         al256(2 * static_cast<size_t>(K) * pM * 2) + al256(2 * static_cast<size_t>(N) * pM * 2) + sp.ws_bytes +
         sp.counters * sizeof(unsigned int);
}

int adjoint_f32(int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B, int64_t ldb,
                const float* dC, int64_t lddc, float* dA, int64_t ldda, float* dB, int64_t lddb, void* ws, bool split,
                int sms, DeviceStatus* status, uint64_t wait_limit_ns, cudaStream_t s) {
  const int64_t pN = pitch64(N), pM = pitch64(M);
  char* w = static_cast<char*>(ws);
  __nv_bfloat16* P1 = reinterpret_cast<__nv_bfloat16*>(w);                      // dC [p][i][j]
  w += al256(2 * static_cast<size_t>(M) * pN * 2);
  __nv_bfloat16* P2 = reinterpret_cast<__nv_bfloat16*>(w);                      // B  [p][k][j]
  w += al256(2 * static_cast<size_t>(K) * pN * 2);
  __nv_bfloat16* P3 = reinterpret_cast<__nv_bfloat16*>(w);                      // A  [p][k][i]
  w += al256(2 * static_cast<size_t>(K) * pM * 2);
  __nv_bfloat16* P4 = reinterpret_cast<__nv_bfloat16*>(w);                      // dC [p][j][i]

  const SplitOperand ops[3] = {
      {dC, M, N, 1, lddc, P1, pN, P4, pM},        // column-major, rows i contiguous: [p][i][j] and [p][j][i]
      {B, K, N, 1, ldb, P2, pN, nullptr, 0},      // rows k contiguous: [p][k][j]
      {A, K, M, lda, 1, P3, pM, nullptr, 0}};     // A^T, rows k, contraction over i contiguous: [p][k][i]
  w += al256(2 * static_cast<size_t>(N) * pM * 2);
  const int64_t big = M > N ? (M > K ? M : K) : (N > K ? N : K);
  const TcTuning tune = tc_tuning_for(TC_KIND_ADJOINT, big, big);
  const bool pair = tune.engine == 2;
  const TcSplit sp = pair && split ? adjoint_split(M, N, K, sms) : TcSplit();
  unsigned int* counters = reinterpret_cast<unsigned int*>(w + sp.ws_bytes);
  int rc = split_bf16_terms(ops, 3, 2, counters, sp.counters, GB_KERNEL_ADJOINT_SPLIT, s);
  if (rc) return rc;

  CUtensorMap ta0, tb0, ta1, tb1;
  rc = make_plane_tmap(&ta0, P1, N, M, 2, pN, TC_BM);
  if (!rc) rc = make_plane_tmap(&tb0, P2, N, K, 2, pN, TC_BN);
  if (!rc) rc = make_plane_tmap(&ta1, P3, M, K, 2, pM, TC_BM);
  if (!rc) rc = make_plane_tmap(&tb1, P4, M, N, 2, pM, TC_BN);
  if (rc) return rc;

  const int64_t tbm = pair ? 256 : TC_BM, tbn = pair ? 256 : TC_BN;
  TcParams prm;
  std::memset(&prm, 0, sizeof(prm));
  prm.band = sp.parts ? TC_SPLIT_BAND : tune.band;
  TcProblem& P = prm.prob[0];   // dA (M x K), contraction N
  P.M = M; P.N = K; P.K = N;
  P.tiles_m = static_cast<int32_t>((M + tbm - 1) / tbm);
  P.tiles_n = static_cast<int32_t>((K + tbn - 1) / tbn);
  P.tile_begin = 0;
  P.kb_total = static_cast<int32_t>((N + TC_BK - 1) / TC_BK);
  P.nchunks = 1;
  P.C = dA; P.ldc = ldda;
  P.alpha = 1.0; P.beta = 0.0;
  TcProblem& Q = prm.prob[1];   // dB (K x N), contraction M
  Q.M = K; Q.N = N; Q.K = M;
  Q.tiles_m = static_cast<int32_t>((K + tbm - 1) / tbm);
  Q.tiles_n = static_cast<int32_t>((N + tbn - 1) / tbn);
  Q.tile_begin = P.tiles_m * P.tiles_n;
  Q.kb_total = static_cast<int32_t>((M + TC_BK - 1) / TC_BK);
  Q.nchunks = 1;
  Q.C = dB; Q.ldc = lddb;
  Q.alpha = 1.0; Q.beta = 0.0;
  prm.nprob = 2;
  prm.total_tiles = Q.tile_begin + Q.tiles_m * Q.tiles_n;
  prm.tws = nullptr;
  prm.status = status;
  prm.wait_limit_ns = wait_limit_ns;
  SliceSchedule sched;
  split3_schedule(sched, P.kb_total > Q.kb_total ? P.kb_total : Q.kb_total);
  if (pair) {
    CUtensorMap tb0h, tb1h;   // 128-row B boxes: each CTA of a pair loads half of the B tile
    rc = make_plane_tmap(&tb0h, P2, N, K, 2, pN, 128);
    if (!rc) rc = make_plane_tmap(&tb1h, P4, M, N, 2, pM, 128);
    if (rc) return rc;
    CUtensorMap tc0, tc1;
    prm.c_tma = (tune.tma_store && make_c_tmap_f32(&tc0, dA, M, K, ldda) && make_c_tmap_f32(&tc1, dB, K, N, lddb))
                    ? 1 : 0;
    const int64_t ctas = 2 * static_cast<int64_t>(prm.total_tiles), cap = sms & ~1;
    prm.split_first = sp.first;
    prm.split_parts = sp.parts;
    prm.split_ws = reinterpret_cast<float*>(w);
    prm.split_count = counters;
    return tc_gemm_pair_launch(TC_EPI_F32, ta0, tb0h, &ta1, &tb1h, sched, prm,
                               sp.parts ? 2 * sp.clusters : static_cast<int>(ctas < cap ? ctas : cap),
                               GB_KERNEL_ADJOINT_MMA, s,
                               prm.c_tma ? &tc0 : nullptr, prm.c_tma ? &tc1 : nullptr);
  }
  const int grid = prm.total_tiles < sms ? prm.total_tiles : sms;
  return tc_gemm_launch(TC_EPI_F32, ta0, tb0, &ta1, &tb1, sched, prm, grid, GB_KERNEL_ADJOINT_MMA, s);
}

}  // namespace gb
