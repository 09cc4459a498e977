// Tile of C for 4-byte elements on the CUDA cores, for native and grouped FP32: register tiles
// on packed pairs of rows.
//
// What bounds it: with one multiply-add per instruction the FMA pipe (one warp instruction per
// clock and SM partition) shares its issue slots with shared-memory reads and address arithmetic;
// the earlier 8 x 8 register tile with 4-byte loads issued on 83% of the cycles, 78% of it FMAs.
// fma.rn.f32x2 and add.rn.f32x2 do two rows per issue slot at the same pipe rate (each half rounds
// as the scalar operation, so results keep their bits), which leaves half of the slots for the
// rest; what remains is register and shared-memory ports (a register-only loop of packed FMAs with
// distinct operands measured 81% of the scalar peak).  Hence:
//  - a pair is two consecutive rows: A's rows lie side by side in shared memory and are read as
//    pairs; B's element is duplicated in registers (two moves for 4 or 8 packed operations);
//  - up to 16 x 8 elements a thread, so that a k takes 6 16-byte reads for 64 packed operations,
//    and natively a tile is one warp's alone: nothing waits at a barrier
//    (two warps a tile: 38 TFLOP/s on 16384 x 64 x 16384, one: 40);
//  - panels come through cp.async: 16 bytes a copy where rows are contiguous and aligned, else 4 (any
//    alignment, either orientation), S4_STAGES - 1 panels ahead, without bounds checks inside the
//    matrix;
//  - the code stays small, as every warp fetches it at a place of its own: the k loop is unrolled by
//    8 (by 16, 128 x 128 tiles fell from 49 to 34 TFLOP/s in the scalar form), and the 64 x 64 tile
//    loads its panels from one place (with the first panels' loads written out before the loop,
//    8192 x 8192 x 4096 took 9.0 ms instead of 8.6; the smaller tiles are the faster for it).
// C has a row and a column stride, so a caller may exchange the operands' roles (C^T = B^T A^T).
// Measured (native FP32, in alternation with the 8 x 8 scalar tile): see native_f32.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "f64_tile.cuh"   // cp.async helpers

namespace gb {

constexpr int S4_BK = 16;
constexpr int S4_STAGES = 3;

__device__ __forceinline__ void cp_async_4(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}

// Two 32-bit elements in one 64-bit register pair: rows i (low) and i + 1 (high).
using pair4 = uint64_t;
__device__ __forceinline__ pair4 pack4(uint32_t lo, uint32_t hi) {
  pair4 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ uint32_t lo4(pair4 v) { return static_cast<uint32_t>(v); }
__device__ __forceinline__ uint32_t hi4(pair4 v) { return static_cast<uint32_t>(v >> 32); }
__device__ __forceinline__ pair4 fma_f32x2(pair4 a, pair4 b, pair4 c) {
  pair4 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// Tile of WM x WN warps, each 4 x 8 lanes of TM x TN elements.
template <int TM_, int TN_, int WM_ = 1, int WN_ = 1>
struct S4Shape {
  static constexpr int TM = TM_, TN = TN_, WM = WM_, WN = WN_, THREADS = 32 * WM * WN;
  static constexpr int BM = WM * 4 * TM, BN = WN * 8 * TN;
  static constexpr int LDA = BM + 4, LDB = BN + 4;   // words; rows 16-byte aligned, k on distinct banks
  static constexpr int PANEL = S4_BK * (LDA + LDB);
  static constexpr int SMEM_BYTES = S4_STAGES * PANEL * 4;
  static_assert(TM % 4 == 0 && TN % 2 == 0, "vector operand reads");
  // A one-warp tile has other warps beside it, a larger one is its CTA's.
  static __device__ __forceinline__ int tid() { return THREADS == 32 ? threadIdx.x & 31 : threadIdx.x; }
  static __device__ __forceinline__ void sync() {
    if constexpr (THREADS == 32) __syncwarp();
    else __syncthreads();
  }
};

// One thread's share of an operand's panels: element (x, k), x < extent <= X, is src[x * xs + k * ks]
// and goes to word k * LD + x of the panel.  Three ways: XV four x a copy (xs = 1, aligned, full
// extent), XF the lanes along x, KF the lanes along k (8 k x 4 x a warp: distinct banks).  Without
// ANY the operand has xs = 1 and KF is not compiled (the code of the three ways and their registers
// cost the largest tile 5%).
template <int X, int LD, int THREADS, bool ANY>
struct S4Loader {
  static constexpr int UNROLL = X > 32 ? 8 : 16;
  static constexpr int XV = 0, XF = 1, KF = 2;
  static constexpr int VX = X / 4, VN = X * S4_BK / 4 / THREADS, VK = THREADS / VX;
  static constexpr int FX = X < THREADS ? X : THREADS, FNX = X / FX, FK = THREADS / FX, FN = S4_BK / FK;
  static constexpr int KX = THREADS / 8, KN = X / KX;
  static_assert(THREADS % VX == 0 && S4_BK % VK == 0 && X % FX == 0 && THREADS % FX == 0 && S4_BK % FK == 0 &&
                X % KX == 0, "panel loads");
  const uint32_t* p;
  int64_t str, adv, xstep;
  uint32_t dst;
  int way, x, k;

  __device__ __forceinline__ void init(const uint32_t* src, int64_t xs, int64_t ks, int extent, int tid) {
    way = (ANY && ks == 1 && xs != 1) ? KF
        : (xs == 1 && extent == X && (reinterpret_cast<uintptr_t>(src) & 15) == 0 && (ks & 3) == 0) ? XV : XF;
    x = way == XV ? tid % VX * 4 : way == XF ? tid % FX : tid / 8;
    k = way == XV ? tid / VX : way == XF ? tid / FX : tid % 8;
    p = src + x * xs + k * ks;
    str = way == XV ? VK * ks : way == XF ? FK * ks : KX * xs;
    xstep = ANY ? FX * xs : FX;
    adv = S4_BK * ks;
    dst = static_cast<uint32_t>(k * LD + x) * 4u;
  }

  // (loops unrolled in part: their code is fetched by warps at many different places)
  template <bool CHECK>
  __device__ __forceinline__ void copy(uint32_t d, int extent, int kc) {
    const uint32_t* q = p;
    if (way == XV) {
#pragma unroll UNROLL
      for (int l = 0; l < VN; ++l, q += str)
        if (!CHECK || k + l * VK < kc) cp_async_16(d + l * (VK * LD * 4), q);
    } else if (!ANY || way == XF) {
#pragma unroll UNROLL
      for (int l = 0; l < FN; ++l, q += str)
#pragma unroll
        for (int h = 0; h < FNX; ++h)
          if (!CHECK || (x + h * FX < extent && k + l * FK < kc)) cp_async_4(d + (l * FK * LD + h * FX) * 4, q + h * xstep);
    } else {
#pragma unroll UNROLL
      for (int l = 0; l < KN; ++l, q += str)
#pragma unroll
        for (int h = 0; h < S4_BK; h += 8)
          if (!CHECK || (x + l * KX < extent && k + h < kc)) cp_async_4(d + (h * LD + l * KX) * 4, q + h);
    }
  }
  // Loads the panel of kc k to the shared address `panel`.
  __device__ __forceinline__ void load(uint32_t panel, int extent, int kc) {
    if (extent == X && kc == S4_BK) copy<false>(panel + dst, extent, kc);
    else copy<true>(panel + dst, extent, kc);
    p += adv;
  }
};

// The r x c tile of C at C (its first element, strides crs and ccs), 1 <= r <= BM, 1 <= c <= BN;
// ra rows of A and cb columns of B are read (r and c, or the whole extents of padded operands).
// The arithmetic is a policy `Op` (an object, for its epilogue):
//   Op::init()                          an accumulator before k = 1 (or C's value, with Op::kInitFromC)
//   Op::step(acc, a, b)                 one k, on a pair of rows (b holds B's element twice)
//   op.reads_c(), op.value(c, acc), op.value(acc)   the element of C, from its old value or without
// k runs 1..K in order; no padded k is folded in.  Rows and columns past the edge compute on stale
// shared memory and are not stored.  A's element (i, k) is A[i * ars + k * aks], B's (k, j) is
// B[k * bks + j * bcs].  Run by S::THREADS threads in shared memory of their own: one warp, or (THREADS >
// 32) the whole CTA.
template <class S, bool ANY, class Op>
__device__ __forceinline__ void simt4_tile(int r, int c, int ra, int cb, int64_t K, const Op& op, const uint32_t* __restrict__ A,
                                           int64_t ars, int64_t aks, const uint32_t* __restrict__ B, int64_t bks,
                                           int64_t bcs, uint32_t* __restrict__ C, int64_t crs, int64_t ccs,
                                           uint32_t* smem) {
  constexpr int TM = S::TM, TN = S::TN, BK = S4_BK;
  constexpr int CV = TN % 4 == 0 ? 4 : 2;   // columns per shared-memory read
  const int tid = S::tid(), lane = tid & 31, warp = tid >> 5;
  const int row0 = (warp % S::WM) * 4 * TM + (lane >> 3) * 4;     // + 16 per four rows
  const int col0 = (warp / S::WM) * 8 * TN + (lane & 7) * CV;     // + 8 CV per CV columns
  // a warp whose part lies outside the tile only helps to load
  const bool idle = S::THREADS > 32 && ((warp % S::WM) * 4 * TM >= r || (warp / S::WM) * 8 * TN >= c);

  S4Loader<S::BM, S::LDA, S::THREADS, ANY> la;
  S4Loader<S::BN, S::LDB, S::THREADS, ANY> lb;
  la.init(A, ars, aks, ra, tid);
  lb.init(B, bcs, bks, cb, tid);
  const uint32_t smem_u = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int64_t panels = (K + BK - 1) / BK;
  pair4 acc[TM / 2][TN];
#pragma unroll
  for (int i = 0; i < TM / 2; ++i) {
    const int row = row0 + (i / 2) * 16 + (i % 2) * 2;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int col = col0 + (j / CV) * (8 * CV) + j % CV;
      uint32_t lo = Op::init(), hi = Op::init();
      if (Op::kInitFromC && col < c) {
        if (row < r) lo = C[row * crs + col * ccs];
        if (row + 1 < r) hi = C[(row + 1) * crs + col * ccs];
      }
      acc[i][j] = pack4(lo, hi);
    }
  }

  auto read = [&](const uint32_t* pa, const uint32_t* pb, int k, pair4 (&a)[TM / 2], uint32_t (&b)[TN]) {
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pa + k * S::LDA + row0 + i * 16);
      a[2 * i] = v.x;
      a[2 * i + 1] = v.y;
    }
#pragma unroll
    for (int j = 0; j < TN; j += CV) {
      const uint32_t* q = pb + k * S::LDB + col0 + j * 8;
      if constexpr (CV == 4) {
        const uint4 v = *reinterpret_cast<const uint4*>(q);
        b[j] = v.x;
        b[j + 1] = v.y;
        b[j + 2] = v.z;
        b[j + 3] = v.w;
      } else {
        const uint2 v = *reinterpret_cast<const uint2*>(q);
        b[j] = v.x;
        b[j + 1] = v.y;
      }
    }
  };
  auto step = [&](const pair4 (&a)[TM / 2], const uint32_t (&b)[TN]) {
#pragma unroll
    for (int j = 0; j < TN; ++j) {   // B's operand stays for TM / 2 operations
      const pair4 bb = pack4(b[j], b[j]);
#pragma unroll
      for (int i = 0; i < TM / 2; ++i) acc[i][j] = Op::step(acc[i][j], a[i], bb);
    }
  };

  int stage = 0, load_stage = 0;
  auto load = [&](int64_t q) {   // panels are loaded in order
    const int64_t left = K - q * BK;
    const int kc = static_cast<int>(left < BK ? left : BK);
    const uint32_t dst = smem_u + static_cast<uint32_t>(load_stage * (S::PANEL * 4));
    la.load(dst, ra, kc);
    lb.load(dst + BK * S::LDA * 4, cb, kc);
    load_stage = (load_stage + 1) % S4_STAGES;
  };
  // Panel q is loaded S4_STAGES - 1 panels before it is used.  The largest tile's copies are written
  // out in one place only, the others' also before the loop (see above).
  int64_t q = 0;
  if constexpr (TM <= 8) {
#pragma unroll
    for (; q < S4_STAGES - 1; ++q) {
      if (q < panels) load(q);
      cp_async_commit();
    }
  }
  for (; q < panels + S4_STAGES - 1; ++q) {
    cp_async_wait<S4_STAGES - 2>();   // panel q - (S4_STAGES - 1), the oldest but S4_STAGES - 2, is in place
    S::sync();                        // for every thread, and all have left the stage to be loaded
    if (q < panels) load(q);
    cp_async_commit();
    const int64_t p = q - (S4_STAGES - 1);
    if (p < 0) continue;
    const uint32_t* pa = smem + stage * S::PANEL;
    const uint32_t* pb = pa + BK * S::LDA;
    stage = (stage + 1) % S4_STAGES;
    const int64_t left = K - p * BK;
    pair4 a0[TM / 2], a1[TM / 2];
    uint32_t b0[TN], b1[TN];
    if (idle) {
    } else if (left >= BK) {
      read(pa, pb, 0, a0, b0);
#pragma unroll 4
      for (int k = 0; k < BK; k += 2) {   // the next k's operands are read before this one's FMAs
        read(pa, pb, k + 1, a1, b1);
        step(a0, b0);
        read(pa, pb, k + 2 < BK ? k + 2 : 0, a0, b0);
        step(a1, b1);
      }
    } else {
      for (int k = 0; k < static_cast<int>(left); ++k) {
        read(pa, pb, k, a0, b0);
        step(a0, b0);
      }
    }
  }
  cp_async_wait<0>();   // (only empty groups are left)
  S::sync();            // the next tile reuses the stages
  if (idle) return;

  // A column of the lane's rows at a time: C's old values, where the epilogue reads them, are all
  // requested before the first is used (one at a time cost 2% at 4096^3).
  const bool rc = op.reads_c();
  // (opaque to the compiler, which would otherwise keep the addresses of the first loads of C alive
  // through the k loop: kernel! at 1024^3 then spilled, 94 us against 70)
  if constexpr (Op::kInitFromC) asm volatile("" : "+l"(C), "+l"(crs), "+l"(ccs));
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int col = col0 + (j / CV) * (8 * CV) + j % CV;
    if (col >= c) continue;
    uint32_t* __restrict__ pc = C + col * ccs;
    uint32_t old[TM];
    if (rc) {
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int row = row0 + (i / 4) * 16 + i % 4;
        old[i] = row < r ? pc[row * crs] : 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int row = row0 + (i / 4) * 16 + i % 4;
      const uint32_t v = i % 2 ? hi4(acc[i / 2][j]) : lo4(acc[i / 2][j]);
      if (row < r) pc[row * crs] = rc ? op.value(old[i], v) : op.value(v);
    }
  }
}

// jmul!'s chain with the BLAS alpha/beta epilogue (beta == 0: C is not read).
struct F32Chain {
  static constexpr bool kInitFromC = false;
  float alpha, beta;
  static __device__ __forceinline__ uint32_t init() { return 0x80000000u; }   // -0.0
  static __device__ __forceinline__ pair4 step(pair4 acc, pair4 a, pair4 b) { return fma_f32x2(a, b, acc); }
  __device__ __forceinline__ bool reads_c() const { return beta != 0.0f; }
  __device__ __forceinline__ uint32_t value(uint32_t acc) const { return __float_as_uint(alpha * __uint_as_float(acc)); }
  __device__ __forceinline__ uint32_t value(uint32_t c, uint32_t acc) const {
    return __float_as_uint(fmaf(alpha, __uint_as_float(acc), beta * __uint_as_float(c)));
  }
};

}  // namespace gb
