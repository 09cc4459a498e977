// FP32 tile of C on the CUDA cores with packed arithmetic: jmul!'s per-element FMA chain.
//
// What bounds it: the FFMA pipe (one warp FFMA per clock and SM partition) needs three operands'
// worth of shared-memory reads and bookkeeping issued beside it, and with one FMA per instruction
// those compete with the FMAs for issue slots.  fma.rn.f32x2 does two FMAs per issue slot at the
// same pipe rate (each half rounds as fmaf does, so the chain keeps its bits), which leaves half of
// the slots free.  A pair is two consecutive rows of C: the rows of A lie side by side in shared
// memory, and B's panel is stored with every element twice, so both operands are read ready-made.
// With 16 x 8 elements a thread, a k costs 64 packed FMAs (128 pipe cycles) and 8 16-byte reads.
// Operand panels come through cp.async, 4 bytes each (any alignment, either orientation),
// F32_STAGES - 1 panels ahead.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "f64_tile.cuh"   // cp.async helpers

namespace gb {

constexpr int F32_BK = 16;
constexpr int F32_STAGES = 3;

__device__ __forceinline__ void cp_async_4(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  return static_cast<uint64_t>(__float_as_uint(lo)) | (static_cast<uint64_t>(__float_as_uint(hi)) << 32);
}
__device__ __forceinline__ float lo_f32x2(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float hi_f32x2(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }

// Tile of WM x WN warps, each 4 x 8 lanes of TM x TN elements.
template <int WM_, int WN_, int TM_, int TN_>
struct F32Shape {
  static constexpr int WM = WM_, WN = WN_, TM = TM_, TN = TN_;
  static constexpr int BM = WM * 4 * TM, BN = WN * 8 * TN, THREADS = WM * WN * 32;
  static constexpr int LDA = BM + 4, LDB = 2 * BN + 4;   // floats; rows 16-byte aligned
  static constexpr int PANEL = F32_BK * (LDA + LDB);
  static constexpr int SMEM_BYTES = F32_STAGES * PANEL * 4;
  static_assert(TM % 4 == 0 && TN % 2 == 0, "16-byte operand reads");
  static_assert(THREADS % F32_BK == 0 && (BM % THREADS == 0 || THREADS % BM == 0) &&
                (BN % THREADS == 0 || THREADS % BN == 0), "panel loads");
};

// One thread's share of an operand's panels: element (x, k), x < extent, is src[x * xs + k * ks] and
// goes to word k * LD + x * DUP of the panel (and the next word, when DUP = 2).  The lanes run along
// the unit stride.
template <int X, int LD, int DUP, int THREADS>
struct F32Loader {
  static constexpr int N = X * F32_BK / THREADS;   // elements per thread
  const float* p;
  int64_t step, adv;
  int x, k, dx, dk;
  uint32_t dst, ddst;

  __device__ __forceinline__ void init(const float* src, int64_t xs, int64_t ks) {
    const int tid = threadIdx.x;
    const bool kfast = ks == 1 && xs != 1;
    // x fastest: X a multiple or a divisor of THREADS
    constexpr int XS = X < THREADS ? X : THREADS;
    x = kfast ? tid / F32_BK : tid % XS;
    k = kfast ? tid % F32_BK : tid / XS;
    dx = kfast ? THREADS / F32_BK : (X > THREADS ? THREADS : 0);
    dk = kfast ? 0 : (X > THREADS ? 0 : THREADS / XS);
    p = src + x * xs + k * ks;
    step = dx * xs + dk * ks;
    adv = F32_BK * ks;
    dst = static_cast<uint32_t>(k * LD + x * DUP) * 4u;
    ddst = static_cast<uint32_t>(dk * LD + dx * DUP) * 4u;
  }
  __device__ __forceinline__ void load(uint32_t panel, int extent, int kc) {
    const float* q = p;
#pragma unroll
    for (int l = 0; l < N; ++l) {
      if (x + l * dx < extent && k + l * dk < kc) {
        cp_async_4(panel + dst + l * ddst, q);
        if (DUP == 2) cp_async_4(panel + dst + l * ddst + 4, q);
      }
      q += step;
    }
    p += adv;
  }
};

// The tile of C at C (its first element, r x c of it inside the matrix): the chain from -0.0, or
// with ONTO from C's value, over k = 0..K-1 in order; `store(c pointer, chain)` writes an element.
// A's element (i, k) is A[i * ars + k * aks], B's (k, j) is B[k * bks + j * bcs].  No padded k is
// folded in; rows and columns past the edge compute on stale shared memory and are not stored.
// The last shared-memory reads are not followed by a barrier.
template <class S, bool ONTO, class Store>
__device__ __forceinline__ void f32_tile(int r, int c, int64_t K, const float* __restrict__ A, int64_t ars,
                                         int64_t aks, const float* __restrict__ B, int64_t bks, int64_t bcs,
                                         float* __restrict__ C, int64_t ldc, const Store& store, float* smem) {
  constexpr int TM = S::TM, TN = S::TN, BK = F32_BK;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row0 = (warp % S::WM) * 4 * TM + (lane >> 3) * 4;    // + 16 per chunk of 4 rows
  const int col0 = (warp / S::WM) * 8 * TN + (lane & 7) * 2;     // + 16 per chunk of 2 columns

  F32Loader<S::BM, S::LDA, 1, S::THREADS> la;
  F32Loader<S::BN, S::LDB, 2, S::THREADS> lb;
  la.init(A, ars, aks);
  lb.init(B, bcs, bks);
  const uint32_t smem_u = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int64_t panels = (K + BK - 1) / BK;
  auto load = [&](int64_t p, int stage) {   // panel p into a stage (panels are loaded in order)
    const int64_t left = K - p * BK;
    const int kc = static_cast<int>(left < BK ? left : BK);
    const uint32_t dst = smem_u + static_cast<uint32_t>(stage * (S::PANEL * 4));
    la.load(dst, r, kc);
    lb.load(dst + BK * S::LDA * 4, c, kc);
  };
#pragma unroll
  for (int p = 0; p < F32_STAGES - 1; ++p) {
    if (p < panels) load(p, p);
    cp_async_commit();
  }

  uint64_t acc[TM / 2][TN];
#pragma unroll
  for (int i = 0; i < TM / 2; ++i) {
    const int row = row0 + (i / 2) * 16 + (i % 2) * 2;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int col = col0 + (j / 2) * 16 + j % 2;
      float lo = -0.0f, hi = -0.0f;
      if (ONTO && col < c) {
        if (row < r) lo = C[row + col * ldc];
        if (row + 1 < r) hi = C[row + 1 + col * ldc];
      }
      acc[i][j] = pack_f32x2(lo, hi);
    }
  }

  auto read = [&](const float* pa, const float* pb, int k, uint64_t (&a)[TM / 2], uint64_t (&b)[TN]) {
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pa + k * S::LDA + row0 + i * 16);
      a[2 * i] = v.x;
      a[2 * i + 1] = v.y;
    }
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pb + k * S::LDB + (col0 + j * 16) * 2);
      b[2 * j] = v.x;
      b[2 * j + 1] = v.y;
    }
  };
  auto step = [&](const uint64_t (&a)[TM / 2], const uint64_t (&b)[TN]) {
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = fma_f32x2(a[i], b[j], acc[i][j]);
  };

  int stage = 0;
  for (int64_t p = 0; p < panels; ++p) {
    cp_async_wait<F32_STAGES - 2>();
    __syncthreads();   // panel p is in place, and every warp has left panel p - 1's stage
    if (p + F32_STAGES - 1 < panels) load(p + F32_STAGES - 1, (stage + F32_STAGES - 1) % F32_STAGES);
    cp_async_commit();
    const float* pa = smem + stage * S::PANEL;
    const float* pb = pa + BK * S::LDA;
    stage = (stage + 1) % F32_STAGES;
    const int64_t left = K - p * BK;
    uint64_t a0[TM / 2], b0[TN], a1[TM / 2], b1[TN];
    if (left >= BK) {
      read(pa, pb, 0, a0, b0);
#pragma unroll
      for (int k = 0; k < BK; k += 2) {   // the next k's operands are read before this one's FMAs
        read(pa, pb, k + 1, a1, b1);
        step(a0, b0);
        if (k + 2 < BK) read(pa, pb, k + 2, a0, b0);
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

#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int col = col0 + (j / 2) * 16 + j % 2;
    if (col >= c) continue;
    float* __restrict__ pc = C + col * ldc;
#pragma unroll
    for (int i = 0; i < TM / 2; ++i) {
      const int row = row0 + (i / 2) * 16 + (i % 2) * 2;
      if (row < r) store(pc + row, lo_f32x2(acc[i][j]));
      if (row + 1 < r) store(pc + row + 1, hi_f32x2(acc[i][j]));
    }
  }
}

}  // namespace gb
