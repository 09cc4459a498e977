// One-warp tile of a semiring product for 4-byte elements: C = [C (+)] (+)_k A[i,k] (x) B[k,j].
//
// What bounds it: a half-rate instruction (a packed add, a three-input minimum) holds its partition's
// dispatch port for two cycles, so (min, +) takes two cycles an element and k whether the adds are
// packed or not (18 to 20 T/s in a register-only loop), and small products an SM that waits.  Panels hold
// two consecutive k of an element side by side, as (k, k + 1) pairs: add.rn.f32x2 on a pair of A and a
// pair of B gives both products of a (+)-step of two k with nothing duplicated or moved.  The rest is
// as in simt4_tile.cuh: a tile is one warp's, panels through cp.async.  32 x 32 tiles: larger ones
// (64 x 64, 64 x 32, 32 x 64) were slower at every size, short of registers or of warps.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "f64_tile.cuh"   // cp.async helpers
#include "simt4_tile.cuh"

namespace gb {

template <int TM_, int TN_>
struct SrShape {
  static constexpr int TM = TM_, TN = TN_, BM = 4 * TM, BN = 8 * TN;
  static constexpr int LDA = 2 * BM + 8, LDB = 2 * BN + 8;       // words of a k pair
  static constexpr int PANEL = S4_BK / 2 * (LDA + LDB);
  static constexpr int SMEM_BYTES = S4_STAGES * PANEL * 4;       // of one warp
  static_assert(TM % 2 == 0 && TN % 2 == 0, "two elements a read");
};

// One lane's share of an operand's panels: element (x, k), x < extent <= X, is src[x * xs + k * ks] and
// goes to word k / 2 * LD + 2 x + k % 2 of the panel.  Ways: KP two k a copy (ks = 1, 8-byte aligned),
// XF the lanes along x, KF the lanes along k.
template <int X, int LD>
struct SrLoader {
  static_assert(X == 32, "a lane per x");
  static constexpr int KP = 0, XF = 1, KF = 2;
  const uint32_t* p;
  int64_t str, adv;
  uint32_t dst;
  int way, x, k;

  __device__ __forceinline__ void init(const uint32_t* src, int64_t xs, int64_t ks) {
    const int lane = threadIdx.x & 31;
    way = (ks == 1 && xs != 1) ? ((reinterpret_cast<uintptr_t>(src) & 7) == 0 && (xs & 1) == 0 ? KP : KF) : XF;
    x = way == KP ? lane / 4 : way == XF ? lane : lane / 8;
    k = way == KP ? lane % 4 * 2 : way == XF ? 0 : lane % 8;
    p = src + x * xs + k * ks;
    str = way == KP ? 8 * xs : way == XF ? ks : 4 * xs;
    adv = S4_BK * ks;
    dst = static_cast<uint32_t>(k / 2 * LD + 2 * x + k % 2) * 4u;
  }
  template <bool CHECK>
  __device__ __forceinline__ void copy(uint32_t d, int extent, int kc) {
    const uint32_t* q = p;
    if (way == KP) {
#pragma unroll 8
      for (int l = 0; l < X / 8; ++l, q += str)
#pragma unroll
        for (int h = 0; h < S4_BK; h += 8) {
          const uint32_t to = d + (h / 2 * LD + l * 16) * 4;
          if (!CHECK || (x + l * 8 < extent && k + h + 1 < kc)) cp_async_8(to, q + h);
          else if (x + l * 8 < extent && k + h < kc) cp_async_4(to, q + h);
        }
    } else if (way == XF) {
#pragma unroll 8
      for (int l = 0; l < S4_BK; ++l, q += str)
        if (!CHECK || (x < extent && l < kc)) cp_async_4(d + (l / 2 * LD + l % 2) * 4, q);
    } else {
#pragma unroll 8
      for (int l = 0; l < X / 4; ++l, q += str)
#pragma unroll
        for (int h = 0; h < S4_BK; h += 8)
          if (!CHECK || (x + l * 4 < extent && k + h < kc)) cp_async_4(d + (h / 2 * LD + l * 8) * 4, q + h);
    }
  }
  __device__ __forceinline__ void load(uint32_t panel, int extent, int kc) {
    if (extent == X && kc == S4_BK) copy<false>(panel + dst, extent, kc);
    else copy<true>(panel + dst, extent, kc);
    p += adv;
  }
};

// The r x c tile of C at C (leading dimension ldc), 1 <= r <= BM, 1 <= c <= BN, by one warp.  `Op`:
//   Op::init()                 the identity of (+)
//   Op::step2(acc, a, b)       two consecutive k at once: a and b hold an element's pair
//   Op::step(acc, a, b)        the low halves only (an odd last k)
//   op.reads_c(), op.value(c, acc), op.value(acc)
// A's element (i, k) is A[i * ars + k * aks], B's (k, j) is B[k * bks + j * bcs].  No padded k is folded in.
template <class S, class Op>
__device__ __forceinline__ void semiring4_tile(int r, int c, int64_t K, const Op& op, const uint32_t* __restrict__ A,
                                               int64_t ars, int64_t aks, const uint32_t* __restrict__ B, int64_t bks,
                                               int64_t bcs, uint32_t* __restrict__ C, int64_t ldc, uint32_t* smem) {
  constexpr int TM = S::TM, TN = S::TN, BK = S4_BK;
  const int lane = threadIdx.x & 31;
  const int row0 = (lane >> 3) * 2;     // + 8 per two rows
  const int col0 = (lane & 7) * 2;      // + 16 per two columns

  SrLoader<S::BM, S::LDA> la;
  SrLoader<S::BN, S::LDB> lb;
  la.init(A, ars, aks);
  lb.init(B, bcs, bks);
  const uint32_t smem_u = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int64_t panels = (K + BK - 1) / BK;
  uint32_t acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = Op::init();

  int stage = 0, load_stage = 0;
  for (int64_t q = 0; q < panels + S4_STAGES - 1; ++q) {
    cp_async_wait<S4_STAGES - 2>();   // panel q - (S4_STAGES - 1), the oldest but S4_STAGES - 2, is in place
    __syncwarp();                     // for every lane, and all have left the stage to be loaded
    if (q < panels) {
      const int64_t left = K - q * BK;
      const int kc = static_cast<int>(left < BK ? left : BK);
      const uint32_t dst = smem_u + static_cast<uint32_t>(load_stage * (S::PANEL * 4));
      la.load(dst, r, kc);
      lb.load(dst + BK / 2 * S::LDA * 4, c, kc);
      load_stage = (load_stage + 1) % S4_STAGES;
    }
    cp_async_commit();
    const int64_t p = q - (S4_STAGES - 1);
    if (p < 0) continue;
    const uint32_t* pa = smem + stage * S::PANEL + 2 * row0;
    const uint32_t* pb = smem + stage * S::PANEL + BK / 2 * S::LDA + 2 * col0;
    stage = (stage + 1) % S4_STAGES;
    const int64_t left = K - p * BK;
    pair4 a[TM], b[TN];
    auto read = [&](int kp) {
#pragma unroll
      for (int i = 0; i < TM; i += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pa + kp * S::LDA + i * 8);
        a[i] = v.x;
        a[i + 1] = v.y;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pb + kp * S::LDB + j * 16);
        b[j] = v.x;
        b[j + 1] = v.y;
      }
    };
    auto step2 = [&]() {
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = Op::step2(acc[i][j], a[i], b[j]);
    };
    if (left >= BK) {
#pragma unroll 4
      for (int kp = 0; kp < BK / 2; ++kp) {
        read(kp);
        step2();
      }
    } else {
      const int kc = static_cast<int>(left);
      for (int kp = 0; kp < kc / 2; ++kp) {
        read(kp);
        step2();
      }
      if (kc & 1) {
        read(kc / 2);
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
          for (int i = 0; i < TM; ++i) acc[i][j] = Op::step(acc[i][j], lo4(a[i]), lo4(b[j]));
      }
    }
  }
  cp_async_wait<0>();   // (only empty groups are left)
  __syncwarp();         // the next tile reuses the stages

  // Two rows at a time where C is aligned for it: the warp then writes whole sectors of a column.  C's
  // old values are all requested before the first is used (2048 x 2048 x 64 with C folded in 110 -> 33 us).
  asm volatile("" : "+l"(C), "+l"(ldc));   // (no address is computed ahead and kept through the k loop)
  const bool rc = op.reads_c();
  const bool wide = ((reinterpret_cast<uintptr_t>(C) | static_cast<uintptr_t>(ldc * 4)) & 7) == 0;
  uint32_t old[TM][TN];
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int col = col0 + (j / 2) * 16 + j % 2;
#pragma unroll
    for (int i = 0; i < TM; i += 2) {
      const int row = row0 + (i / 2) * 8;
      const uint32_t* pc = C + row + col * ldc;
      old[i][j] = old[i + 1][j] = 0u;
      if (!rc || col >= c) continue;
      if (wide && row + 1 < r) {
        const uint2 v = *reinterpret_cast<const uint2*>(pc);
        old[i][j] = v.x;
        old[i + 1][j] = v.y;
      } else {
        if (row < r) old[i][j] = pc[0];
        if (row + 1 < r) old[i + 1][j] = pc[1];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int col = col0 + (j / 2) * 16 + j % 2;
    if (col >= c) continue;
#pragma unroll
    for (int i = 0; i < TM; i += 2) {
      const int row = row0 + (i / 2) * 8;
      uint32_t* pc = C + row + col * ldc;
      const uint32_t lo = rc ? op.value(old[i][j], acc[i][j]) : op.value(acc[i][j]);
      const uint32_t hi = rc ? op.value(old[i + 1][j], acc[i + 1][j]) : op.value(acc[i + 1][j]);
      if (wide && row + 1 < r) {
        *reinterpret_cast<uint2*>(pc) = make_uint2(lo, hi);
      } else {
        if (row < r) pc[0] = lo;
        if (row + 1 < r) pc[1] = hi;
      }
    }
  }
}

}  // namespace gb
