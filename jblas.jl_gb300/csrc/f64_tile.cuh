// One FP64 tile of C on the CUDA cores, shared by the native GEMM (native_gemm.cu) and the
// grouped GEMM (grouped.cu), jmul!'s per-element FMA chain (src/gemm.jl:76-89, 154-168), and by the
// FP64 semirings (semiring_f64.cu).  What an element does with each k is a policy (F64Chain below).
//
// What bounds it: GB300 executes half an FP64 lane per clock and SM partition, so a warp's DFMA
// holds its partition's FP64 pipe for 64 cycles (measured; the same for 1 or 32 active lanes, and
// one warp with one dependent chain already fills the pipe).  Register tiles, shared-memory
// bandwidth and occupancy do not matter at that rate; what does is that no DFMA lane is spent on
// padding and that the four partitions of every SM get the same number of them.  Therefore:
//  - the elements of the r x c tile are numbered down its columns and dealt 32 at a time ("units")
//    to the CTA's 4 warps, one on each partition, so a ragged tile pads to a multiple of 32
//    elements instead of to a multiple of a register tile in both directions (33 x 17: 18 units;
//    six 16 x 16 tiles: 48);
//  - each lane reads its row of A and column of B from shared memory for every DFMA (two 8-byte
//    reads against 64 cycles);
//  - the CTA is small (128 threads, at most 128 registers each, four CTAs an SM), so that one tile's
//    loads, barriers and stores hide behind the DFMAs of three others;
//  - the tile's extent is a run-time choice, so a caller picks the one that spreads its work over
//    the SMs.
// The operand panels come through cp.async, 8 bytes each (any alignment, either orientation),
// F64_STAGES - 1 panels ahead; the smaller the tile, the more k a panel holds.  Only elements
// inside the tile and inside K are loaded, and only those are multiplied: no padded k is ever
// folded in.
// Measured, against register tiles of 4 x 4 (native) and 1 x 1 (grouped) a thread: native 256^3
// 141 -> 36.9 us a call (27 at the DFMA peak), 16 x 14 x 32 20.5 -> 12.4 us a call, 777 x 1001 x 555
// 0.85 -> 0.75 ms, 1024^3 1.92 -> 1.79 ms, 2048^3 and above the same (99% of the pipe); 4096
// log-uniform problems (8..512) 14.4 -> 12.0 ms (11.6 at the peak), 8192 of 33 x 17 x 65 1.66 -> 0.67 ms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gb {

constexpr int F64_THREADS = 128;
constexpr int F64_WARPS = F64_THREADS / 32;
constexpr int F64_CTAS = 4;         // resident CTAs per SM
constexpr int F64_MAX_UNITS = 8;    // units per warp: tiles of at most 1024 elements
constexpr int F64_MAX_ELEMS = F64_MAX_UNITS * F64_WARPS * 32;
constexpr int F64_STAGES = 4;

// Shapes of shared panels: tiles of at most XA x XB elements, BK k per panel, rows padded by one
// (k-fastest writes then hit distinct banks).
template <int XA, int XB>
struct F64Shape {
  static constexpr int BK = 512 / XA;
  static constexpr int LDA = XA + 1, LDB = XB + 1;
  static constexpr int PANEL = BK * (LDA + LDB);   // elements of one stage
  static constexpr int SMEM = F64_STAGES * PANEL;
  static_assert(XA * BK % F64_THREADS == 0 && XB * BK % F64_THREADS == 0, "FP64 tile shape");
};
// The three shapes: 64 x 32 (BK 8), 32 x 32 (BK 16), 16 x 16 (BK 32); 1024 elements at most in each.
constexpr int F64_SMEM_ELEMS = F64Shape<16, 16>::SMEM;   // 34,816 bytes, the largest
static_assert(F64Shape<32, 32>::SMEM <= F64_SMEM_ELEMS && F64Shape<64, 32>::SMEM <= F64_SMEM_ELEMS, "shared panels");

__device__ __forceinline__ void cp_async_8(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One thread's share of an operand's panels: element (x, k), x < extent <= X, of the operand is
// src[x * xs + k * ks] and goes to [k][x] of the panel.  The lanes run along the unit stride.
template <int X, int BK>
struct F64Loader {
  static constexpr int N = X * BK / F64_THREADS;   // elements per thread
  const double* p;          // the thread's first element of the next panel
  int64_t step, adv;        // between the thread's elements; to the next panel
  int x, k, dx, dk;         // first element and the step in (x, k)
  uint32_t dst, ddst;       // byte offsets in the panel

  __device__ __forceinline__ void init(const double* src, int64_t xs, int64_t ks) {
    const int tid = threadIdx.x;
    const bool kfast = ks == 1 && xs != 1;
    x = kfast ? tid / BK : tid % X;
    k = kfast ? tid % BK : tid / X;
    dx = kfast ? F64_THREADS / BK : 0;
    dk = kfast ? 0 : F64_THREADS / X;
    p = src + x * xs + k * ks;
    step = dx * xs + dk * ks;
    adv = BK * ks;
    dst = static_cast<uint32_t>(k * (X + 1) + x) * 8u;
    ddst = static_cast<uint32_t>(dk * (X + 1) + dx) * 8u;
  }
  // Rewrites the elements of a panel that this thread loaded (its copies have arrived).
  template <class Op>
  __device__ __forceinline__ void encode(unsigned long long* panel, int extent, int kc) const {
#pragma unroll
    for (int l = 0; l < N; ++l) {
      unsigned long long* e = panel + (dst + l * ddst) / 8;
      if (x + l * dx < extent && k + l * dk < kc) *e = Op::encode(*e);
    }
  }
  // Loads the panel of kc k to the shared address `panel`.
  __device__ __forceinline__ void load(uint32_t panel, int extent, int kc) {
    const double* q = p;
#pragma unroll
    for (int l = 0; l < N; ++l) {
      if (x + l * dx < extent && k + l * dk < kc) cp_async_8(panel + dst + l * ddst, q);
      q += step;
    }
    p += adv;
  }
};

// The policy of the FMA chains:
//   ONTO = false   the chain starts at -0.0 (fma(a1, x1, -0.0) is the rounded product a1 x1) and
//                  C = alpha * chain [+ beta * C]; `out` (f64_out) says which of the terms there are, so
//                  that the epilogue issues no other FP64 instruction, comparisons of alpha and beta
//                  included: each costs an element as much as one k
//   ONTO = true    the chain starts at C's value and is stored as it is (jBLAS's kernel!)
enum { F64_CHAIN, F64_SCALED, F64_WITH_C };
// On the bits: 1.0 is the only double with its pattern, and a shift drops the sign of zero.
__host__ __device__ inline int f64_out(long long alpha_bits, long long beta_bits) {
  return (static_cast<unsigned long long>(beta_bits) << 1) != 0 ? F64_WITH_C
       : alpha_bits != 0x3FF0000000000000ll ? F64_SCALED : F64_CHAIN;
}
template <bool ONTO>
struct F64Chain {
  using Elem = double;   // an element in shared memory, and
  using Acc = double;    // what a lane keeps for an element of C
  static constexpr bool ENCODE = false;   // no rewriting of the panels
  static constexpr int AHEAD = 4;         // old values of C in flight (8: the same, and more spilled)
  double alpha, beta;
  int out;
  __device__ __forceinline__ double init(const double* c, bool in) const { return (ONTO && in) ? *c : -0.0; }
  static __device__ __forceinline__ double step(double acc, double a, double b) { return fma(a, b, acc); }
  __device__ __forceinline__ bool reads_c() const { return !ONTO && out == F64_WITH_C; }
  __device__ __forceinline__ double value(double c, double acc) const { return fma(alpha, acc, beta * c); }
  __device__ __forceinline__ bool plain() const { return ONTO || out == F64_CHAIN; }
  static __device__ __forceinline__ double raw(double acc) { return acc; }
  __device__ __forceinline__ double value(double acc) const { return alpha * acc; }
};

// NU chains per lane over the kc k of one panel; off[i] holds the byte offsets of the lane's row
// of A (low half) and column of B (high half) inside a panel row.  The operands of the next k are
// read before the DFMAs of this one: with one CTA on an SM nothing else hides the reads' latency.
// (16 chains, which leave no registers for that, ran at 73% of the pipe on a ragged product.)
template <class Op, int NU, int LDA, int LDB>
__device__ __forceinline__ void f64_panel(const char* __restrict__ pa, const char* __restrict__ pb, int kc,
                                          const uint32_t (&off)[F64_MAX_UNITS],
                                          typename Op::Acc (&acc)[F64_MAX_UNITS]) {
  using E = typename Op::Elem;
  auto read = [&](int k, E (&a)[NU], E (&b)[NU]) {
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      a[i] = *reinterpret_cast<const E*>(pa + k * (LDA * 8) + (off[i] & 0xFFFFu));
      b[i] = *reinterpret_cast<const E*>(pb + k * (LDB * 8) + (off[i] >> 16));
    }
  };
  auto step = [&](const E (&a)[NU], const E (&b)[NU]) {
#pragma unroll
    for (int i = 0; i < NU; ++i) acc[i] = Op::step(acc[i], a[i], b[i]);
  };
  E a0[NU], b0[NU], a1[NU], b1[NU];
  read(0, a0, b0);
  int k = 0;
  for (; k + 2 < kc; k += 2) {
    read(k + 1, a1, b1);
    step(a0, b0);
    read(k + 2, a0, b0);
    step(a1, b1);
  }
  if (k + 1 < kc) {
    read(k + 1, a1, b1);
    step(a0, b0);
    step(a1, b1);
  } else {
    step(a0, b0);
  }
}

// The r x c tile of C at C (its first element; leading dimension ldc), 1 <= r <= XA, 1 <= c <= XB,
// r c <= F64_MAX_ELEMS.  A's element (i, k) is A[i * ars + k * aks], B's (k, j) is B[k * bks + j * bcs].  `rot` deals the
// units from another warp in each tile, so the partitions share the remainders.  K >= 0.
// The tile's last shared-memory reads are not followed by a barrier.
template <int XA, int XB, class Op>
__device__ __forceinline__ void f64_tile(int r, int c, int64_t K, const double* __restrict__ A, int64_t ars,
                                         int64_t aks, const double* __restrict__ B, int64_t bks, int64_t bcs,
                                         const Op& op, double* __restrict__ C, int64_t ldc, int rot, double* smem) {
  using S = F64Shape<XA, XB>;
  constexpr int BK = S::BK;
  constexpr int MAXU = XA * XB < F64_MAX_ELEMS ? XA * XB / 32 / F64_WARPS : F64_MAX_UNITS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int elems = r * c;
  const int v = (warp + rot) & (F64_WARPS - 1);
  const int units = (elems + 31) >> 5;
  const int nu = units > v ? (units - v + F64_WARPS - 1) / F64_WARPS : 0;   // this warp's units

  F64Loader<XA, BK> la;
  F64Loader<XB, BK> lb;
  la.init(A, ars, aks);
  lb.init(B, bcs, bks);
  const uint32_t smem_a = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int64_t panels = (K + BK - 1) / BK;
  auto load = [&](int64_t p, int stage) {   // panel p into a stage (panels are loaded in order)
    const int64_t left = K - p * BK;
    const int kc = static_cast<int>(left < BK ? left : BK);
    const uint32_t dst = smem_a + static_cast<uint32_t>(stage * (S::PANEL * 8));
    la.load(dst, r, kc);
    lb.load(dst + BK * S::LDA * 8, c, kc);
  };
#pragma unroll
  for (int p = 0; p < F64_STAGES - 1; ++p) {
    if (p < panels) load(p, p);
    cp_async_commit();
  }

  // Row and column of each of the lane's elements v * 32 + lane, + 128, ...; past the last element
  // the lane repeats it (and does not store).
  uint32_t off[F64_MAX_UNITS];
  typename Op::Acc acc[F64_MAX_UNITS];
  {
    const int e0 = v * 32 + lane;
    int col = e0 / r, row = e0 - col * r;
    const int dcol = F64_THREADS / r, drow = F64_THREADS - dcol * r;
#pragma unroll
    for (int i = 0; i < MAXU; ++i) {
      if (i >= nu) break;
      const bool in = e0 + i * F64_THREADS < elems;
      const int rr = in ? row : r - 1, cc = in ? col : c - 1;
      off[i] = static_cast<uint32_t>(rr * 8) | (static_cast<uint32_t>(cc * 8) << 16);
      acc[i] = op.init(C + rr + cc * ldc, in);
      row += drow;
      col += dcol;
      if (row >= r) {
        row -= r;
        ++col;
      }
    }
  }

  int stage = 0;
  for (int64_t p = 0; p < panels; ++p) {
    const int64_t left = K - p * BK;
    const int kc = static_cast<int>(left < BK ? left : BK);
    cp_async_wait<F64_STAGES - 2>();
    if constexpr (Op::ENCODE) {
      unsigned long long* panel = reinterpret_cast<unsigned long long*>(smem) + stage * S::PANEL;
      la.template encode<Op>(panel, r, kc);
      lb.template encode<Op>(panel + BK * S::LDA, c, kc);
    }
    __syncthreads();   // panel p is in place, and every warp has left panel p - 1's stage
    if (p + F64_STAGES - 1 < panels) load(p + F64_STAGES - 1, (stage + F64_STAGES - 1) % F64_STAGES);
    cp_async_commit();
    const char* pa = reinterpret_cast<const char*>(smem + stage * S::PANEL);
    const char* pb = pa + BK * S::LDA * 8;
    stage = (stage + 1) % F64_STAGES;
    switch (nu) {   // uniform in the warp
#define GB_F64_CASE(n_) \
  case n_: if constexpr (n_ <= MAXU) f64_panel<Op, n_, S::LDA, S::LDB>(pa, pb, kc, off, acc); break;
      GB_F64_CASE(1) GB_F64_CASE(2) GB_F64_CASE(3) GB_F64_CASE(4) GB_F64_CASE(5) GB_F64_CASE(6) GB_F64_CASE(7)
      GB_F64_CASE(8)
#undef GB_F64_CASE
      default: break;
    }
  }
  cp_async_wait<0>();   // (only empty groups are left)

  // C's old values, where the epilogue reads them, are requested AHEAD at a time before the first is
  // used; the three ways are written out, so that none issues another's FP64 instructions: with one
  // expression for all and a value at a time, 4096 x 4096 x 8 with alpha and beta took 372 us instead of
  // 312 (alpha = 1, beta = 0: 231).  (The addresses are opaque before this point: computed ahead
  // and kept through the k loop, they spilled.)
  if constexpr (Op::AHEAD > 1) asm volatile("" : "+l"(C), "+l"(ldc));
  auto at = [&](int i) { return C + (off[i] & 0xFFFFu) / 8 + static_cast<int64_t>(off[i] >> 19) * ldc; };
  constexpr int AHEAD = MAXU < Op::AHEAD ? MAXU : Op::AHEAD;
  const int mine = elems - v * 32 - lane;   // element i is the lane's when i * F64_THREADS < mine
  if (op.reads_c()) {
#pragma unroll
    for (int i0 = 0; i0 < MAXU; i0 += AHEAD) {
      double old[AHEAD];
#pragma unroll
      for (int i = 0; i < AHEAD; ++i)
        if ((i0 + i) * F64_THREADS < mine) old[i] = *at(i0 + i);
#pragma unroll
      for (int i = 0; i < AHEAD; ++i)
        if ((i0 + i) * F64_THREADS < mine) *at(i0 + i) = op.value(old[i], acc[i0 + i]);
    }
  } else if (op.plain()) {
#pragma unroll
    for (int i = 0; i < MAXU; ++i)
      if (i * F64_THREADS < mine) *at(i) = Op::raw(acc[i]);
  } else {
#pragma unroll
    for (int i = 0; i < MAXU; ++i)
      if (i * F64_THREADS < mine) *at(i) = op.value(acc[i]);
  }
}

// The tile on the panel shape that fits it (64 x 32, 32 x 32 or 16 x 16: the smaller ones take
// fewer barriers per k).
template <class Op>
__device__ __forceinline__ void f64_tile_any(int r, int c, int64_t K, const double* __restrict__ A, int64_t ars,
                                             int64_t aks, const double* __restrict__ B, int64_t bks, int64_t bcs,
                                             const Op& op, double* __restrict__ C, int64_t ldc, int rot,
                                             double* smem) {
  if (r <= 16 && c <= 16)
    f64_tile<16, 16>(r, c, K, A, ars, aks, B, bks, bcs, op, C, ldc, rot, smem);
  else if (r <= 32)
    f64_tile<32, 32>(r, c, K, A, ars, aks, B, bks, bcs, op, C, ldc, rot, smem);
  else
    f64_tile<64, 32>(r, c, K, A, ars, aks, B, bks, bcs, op, C, ldc, rot, smem);
}

}  // namespace gb
