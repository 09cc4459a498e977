// Grouped GEMM: thousands of independent, uneven C_i = alpha_i A_i B_i + beta_i C_i in one
// persistent launch (FP64 or FP32, CUDA cores, jmul!'s per-element FMA order).
//
// jBLAS multiplies small static matrices one call at a time (fastmul!/kernel!,
// src/kernels.jl:202-208, 239) with a tile size fixed at code-generation time
// (pick_kernel_size, src/kernel_structure.jl:76-99; BLASOptions, src/blas_options.jl:2-7).
// Here one launch walks every tile of every problem:
//   1. a prologue kernel classifies each problem by max(m, n) into a size class, takes
//      that class's tile configuration from the tuning table (chosen by the autotuner,
//      gb_autotune_grouped), counts its tiles and writes the exclusive prefix sum;
//   2. the CTAs of the persistent kernel (grid = SMs x resident CTAs) take one global tile
//      index after another, find its problem by a search in the prefix sums and run that
//      configuration's tile routine.
// Both kernels read only device memory, so a call can be captured in a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <vector>

#include "f64_tile.cuh"
#include "gb_common.cuh"
#include "grouped.cuh"
#include "profile.cuh"
#include "simt4_tile.cuh"

namespace gb {

struct TileCfg {
  int bm, bn;
};
// 0-3 serve both element types; 4-9, the larger and rectangular tiles, are FP32 only.  FP64 takes bm
// and bn as the largest extents of its tiles (f64_tiles); FP32 runs a tile in pieces of 64 x 64.
__host__ __device__ constexpr TileCfg tile_cfg(int c) {
  return c == 0 ? TileCfg{16, 16}
       : c == 1 ? TileCfg{32, 32}
       : c == 2 ? TileCfg{64, 32}
       : c == 3 ? TileCfg{64, 64}
       : c == 4 ? TileCfg{128, 64}
       : c == 5 ? TileCfg{128, 128}
       : c == 6 ? TileCfg{32, 64}
       : c == 7 ? TileCfg{64, 128}
       : c == 8 ? TileCfg{128, 32}
                : TileCfg{32, 128};
}
// ceil(x / d) for a tile extent, a power of two: without the division of 64 bits.
__host__ __device__ inline int64_t tiles_along(int64_t x, int d) {
#ifdef __CUDA_ARCH__
  return (x + d - 1) >> (31 - __clz(d));
#else
  return (x + d - 1) / d;
#endif
}
constexpr int GROUPED_CONFIGS_F64 = 4;
constexpr int GROUPED_CONFIGS_F32 = 10;

__host__ __device__ inline int size_class(int64_t m, int64_t n) {
  const int64_t d = m > n ? m : n;
  return d <= 16 ? 0 : d <= 32 ? 1 : d <= 64 ? 2 : d <= 128 ? 3 : d <= 256 ? 4 : 5;
}

// GB_GROUPED_AUTO in FP32, one choice for the whole table: 64 x 64 pieces, or 32 x 32 ones (one warp at
// work on each) where the outputs together have fewer elements than three quarters of such a piece an
// SM.  Measured, 32 x 32 and 64 x 64: 50 problems of 65 x 65 x 100 15.4 and 18.1 us, 10 of 200 x 200 x 64
// 14.1 and 14.8, one of 512^3 31.8 and 30.1, 32 of 128^3 17.4 and 15.7, 64 of 128^3 26 and 19, 16 of
// 300^3 61 and 40, 4 of 1000 x 1000 x 200 98 and 63 (with the line at three pieces a CTA all of these took
// the former).
__host__ __device__ inline int auto_config_f32(bool large) { return large ? 3 : 1; }
static int64_t f32_large_elems(int sms) { return static_cast<int64_t>(sms) * (64 * 64 * 3 / 4); }

// Extents of an FP64 problem's tiles under a configuration: equal tiles as large as the
// configuration, 32 columns and F64_MAX_ELEMS allow (33 rows on 32-row tiles: 17 + 16, not 32 + 1).
// In 32-bit arithmetic: a 64-bit division is some hundred instructions, of which the one-block prologue
// would make a dozen per problem; beyond it tiles are not made equal.
struct F64Tiles {
  int tm, tn, fm, fn;
};
__host__ __device__ inline F64Tiles f64_tiles(const TileCfg& c, int64_t m, int64_t n) {
  if (m <= 0 || n <= 0) return F64Tiles{0, 0, 0, 0};
  if (m > 0x7FFFFFFF - 64 || n > 0x7FFFFFFF - 64)
    return F64Tiles{static_cast<int>(tiles_along(m, c.bm)), static_cast<int>((n + 15) / 16), c.bm, 16};
  const uint32_t m32 = static_cast<uint32_t>(m), n32 = static_cast<uint32_t>(n);
  const uint32_t tm = static_cast<uint32_t>(tiles_along(m, c.bm)), fm = (m32 + tm - 1) / tm;
  const uint32_t room = F64_MAX_ELEMS / fm, most = c.bn < 32 ? c.bn : 32, width = room < most ? room : most;
  const uint32_t tn = (n32 + width - 1) / width, fn = (n32 + tn - 1) / tn;
  return F64Tiles{static_cast<int>(tm), static_cast<int>(tn), static_cast<int>(fm), static_cast<int>(fn)};
}

// GB_GROUPED_AUTO in FP64, where the DFMA pipe bounds everything (f64_tile.cuh).  A tile costs its units
// of 32 elements times k and, for its barriers, first loads and stores, 26 unit-k (measured on 8192
// problems of 32 x 32 x 64: 1.01 ms on 16 x 16 tiles, 0.96 on 32 x 32).  A call takes the sum of these
// over the SM partitions, or the longest tile's time on one of the four warps if that is longer.
struct F64Load {
  long long total = 0, longest = 0;
  __host__ __device__ void add(const F64Tiles& t, int64_t k, long long problems = 1) {
    const long long kk = k > 1 ? k : 1, units = (t.fm * t.fn + 31) / 32;
    const long long one = ((units + 3) / 4) * kk;
    total += problems * t.tm * t.tn * (units * kk + 26);
    longest = one > longest ? one : longest;
  }
  __host__ __device__ long long time(int sms) const {   // times 4 sms
    const long long l = longest * 4 * sms;
    return total > l ? total : l;
  }
};
// Per problem the configuration with the smallest total (0-2; 3 has 2's tiles), among those whose tiles
// F64_MAX_ELEMS does not cut (64 of 100^3 on cut 64 x 32 tiles, 10 a problem: 199 us, on 32 x 32 141), or, if a
// call has too little work for that, 16 x 16 for all: one problem of 100^3 32 -> 18 us, 10 of 64^3 31 -> 17,
// one of 64 x 64 x 200 78 -> 27; 16 of 100^3 stay (45 us, 63 on 16 x 16).
__host__ __device__ inline int auto_config_f64(int64_t m, int64_t n, int64_t k, F64Tiles* tiles) {
  *tiles = f64_tiles(tile_cfg(0), m, n);
  if (m <= 16 && n <= 16) return 0;   // one tile under any of them
  F64Load first;
  first.add(*tiles, k);
  long long best = first.total;
  int arg = 0;
  for (int c = 1; c < 3; ++c) {
    const F64Tiles t = f64_tiles(tile_cfg(c), m, n);
    if (c == 2 && t.tn > (n + 31) / 32) continue;
    F64Load l;
    l.add(t, k);
    if (l.total < best) {
      best = l.total;
      arg = c;
      *tiles = t;
    }
  }
  return arg;
}
// (From eight problems an SM the first choice stands, which saves the prologue the second.)
__host__ __device__ inline bool f64_may_be_small(int count, int sms) { return count < 8 * sms; }
__host__ __device__ inline bool f64_small(const F64Load& chosen, const F64Load& small, int sms) {
  return small.time(sms) < chosen.time(sms);
}

// tuning.config[cls] without a dynamically indexed (local-memory) array
__device__ __forceinline__ int config_of(const gb_grouped_tuning_t& t, int cls) {
  int v = t.config[0];
#pragma unroll
  for (int c = 1; c < GB_GROUPED_CLASSES; ++c) v = (cls == c) ? t.config[c] : v;
  return v;
}


// alpha = 0: C = beta C on one bm x bn tile (beta = 0 writes zeros without reading C; A and B
// are not read), as jBLAS's alpha/beta extension of gb_gemm_* defines it.
// Run by `threads` threads numbered `tid`.
template <typename T>
__device__ __forceinline__ void scale_tile(const gb_problem_t& p, int64_t m0, int64_t n0, int bm, int bn, int tid,
                                           int threads) {
  T* __restrict__ C = static_cast<T*>(p.C);
  const T beta = static_cast<T>(p.beta);
  for (int e = tid; e < bm * bn; e += threads) {
    const int64_t m = m0 + e % bm, n = n0 + e / bm;
    if (m < p.m && n < p.n) {
      T* c = &C[m + n * p.ldc];
      *c = (beta == T(0)) ? T(0) : beta * *c;
    }
  }
}

// Workspace of a call over `count` problems (int64 words): the tile prefix sums in schedule
// order offsets[0..count], then the schedule order (count int32 entries: the problem index,
// and for count <= 2^24 its tile configuration in bits 24-30, so the tile loop need not
// evaluate the per-problem choice again for every tile).  The first problem's tiles start at 0, so
// the tile loop takes that as known and counts the tiles it has handed out in offsets[0].
__host__ __device__ inline long long* grouped_order_words(long long* ws, int count) { return ws + count + 1; }
constexpr int GROUPED_PACK_LIMIT = 1 << 24;
__host__ __device__ inline int grouped_order_entry(int i, int cfg, int count) {
  return count <= GROUPED_PACK_LIMIT ? (i | (cfg << 24)) : i;
}

// The configuration of a problem of a table too long for packed order entries.
__device__ __forceinline__ int unpacked_config(const gb_grouped_tuning_t& tuning, const gb_problem_t& p, bool f32) {
  const int c = config_of(tuning, size_class(p.m, p.n));
  F64Tiles t;
  return c != GB_GROUPED_AUTO ? c : f32 ? auto_config_f32(true) : auto_config_f64(p.m, p.n, p.k, &t);
}

__device__ __forceinline__ long long tile_count(const gb_problem_t& p, const TileCfg& c, bool f32) {
  if (p.m <= 0 || p.n <= 0) return 0;
  if (f32) return tiles_along(p.m, c.bm) * tiles_along(p.n, c.bn);
  const F64Tiles t = f64_tiles(c, p.m, p.n);
  return static_cast<long long>(t.tm) * t.tn;
}

// What the prologue decides for a problem: its configuration under the table, with the library's choice
// for a table of enough work or for a small one (auto_config_f32, f64_small), and the bucket of the
// schedule each puts it in.  Kept in the workspace's prefix sums until these are written.
__device__ __forceinline__ int choice_word(int cfg, int bucket, int cfg_small, int bucket_small) {
  return cfg | bucket << 5 | cfg_small << 10 | bucket_small << 15;
}
__device__ __forceinline__ int choice_config(int word, bool small) { return word >> (small ? 10 : 0) & 31; }
__device__ __forceinline__ int choice_bucket(int word, bool small) { return word >> (small ? 15 : 5) & 31; }

// Prologue (one block): the schedule orders the problems by the work of one of their tiles
// (rows x columns x k of what a tile holds, in 32 power-of-two buckets, heaviest first), so that the
// CTAs take tiles of similar length side by side and the short ones fill the tail; it writes the order and
// the exclusive prefix sums of the tiles in that order.
// The order inside a bucket depends on timing, which changes no result (each tile is
// independent).  Each problem's choice is made once: made again for the histogram, the order and with
// 64-bit divisions it was a third of a call on 4000 FP64 problems of 8^3 (65 us, now 45).
// The block has a thread per problem, up to 1024 (grouped_prefix_threads): the sums and the scan take every
// warp through their shuffles and barriers, which was most of the time of a small table (10 FP64 problems
// 8.8 us with 1024 threads, 6.1 with 32; a whole call 17.4, 14.5).  What is left there is latency: table
// loads, the choices' 32-bit divisions, two rounds of atomics.
static int grouped_prefix_threads(int count) {
  int threads = 32;
  while (threads < count && threads < 1024) threads *= 2;
  return threads;
}
__global__ void __launch_bounds__(1024, 1) grouped_prefix_kernel(const gb_problem_t* __restrict__ probs, int count,
                                                              gb_grouped_tuning_t tuning, bool f32, int sms,
                                                              long long large_elems, long long* __restrict__ ws) {
  __shared__ long long sums[4][32];
  __shared__ bool small_table;
  __shared__ int hist[32], start[32];
  long long* offsets = ws;
  int* words = reinterpret_cast<int*>(ws);
  int* order = reinterpret_cast<int*>(grouped_order_words(ws, count));
  const int t = threadIdx.x, threads = static_cast<int>(blockDim.x);
  const bool packed = count <= GROUPED_PACK_LIMIT;   // (a longer table keeps the choice for enough work)
  if (t < 32) hist[t] = 0;
  auto bucket = [](long long held, int64_t k) {
    const long long w = held * (k > 1 ? k : 1);
    const int lg = 63 - __clzll(w > 1 ? w : 1);
    return 31 - (lg > 31 ? 31 : lg);                 // heavy first
  };
  auto held_f32 = [](const gb_problem_t& p, int cfg) {
    const TileCfg c = tile_cfg(cfg);
    return min(p.m, static_cast<int64_t>(c.bm)) * min(p.n, static_cast<int64_t>(c.bn));
  };
  const bool may_be_small = f32 ? packed : f64_may_be_small(count, sms);
  F64Load chosen, least;
  for (int i = t; i < count; i += threads) {
    const gb_problem_t& p = probs[i];
    const int c = config_of(tuning, size_class(p.m, p.n));
    if (f32) {
      const int a = c == GB_GROUPED_AUTO ? auto_config_f32(true) : c, b = c == GB_GROUPED_AUTO ? auto_config_f32(false) : c;
      if (p.m > 0 && p.n > 0) chosen.total += p.m * p.n;   // elements of C
      words[i] = choice_word(a, bucket(held_f32(p, a), p.k), b, bucket(held_f32(p, b), p.k));
    } else {
      F64Tiles ta;
      int a = c, b = c, bucket_b = 0;
      if (c == GB_GROUPED_AUTO) a = auto_config_f64(p.m, p.n, p.k, &ta);
      else ta = f64_tiles(tile_cfg(c), p.m, p.n);
      if (may_be_small) {
        F64Tiles tb = ta;
        if (c == GB_GROUPED_AUTO) {
          b = 0;
          tb = f64_tiles(tile_cfg(0), p.m, p.n);
        }
        chosen.add(ta, p.k);
        least.add(tb, p.k);
        bucket_b = bucket(tb.fm * tb.fn, p.k);
      }
      words[i] = choice_word(a, bucket(ta.fm * ta.fn, p.k), b, bucket_b);
    }
  }
  // The sums over the block, where the choice needs them, in two steps: a warp each, then the first warp.
  bool small = false;
  if (may_be_small) {
    auto combine = [](F64Load& l) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        l.total += __shfl_xor_sync(0xffffffffu, l.total, off);
        l.longest = max(l.longest, __shfl_xor_sync(0xffffffffu, l.longest, off));
      }
    };
    combine(chosen);
    if (!f32) combine(least);
    if ((t & 31) == 0) {
      sums[0][t >> 5] = chosen.total;
      sums[1][t >> 5] = chosen.longest;
      sums[2][t >> 5] = least.total;
      sums[3][t >> 5] = least.longest;
    }
    __syncthreads();
    if (t < 32) {
      const bool there = t < threads / 32;
      chosen.total = there ? sums[0][t] : 0;
      chosen.longest = there ? sums[1][t] : 0;
      least.total = there ? sums[2][t] : 0;
      least.longest = there ? sums[3][t] : 0;
      combine(chosen);
      if (!f32) combine(least);
      if (t == 0) small_table = f32 ? chosen.total < large_elems : f64_small(chosen, least, sms);
    }
  }
  __syncthreads();
  if (may_be_small) small = small_table;
  for (int i = t; i < count; i += threads) atomicAdd(&hist[choice_bucket(words[i], small)], 1);
  __syncthreads();
  if (t < 32) {   // exclusive prefix sums over the 32 buckets
    int run = hist[t];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, run, off);
      if (t >= off) run += v;
    }
    start[t] = run - hist[t];
  }
  __syncthreads();
  for (int i = t; i < count; i += threads) {
    const int w = words[i];
    order[atomicAdd(&start[choice_bucket(w, small)], 1)] = grouped_order_entry(i, choice_config(w, small), count);
  }
  __syncthreads();
  const int per = (count + threads - 1) / threads;
  const int b = t * per, e = min(count, b + per);
  auto tiles_of = [&](int pos) -> long long {
    const int e = order[pos];
    const gb_problem_t& p = probs[packed ? (e & 0xFFFFFF) : e];
    return tile_count(p, tile_cfg(packed ? (e >> 24) : unpacked_config(tuning, p, f32)), f32);
  };
  long long sum = 0;
  for (int i = b; i < e; ++i) sum += tiles_of(i);
  // inclusive scan over the block: inside each warp, then over the warps' totals
  auto scan = [&](long long v) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, v, off);
      if ((t & 31) >= off) v += u;
    }
    return v;
  };
  const long long in_warp = scan(sum);
  if ((t & 31) == 31) sums[0][t >> 5] = in_warp;
  __syncthreads();
  if (t < 32) sums[1][t] = scan(t < threads / 32 ? sums[0][t] : 0);
  __syncthreads();
  const long long end = in_warp + (t >= 32 ? sums[1][(t >> 5) - 1] : 0);
  long long run = end - sum;
  for (int i = b; i < e; ++i) {
    offsets[i] = run;   // offsets[0] = 0: the tile counter's start
    if (i + 1 < e) run += tiles_of(i);
  }
  if (t == threads - 1) offsets[count] = end;
}

// The schedule position of tile w: the last pos with offsets[pos] <= w (problems without
// tiles share their successor's offset), searched from `from` (a position with
// offsets[from] <= w: a CTA's tiles come in increasing order, so its previous tile's position).
// Each warp searches on its own: its 32 lanes probe 32 points of the remaining interval at
// once (never offsets[0]), so 4096 problems take at most 3 rounds of loads instead of the 12 dependent loads of a
// binary search.  Every warp reaches the same position.
__device__ __forceinline__ int schedule_pos(const long long* __restrict__ offsets, int count, long long w, int from) {
  const int lane = threadIdx.x & 31;
  int lo = from, hi = count - 1;   // offsets[lo] <= w holds throughout
  while (lo < hi) {
    const long long span = hi - lo;
    const int p = lo + static_cast<int>((span * (lane + 1) + 31) / 32);   // in (lo, hi]; lane 31: hi
    const unsigned ok = __ballot_sync(0xffffffffu, offsets[p] <= w);   // monotone in the lane
    if (ok == 0u) {
      hi = __shfl_sync(0xffffffffu, p, 0) - 1;
    } else {
      const int L = 31 - __clz(ok);
      const int pl = __shfl_sync(0xffffffffu, p, L);
      const int pn = __shfl_sync(0xffffffffu, p, L < 31 ? L + 1 : 31);
      hi = (L == 31) ? hi : pn - 1;
      lo = pl;
    }
  }
  return lo;
}

// A tile of the schedule: its problem and its place in it.  `lo` is the caller's schedule position.
struct GroupedTile {
  gb_problem_t p;
  TileCfg c;
  int64_t tm, tn;   // tile row and column
};
__device__ __forceinline__ void grouped_find(const gb_problem_t* __restrict__ probs, int count,
                                             const gb_grouped_tuning_t& tuning, bool f32,
                                             const long long* __restrict__ offsets, const int* __restrict__ order,
                                             long long w, int& lo, GroupedTile& t) {
  lo = schedule_pos(offsets, count, w, lo);
  const int e = order[lo];
  const bool packed = count <= GROUPED_PACK_LIMIT;
  t.p = probs[packed ? (e & 0xFFFFFF) : e];
  t.c = tile_cfg(packed ? (e >> 24) : unpacked_config(tuning, t.p, f32));
  // in 32-bit arithmetic (a problem's tile count is below 2^31); the first problem's tiles start at 0
  const int local = static_cast<int>(lo ? w - offsets[lo] : w);
  const int tiles_m = static_cast<int>(tiles_along(t.p.m, t.c.bm));
  const int tn = local / tiles_m;
  t.tm = local - tn * tiles_m;
  t.tn = tn;
}
__device__ __forceinline__ bool alpha_is_zero(const gb_problem_t& p) {
  return (__double_as_longlong(p.alpha) & 0x7FFFFFFFFFFFFFFFll) == 0;
}

constexpr int GROUPED_CTAS = 4;   // resident CTAs an SM, both element types
static_assert(GROUPED_CTAS == F64_CTAS, "grid of the grouped kernels");

// Persistent tile loop: each CTA takes a tile of the schedule, then the next one that no CTA has taken (a
// counter in offsets[0]; its answer is fetched while the tile runs).  Against a fixed stride, where
// the busiest SM of 4096 log-uniform problems gets 3.5% more than its share.  The first tiles go to the
// CTAs from the second quarter of the grid on, which are one to an SM; with the grid's first CTAs, which
// put three on each of four SMs, calls of less than a grid of tiles were slower (f32, 16 problems of
// 300^3 47 -> 40 us, one of 1000^3 96 -> 75, 64 of 128^3 23 -> 19; f64, 100 of 64^3 78 -> 62).
// run(tile, index) may leave its shared memory without a barrier: one follows.
template <class Run>
__device__ __forceinline__ void grouped_loop(const gb_problem_t* __restrict__ probs, int count,
                                             const gb_grouped_tuning_t& tuning, bool f32, long long* __restrict__ ws,
                                             const Run& run) {
  __shared__ long long next_tile[2];   // two slots: one is written again only after another barrier
  const long long* offsets = ws;
  const int* order = reinterpret_cast<const int*>(grouped_order_words(ws, count));
  const long long total = offsets[count];
  int lo = 0, slot = 0;
  const unsigned skip = gridDim.x / GROUPED_CTAS;
  const bool one_each = total <= gridDim.x;   // nothing to hand out
  for (long long w = blockIdx.x + (blockIdx.x < skip ? gridDim.x : 0) - skip; w < total; slot ^= 1) {
    long long next = 0;
    if (threadIdx.x == 0 && !one_each)
      next = gridDim.x + static_cast<long long>(atomicAdd(reinterpret_cast<unsigned long long*>(ws), 1ull));
    GroupedTile t;
    grouped_find(probs, count, tuning, f32, offsets, order, w, lo, t);
    run(t, w);
    if (one_each) return;
    if (threadIdx.x == 0) next_tile[slot] = next;
    __syncthreads();
    w = next_tile[slot];
  }
}

__global__ void __launch_bounds__(F64_THREADS, F64_CTAS)
    grouped_f64_kernel(const gb_problem_t* __restrict__ probs, int count, gb_grouped_tuning_t tuning,
                       long long* __restrict__ ws) {
  __shared__ __align__(16) double smem[F64_SMEM_ELEMS];
  grouped_loop(probs, count, tuning, false, ws, [&](const GroupedTile& t, long long w) {
    const gb_problem_t& p = t.p;
    const F64Tiles ft = f64_tiles(t.c, p.m, p.n);
    const int64_t m0 = t.tm * ft.fm, n0 = t.tn * ft.fn;
    const int r = static_cast<int>(p.m - m0 < ft.fm ? p.m - m0 : ft.fm);
    const int c = static_cast<int>(p.n - n0 < ft.fn ? p.n - n0 : ft.fn);
    if (r <= 0 || c <= 0) return;   // equal tiles can need one fewer
    if (alpha_is_zero(p)) {
      scale_tile<double>(p, m0, n0, r, c, threadIdx.x, F64_THREADS);
      return;
    }
    const F64Chain<false> chain{p.alpha, p.beta, f64_out(__double_as_longlong(p.alpha), __double_as_longlong(p.beta))};
    f64_tile_any(r, c, p.k, static_cast<const double*>(p.A) + m0, 1, p.lda, static_cast<const double*>(p.B) + n0 * p.ldb, 1,
                 p.ldb, chain, static_cast<double*>(p.C) + m0 + n0 * p.ldc, p.ldc, static_cast<int>(w ^ (w >> 2)), smem);
  });
}

// FP32: CTAs of four warps run a tile in pieces of up to 64 x 64 on the packed pairs of
// simt4_tile.cuh: a warp takes a 32 x 32 part, so a piece pads to multiples of 32, and the operands are
// read once per 64 rows or columns.  Independent warps on tiles of their own, as native FP32 runs
// them, were slower here (start: 0.88 ms, now 0.66): warps on tiles of different extents execute different code, and with 64 x 64
// tiles three quarters of their time was waiting for instructions (4096 log-uniform problems 1.1 to
// 1.8 ms; 32 x 32 tiles 0.85 ms, bound by their 4-byte copies).
using GroupedPiece = S4Shape<8, 4, 2, 2>;
__global__ void __launch_bounds__(GroupedPiece::THREADS, GROUPED_CTAS)
    grouped_f32_kernel(const gb_problem_t* __restrict__ probs, int count, gb_grouped_tuning_t tuning,
                       long long* __restrict__ ws) {
  __shared__ __align__(16) uint32_t smem[GroupedPiece::SMEM_BYTES / 4];
  grouped_loop(probs, count, tuning, true, ws, [&](const GroupedTile& t, long long) {
    const gb_problem_t& p = t.p;
    const int64_t m0 = t.tm * t.c.bm, n0 = t.tn * t.c.bn;
    const int rows = static_cast<int>(p.m - m0 < t.c.bm ? p.m - m0 : t.c.bm);
    const int cols = static_cast<int>(p.n - n0 < t.c.bn ? p.n - n0 : t.c.bn);
    if (alpha_is_zero(p)) {
      scale_tile<float>(p, m0, n0, rows, cols, threadIdx.x, GroupedPiece::THREADS);
      return;
    }
    const F32Chain op{static_cast<float>(p.alpha), static_cast<float>(p.beta)};
    for (int j0 = 0; j0 < cols; j0 += 64) {
      for (int i0 = 0; i0 < rows; i0 += 64) {
        const int r = min(64, rows - i0), c = min(64, cols - j0);
        simt4_tile<GroupedPiece, true>(r, c, r, c, p.k, op, static_cast<const uint32_t*>(p.A) + m0 + i0, 1, p.lda,
                                       static_cast<const uint32_t*>(p.B) + (n0 + j0) * p.ldb, 1, p.ldb,
                                       static_cast<uint32_t*>(p.C) + m0 + i0 + (n0 + j0) * p.ldc, 1, p.ldc, smem);
      }
    }
  });
}

gb_grouped_tuning_t grouped_default_tuning(int dtype_bytes) {
  gb_grouped_tuning_t t;
  std::memset(&t, 0, sizeof(t));
  // classes: <=16, <=32, <=64, <=128, <=256, >256
  // The library's choice in every class (auto_config_f32, auto_config_f64).
  (void)dtype_bytes;
  for (int c = 0; c < GB_GROUPED_CLASSES; ++c) t.config[c] = GB_GROUPED_AUTO;
  return t;
}

int grouped_configs(int dtype_bytes) { return dtype_bytes == 8 ? GROUPED_CONFIGS_F64 : GROUPED_CONFIGS_F32; }

int grouped_validate_tuning(int dtype_bytes, const gb_grouped_tuning_t& t) {
  for (int c = 0; c < GB_GROUPED_CLASSES; ++c)
    if (t.config[c] != GB_GROUPED_AUTO && (t.config[c] < 0 || t.config[c] >= grouped_configs(dtype_bytes)))
      return GB_ERR_INVALID_VALUE;
  return GB_OK;
}

static int launch_f64_tiles(const gb_problem_t* d_probs, int count, const gb_grouped_tuning_t& tuning, long long* ws,
                            int sms, cudaStream_t s) {
  grouped_f64_kernel<<<sms * GROUPED_CTAS, F64_THREADS, 0, s>>>(d_probs, count, tuning, ws);
  return GB_OK;
}

static int launch_tiles(int dtype_bytes, const gb_problem_t* d_probs, int count, const gb_grouped_tuning_t& tuning,
                        long long* d_ws, int sms, cudaStream_t s) {
  if (dtype_bytes == 8)
    GB_LAUNCH(GB_KERNEL_GROUPED_GEMM, s, launch_f64_tiles(d_probs, count, tuning, d_ws, sms, s));
  else
    GB_LAUNCH(GB_KERNEL_GROUPED_GEMM, s,
              (grouped_f32_kernel<<<sms * GROUPED_CTAS, GroupedPiece::THREADS, 0, s>>>(d_probs, count, tuning,
                                                                                           d_ws)));
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

int grouped_launch(int dtype_bytes, const gb_problem_t* d_probs, int count, const gb_grouped_tuning_t& tuning,
                   long long* d_offsets, int sms, cudaStream_t s) {
  if (count <= 0) return GB_OK;
  GB_LAUNCH(GB_KERNEL_GROUPED_GEMM, s,
            (grouped_prefix_kernel<<<1, grouped_prefix_threads(count), 0, s>>>(d_probs, count, tuning, dtype_bytes == 4, sms,
                                                      f32_large_elems(sms), d_offsets)));
  GB_CUDA_TRY(cudaGetLastError());
  return launch_tiles(dtype_bytes, d_probs, count, tuning, d_offsets, sms, s);
}

size_t grouped_workspace_bytes(int count) {
  // prefix sums (count + 1), the order (count int32 in (count + 1) / 2 words)
  return (static_cast<size_t>(count) + 1 + (static_cast<size_t>(count) + 1) / 2) * sizeof(long long);
}

// Autotuner: for every size class present, time each configuration on that class's
// problems alone (C redirected to scratch, beta = 0, so the caller's C is untouched) and
// keep the fastest.  Replaces BLASOptions' fixed block sizes (src/blas_options.jl:2-7).
int grouped_autotune(int dtype_bytes, const gb_problem_t* h_probs, int count, int sms, cudaMemPool_t pool,
                     int reps, gb_grouped_tuning_t* out, float* class_ms, cudaStream_t s) {
  gb_grouped_tuning_t best = grouped_default_tuning(dtype_bytes);
  std::vector<std::vector<gb_problem_t>> by_class(GB_GROUPED_CLASSES);
  size_t max_c = 1;
  for (int i = 0; i < count; ++i) {
    const gb_problem_t& p = h_probs[i];
    if (p.m <= 0 || p.n <= 0) continue;
    by_class[size_class(p.m, p.n)].push_back(p);
    max_c = std::max(max_c, static_cast<size_t>(p.m * p.n));
  }
  void* scratch = nullptr;
  gb_problem_t* d_sub = nullptr;
  long long* d_off = nullptr;
  GB_CUDA_TRY(cudaMallocFromPoolAsync(&scratch, max_c * dtype_bytes, pool, s));
  GB_CUDA_TRY(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&d_sub), sizeof(gb_problem_t) * (count + 1), pool, s));
  GB_CUDA_TRY(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&d_off), grouped_workspace_bytes(count), pool, s));
  cudaEvent_t e0, e1;
  GB_CUDA_TRY(cudaEventCreate(&e0));
  GB_CUDA_TRY(cudaEventCreate(&e1));
  int rc = GB_OK;
  for (int c = 0; c < GB_GROUPED_CLASSES && rc == GB_OK; ++c) {
    if (class_ms) class_ms[c] = 0.f;
    auto& v = by_class[c];
    if (v.empty()) continue;
    for (auto& p : v) {
      p.C = scratch;
      p.ldc = p.m;
      p.beta = 0.0;
    }
    if (cudaMemcpyAsync(d_sub, v.data(), v.size() * sizeof(gb_problem_t), cudaMemcpyHostToDevice, s) != cudaSuccess) {
      rc = GB_ERR_CUDA;
      break;
    }
    float best_ms = 1e30f;
    for (int ci = 0; ci <= grouped_configs(dtype_bytes); ++ci) {
      const int cfg = (ci == grouped_configs(dtype_bytes)) ? GB_GROUPED_AUTO : ci;
      gb_grouped_tuning_t t = best;
      t.config[c] = cfg;
      rc = grouped_launch(dtype_bytes, d_sub, static_cast<int>(v.size()), t, d_off, sms, s);   // warm-up
      if (rc) break;
      cudaEventRecord(e0, s);
      for (int r = 0; r < reps; ++r) grouped_launch(dtype_bytes, d_sub, static_cast<int>(v.size()), t, d_off, sms, s);
      cudaEventRecord(e1, s);
      if (cudaEventSynchronize(e1) != cudaSuccess) {
        rc = GB_ERR_CUDA;
        break;
      }
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      ms /= reps;
      if (ms < best_ms) {
        best_ms = ms;
        best.config[c] = cfg;
      }
    }
    if (class_ms) class_ms[c] = best_ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(scratch, s);
  cudaFreeAsync(d_sub, s);
  cudaFreeAsync(d_off, s);
  if (rc == GB_OK) *out = best;
  return rc;
}

}  // namespace gb

// ============================================================ allocation-free variant
//
// For callers that cannot allocate device memory at call time (see gbblas.h): the tile
// prefix sums live in a fixed file-scope device array instead of pool or caller memory.
// Every GPU that loads the library holds this array until the process exits.
namespace gb {

constexpr int GROUPED_NOALLOC_MAX = GB_GROUPED_NOALLOC_MAX;
constexpr int NOALLOC_MAX_DEVICES = 64;

// int64 words of grouped_workspace_bytes(GROUPED_NOALLOC_MAX): 98,305 (768 KiB)
constexpr int GROUPED_NOALLOC_WORDS = GROUPED_NOALLOC_MAX + 1 + (GROUPED_NOALLOC_MAX + 1) / 2;
static __device__ __align__(256) long long g_noalloc_offsets[GROUPED_NOALLOC_WORDS];

// Device address of g_noalloc_offsets per device.  In host code the symbol names a host
// stand-in, so the address is looked up once per device (with that device current) and
// reused; the lookup neither allocates nor launches.
static std::mutex g_noalloc_mu;
static long long* g_noalloc_ptr[NOALLOC_MAX_DEVICES];
static int g_noalloc_sms[NOALLOC_MAX_DEVICES];

static int noalloc_setup(long long** ptr, int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return gb_set_cuda_error(e, "cudaGetDevice");
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return GB_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    int major = 0, minor = 0, n = 0;
    e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return gb_set_cuda_error(e, "device attributes");
    if (major != 10 || minor != 3) return GB_ERR_NO_DEVICE;
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_offsets);
    if (e != cudaSuccess) return gb_set_cuda_error(e, "cudaGetSymbolAddress(g_noalloc_offsets)");
    g_noalloc_sms[dev] = n;
    g_noalloc_ptr[dev] = static_cast<long long*>(p);
  }
  *ptr = g_noalloc_ptr[dev];
  *sms = g_noalloc_sms[dev];
  return GB_OK;
}

int grouped_f64_noalloc(const gb_problem_t* d_probs, int count, const gb_grouped_tuning_t* tuning, cudaStream_t s) {
  if (count < 0 || count > GROUPED_NOALLOC_MAX) return GB_ERR_INVALID_VALUE;
  long long* offsets = nullptr;
  int sms = 0;
  int rc = noalloc_setup(&offsets, &sms);
  if (rc) return rc;
  if (count == 0) return GB_OK;
  const gb_grouped_tuning_t t = tuning ? *tuning : grouped_default_tuning(8);
  rc = grouped_validate_tuning(8, t);
  if (rc) return rc;
  // The prologue rewrites the prefix sums and the order on every call, so nothing needs
  // clearing.
  // Launched directly, not through the timing hooks (which create CUDA events while profiling
  // is on); gb_launch_counts still counts both launches.
  grouped_prefix_kernel<<<1, grouped_prefix_threads(count), 0, s>>>(d_probs, count, t, false, sms, 0, offsets);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return gb_set_cuda_error(e, "grouped prologue launch");
  prof_count(GB_KERNEL_GROUPED_GEMM);
  launch_f64_tiles(d_probs, count, t, offsets, sms, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) return gb_set_cuda_error(e, "grouped launch");
  prof_count(GB_KERNEL_GROUPED_GEMM);
  return GB_OK;
}


// ------------------------------------------------------------------ strided batches
// The table of a strided batch and, as all its problems have one configuration of `tiles` tiles, its
// schedule: the offsets and the order that the prologue would write (`cfg` < 0: the prologue runs).
__global__ void grouped_fill_strided_kernel(gb_problem_t* __restrict__ probs, int count, int64_t M, int64_t N,
                                            int64_t K, int64_t lda, int64_t ldb, int64_t ldc, const char* A,
                                            const char* B, char* C, int64_t sa, int64_t sb, int64_t sc, double alpha,
                                            double beta, int cfg, long long tiles, long long* __restrict__ ws) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  gb_problem_t p;
  p.m = M;
  p.n = N;
  p.k = K;
  p.lda = lda;
  p.ldb = ldb;
  p.ldc = ldc;
  p.A = A + static_cast<int64_t>(i) * sa;
  p.B = B + static_cast<int64_t>(i) * sb;
  p.C = C + static_cast<int64_t>(i) * sc;
  p.alpha = alpha;
  p.beta = beta;
  probs[i] = p;
  if (cfg >= 0) {
    ws[i] = i * tiles;
    if (i == count - 1) ws[count] = count * tiles;
    reinterpret_cast<int*>(grouped_order_words(ws, count))[i] = grouped_order_entry(i, cfg, count);
  }
}

// `count` products of one shape under the default tuning: one launch fills the table and the schedule
// (the one-block prologue took 8 us of a call on 668 products of 10 x 35 x 19), one runs it.
int grouped_strided_launch(int dtype_bytes, gb_problem_t* d_probs, long long* d_ws, int count, int64_t M, int64_t N,
                           int64_t K, int64_t lda, int64_t ldb, int64_t ldc, const void* A, const void* B, void* C,
                           int64_t strideA_bytes, int64_t strideB_bytes, int64_t strideC_bytes, double alpha,
                           double beta, int sms, cudaStream_t s) {
  if (count <= 0) return GB_OK;
  int cfg = -1;
  long long tiles = 0;
  if (count <= GROUPED_PACK_LIMIT) {
    // (M N count >= the line, without the product)
    const bool large = M * N >= (f32_large_elems(sms) + count - 1) / count;
    if (dtype_bytes == 8) {
      F64Tiles t;
      cfg = auto_config_f64(M, N, K, &t);
      const F64Tiles t0 = f64_tiles(tile_cfg(0), M, N);
      F64Load chosen, least;
      chosen.add(t, K, count);
      least.add(t0, K, count);
      if (f64_may_be_small(count, sms) && f64_small(chosen, least, sms)) {
        cfg = 0;
        t = t0;
      }
      tiles = static_cast<long long>(t.tm) * t.tn;
    } else {
      cfg = auto_config_f32(large);
      const TileCfg c = tile_cfg(cfg);
      tiles = ((M + c.bm - 1) / c.bm) * ((N + c.bn - 1) / c.bn);
    }
  }
  const int blocks = (count + 255) / 256;
  grouped_fill_strided_kernel<<<blocks, 256, 0, s>>>(d_probs, count, M, N, K, lda, ldb, ldc,
                                                      static_cast<const char*>(A), static_cast<const char*>(B),
                                                      static_cast<char*>(C), strideA_bytes, strideB_bytes,
                                                      strideC_bytes, alpha, beta, cfg, tiles, d_ws);
  GB_CUDA_TRY(cudaGetLastError());
  const gb_grouped_tuning_t tuning = grouped_default_tuning(dtype_bytes);
  return cfg < 0 ? grouped_launch(dtype_bytes, d_probs, count, tuning, d_ws, sms, s)
                 : launch_tiles(dtype_bytes, d_probs, count, tuning, d_ws, sms, s);
}
}  // namespace gb
