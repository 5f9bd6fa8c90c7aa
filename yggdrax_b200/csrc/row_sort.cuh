// Row finalize of rows up to kCtaRowCap entries: sorted in registers,
// widened and written.  Included by traverse.cu.
//
// A row of n entries is sorted by a group of T threads holding R entries
// each: a warp (T = 32) up to 1,024 entries, 4, 8 or 16 warps above.  Every
// thread sorts its R entries with Batcher's odd-even merge network (R may be
// any size), then blocks of threads are merged: the first step of a merge
// pairs element g of a block with its mirror image, the later ones elements
// half a block apart, so every comparator puts the minimum at the lower
// index and short rows are padded with INT32_MAX.  Partners are in another
// lane (shuffles), in another warp (shared memory) or in the same thread.
//
// What bounds it: instruction issue (0.5 to 0.6 per cycle and scheduler) and
// the shuffles' throughput, not the 12 or 28 bytes an entry moves.  Hence:
//  * R = 3 * 2^k between the powers of two: a row pads to at most 1.5 times
//    its length and to 1.2 times on average (1.4 with powers of two alone).
//  * Entries are read in any order (they are unsorted anyway), so only the
//    sorted ones pass through shared memory, for coalesced writes.
//  * The next row's place is read while this one is sorted.
//  * Rows of 1,025 to 8,192 entries are sorted by groups of a long-row CTA,
//    which takes them when no long row is left (they went through the long
//    rows' bitmap at 22 us a row; by a launch of their own, the octree's rows
//    took 264 + 123 us, together 195).
//  * The classes of a launch run one after the other in one kernel: their
//    tails overlap, and a small tree pays 5 launches instead of 8.
// All row kernels together, against one launch per power of two up to 1,024
// entries and the bitmap above:
//   16,777,216 Plummer, leaf 32 (494 M entries)   4.99 -> 3.94 ms
//   512 sets of 256 to 65,536 (165 M)             1.52 -> 1.05 ms
//    4,194,304 Plummer (octree, 90 M)             0.79 -> 0.61 ms
//    4,194,304 clumps, fixed depth (75 M)         0.57 -> 0.46 ms
//    1,000,003 Plummer (32 M)                     0.33 -> 0.25 ms
// Taken back: ids below 2^23 sorted as fp32 with half of the comparators as
// saturating additions on the full-rate pipe (3.20 against 2.75 ms for the
// warp rows of the first case), and select by comparison (y < v) == lower
// instead of min and max (2.93).
#pragma once
#include "rows.cuh"

namespace ygx {
namespace {

constexpr int kWarpClasses = 10;  // R = 1, 2, 3, 4, 6, 8, 12, 16, 24, 32; 32 R entries
constexpr int kCtaClasses = 6;    // R = 12, 16 of 4, 8, 16 warps
constexpr int kLongClasses = 3;   // longer rows: up to 16,384, up to 65,536, any
constexpr int kRowClasses = kWarpClasses + kCtaClasses + kLongClasses;
constexpr int kRowLists = (kRowClasses + 1) / 2;  // two classes share a list
constexpr int kRowWork = kRowClasses;             // counter: long rows taken
constexpr int kCtaRowCap = 8192;
constexpr int kCtaThreads = 1024;  // CTAs of the rows above 1,024 entries

__device__ __forceinline__ int row_class(int n) {
  constexpr int kMax[kRowClasses - 1] = {32,   64,   96,   128,  192,  256,  384,  512,   768,
                                         1024, 1536, 2048, 3072, 4096, 6144, 8192, 16384, 65536};
  int c = 0;
#pragma unroll
  for (int k = 0; k < kRowClasses - 1; ++k) c += n > kMax[k] ? 1 : 0;
  return c;
}

// Class c's k-th row: even classes fill list c / 2 from the front, odd ones
// from the back (together they hold no more rows than there are).
__device__ __forceinline__ int64_t row_slot(int c, int64_t k, int64_t stride) {
  return (int64_t)(c >> 1) * stride + ((c & 1) ? stride - 1 - k : k);
}

// Rows of two tables in one pass: row r < ta.rows is ta's row r, the others
// are tb's row r - ta.rows.  One global atomic per class and 1,024 rows.
__global__ void __launch_bounds__(256) k_rows_classify(RowTable ta, RowTable tb,
                                                       int32_t* __restrict__ lists,
                                                       int64_t stride,
                                                       uint32_t* __restrict__ counts) {
  constexpr int kU = 4;
  __shared__ unsigned s_n[kRowClasses], s_base[kRowClasses];
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t rows = ta.rows + tb.rows;
  for (int64_t tile = (int64_t)blockIdx.x * 256 * kU; tile < rows;
       tile += (int64_t)gridDim.x * 256 * kU) {
    if (tid < kRowClasses) s_n[tid] = 0u;
    __syncthreads();
    int cls[kU];
    unsigned pos[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int64_t r = tile + u * 256 + tid;
      const int n = r >= rows ? 0 : r < ta.rows ? ta.cnt[r] : tb.cnt[r - ta.rows];
      cls[u] = n > 0 ? row_class(n) : -1;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const unsigned peers = __match_any_sync(0xffffffffu, cls[u]);
      const int leader = __ffs(peers) - 1;
      unsigned base = 0;
      if (lane == leader && cls[u] >= 0) base = atomicAdd(&s_n[cls[u]], (unsigned)__popc(peers));
      base = __shfl_sync(0xffffffffu, base, leader);
      pos[u] = base + __popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (tid < kRowClasses) s_base[tid] = s_n[tid] ? atomicAdd(&counts[tid], s_n[tid]) : 0u;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (cls[u] >= 0)
        lists[row_slot(cls[u], (int64_t)s_base[cls[u]] + pos[u], stride)] =
            (int32_t)(tile + u * 256 + tid);
    __syncthreads();
  }
}

__device__ __forceinline__ void cmp_swap(int32_t& a, int32_t& b) {
  const int32_t x = a, y = b;
  a = min(x, y);
  b = max(x, y);
}

// Batcher's odd-even merge sort of R registers (Knuth, algorithm 5.2.2M, in
// its form for any R): rounds (P, K), P = 1, 2, 4, ..., K = P, P / 2, ..., 1.
template <int R, int P, int K>
__device__ __forceinline__ void batcher(int32_t (&v)[R]) {
  if constexpr (P < R) {
#pragma unroll
    for (int x = K % P; x + K < R; ++x)
      if ((x - K % P) % (2 * K) < K && x / (2 * P) == (x + K) / (2 * P)) cmp_swap(v[x], v[x + K]);
    if constexpr (K > 1) batcher<R, P, K / 2>(v);
    else batcher<R, 2 * P, 2 * P>(v);
  }
}

// A bitonic sequence of R registers, sorted: halvings while R is even, then
// runs of 3.
template <int R>
__device__ __forceinline__ void merge_regs(int32_t (&v)[R]) {
  constexpr int O = R % 3 == 0 ? 3 : 1;
#pragma unroll
  for (int s = R / 2; s >= O; s >>= 1) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((r / s) % 2 == 0) cmp_swap(v[r], v[r + s]);
  }
  if constexpr (O == 3) {
#pragma unroll
    for (int b = 0; b < R; b += 3) {
      cmp_swap(v[b], v[b + 1]);
      cmp_swap(v[b + 1], v[b + 2]);
      cmp_swap(v[b], v[b + 1]);
    }
  }
}

// The threads of one row: T = 32 (a warp) or kW warps with their own named
// barrier.
template <int kW>
struct RowGroup {
  static constexpr int kT = 32 * kW;
  static __device__ __forceinline__ void sync(int id) {
    if constexpr (kW == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kT) : "memory");
  }
};

// One merge step across threads: partner thread t ^ m; mirrored (element r
// with R - 1 - r) or straight.  The thread with bit `hi` of t clear keeps the
// minima.
template <int R, int kW, bool kMirror>
__device__ __forceinline__ void merge_step(int32_t (&v)[R], int t, int m, int hi, int bar,
                                           int32_t* sm) {
  constexpr int kT = 32 * kW;
  const bool lower = (t & hi) == 0;
  if (kW == 1 || m < 32) {
    if constexpr (kMirror) {
#pragma unroll
      for (int r = 0; r < (R + 1) / 2; ++r) {
        const int32_t y0 = __shfl_xor_sync(0xffffffffu, v[R - 1 - r], m);
        if (r != R - 1 - r) {
          const int32_t y1 = __shfl_xor_sync(0xffffffffu, v[r], m);
          v[R - 1 - r] = lower ? min(v[R - 1 - r], y1) : max(v[R - 1 - r], y1);
        }
        v[r] = lower ? min(v[r], y0) : max(v[r], y0);
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int32_t y = __shfl_xor_sync(0xffffffffu, v[r], m);
        v[r] = lower ? min(v[r], y) : max(v[r], y);
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) sm[r * kT + t] = v[r];
    RowGroup<kW>::sync(bar);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int32_t y = sm[(kMirror ? R - 1 - r : r) * kT + (t ^ m)];
      v[r] = lower ? min(v[r], y) : max(v[r], y);
    }
    RowGroup<kW>::sync(bar);
  }
}

// Where row number b of class c is and what it needs (n = 0: no such row).
struct RowAt {
  int64_t off, roff;
  int32_t n, tgt, vbase, lvl;
  bool second;
};
__device__ __forceinline__ RowAt row_at(const RowTable& ta, const RowTable& tb, int32_t g) {
  RowAt a;
  a.second = g >= ta.rows;
  const RowTable& T = a.second ? tb : ta;
  const int32_t r = a.second ? g - (int32_t)ta.rows : g;
  a.off = T.off[r];
  a.roff = T.roff ? T.roff[r] : a.off;
  a.n = T.cnt[r];
  a.vbase = T.rbase ? T.rbase[r] : 0;
  a.lvl = T.lvl ? T.lvl[r] : 0;
  a.tgt = r - a.vbase;
  return a;
}

// Rows of class c, each by this group: thread t of kT, `sm` its R * kT + R *
// kW words of shared memory (not restrict: other threads write it, which a
// compiler may take a barrier not to do).  A warp takes rows first, first +
// step, ...; larger groups take the next one left (counter `work`), since
// their CTA may come to them late, from a long row.
template <int R, int kW, typename Idx>
__device__ __forceinline__ void sort_rows(const RowTable& ta, const RowTable& tb,
                                          const int32_t* __restrict__ lists, int64_t stride,
                                          const uint32_t* __restrict__ counts, int c,
                                          uint32_t first, uint32_t step, uint32_t* work,
                                          uint32_t* s_next, int t, int bar, int32_t* sm) {
  constexpr int kT = 32 * kW;
  const uint32_t rows = counts[c];
  if (rows == 0) return;
  if constexpr (kW > 1) {
    if (t == 0) *s_next = atomicAdd(work, 1u);
    RowGroup<kW>::sync(bar);
    first = *s_next;  // written again only after the row's first exchange
  }
  if (first >= rows) return;
  RowAt a = row_at(ta, tb, lists[row_slot(c, first, stride)]);
  int32_t g = 0;
  if (kW == 1 && first + step < rows) g = lists[row_slot(c, first + step, stride)];
  for (uint32_t b = first; b < rows;) {
    int32_t v[R];
    {
      const int32_t* __restrict__ raw = (a.second ? tb : ta).raw + a.roff + t;
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = r * kT + t < a.n ? raw[r * kT] : INT32_MAX;
    }
    RowAt next = a;
    uint32_t taken = 0;
    if constexpr (kW > 1) {
      if (t == 0) taken = atomicAdd(work, 1u);
    } else if (b + step < rows) {
      next = row_at(ta, tb, g);
      if (b + 2 * step < rows && b + 2 * step > b)
        g = lists[row_slot(c, (int64_t)b + 2 * step, stride)];
    }
    batcher<R, 1, 1>(v);
#pragma unroll
    for (int p = 1; p < kT; p <<= 1) {  // blocks of p threads -> 2 p
      merge_step<R, kW, true>(v, t, 2 * p - 1, p, bar, sm);
#pragma unroll
      for (int j = p >> 1; j > 0; j >>= 1) merge_step<R, kW, false>(v, t, j, j, bar, sm);
      merge_regs<R>(v);
    }
    // through shared memory (a word skipped every 32: few conflicts)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = t * R + r;
      sm[e + (e >> 5)] = v[r];
    }
    if constexpr (kW > 1) {
      if (t == 0) *s_next = taken;
    }
    RowGroup<kW>::sync(bar);
    if constexpr (kW > 1) {
      b = *s_next;
      if (b < rows) next = row_at(ta, tb, lists[row_slot(c, b, stride)]);
    } else {
      b += step;
    }
    const RowTable& T = a.second ? tb : ta;
    Idx* __restrict__ vals = static_cast<Idx*>(T.vals) + a.off + t;
    const int32_t* out = sm + t + (t >> 5);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r * kT + t < a.n) vals[r * kT] = (Idx)(out[r * (kT + kW)] - a.vbase);
    if (T.tgts) {
      Idx* __restrict__ tgts = static_cast<Idx*>(T.tgts) + a.off + t;
      Idx* __restrict__ lvls = static_cast<Idx*>(T.lvls) + a.off + t;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r * kT + t < a.n) {
          tgts[r * kT] = (Idx)a.tgt;
          lvls[r * kT] = (Idx)a.lvl;
        }
    }
    RowGroup<kW>::sync(bar);
    a = next;
  }
}

// A warp per row: kTier 0 up to 256 entries, 1 up to 512, 2 up to 1,024.  The
// tiers differ in the CTAs per SM that their registers allow without spills
// (6 or 8 for tier 0: 512 sets of 256 to 65,536 particles 468 -> 482, 535 us;
// 3 for tier 1: no difference; 2 for tier 2: 89 -> 103 us).
constexpr int row_tier_ctas(int tier) { return tier == 0 ? 5 : tier == 1 ? 4 : 3; }
template <typename Idx, int kTier>
__global__ void __launch_bounds__(256, row_tier_ctas(kTier))
    k_rows_warp(RowTable ta, RowTable tb, const int32_t* __restrict__ lists, int64_t stride,
                const uint32_t* __restrict__ counts) {
  constexpr int kWords = 33 * (8 << kTier);
  __shared__ int32_t s_rows[8][kWords];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t first = blockIdx.x * 8 + w, step = gridDim.x * 8;
  int32_t* sm = s_rows[w];
#define YGX_ROWS(R, C)                                                                  \
  sort_rows<R, 1, Idx>(ta, tb, lists, stride, counts, C, first, step, nullptr, nullptr, \
                       lane, 0, sm)
  if constexpr (kTier == 2) {
    YGX_ROWS(32, 9);
    YGX_ROWS(24, 8);
  } else if constexpr (kTier == 1) {
    YGX_ROWS(16, 7);
    YGX_ROWS(12, 6);
  } else {
    YGX_ROWS(8, 5);
    YGX_ROWS(6, 4);
    YGX_ROWS(4, 3);
    YGX_ROWS(3, 2);
    YGX_ROWS(2, 1);
    YGX_ROWS(1, 0);
  }
#undef YGX_ROWS
}

// The classes of 1,025 to kCtaRowCap entries, by groups of a CTA of kCtaThreads
// threads (every thread calls it): 16, 8 or 4 warps a row.  sm: kCtaWords words.
constexpr int kCtaWords = kCtaThreads / 32 * 33 * 16;
template <typename Idx>
__device__ __forceinline__ void sort_cta_rows(const RowTable& ta, const RowTable& tb,
                                              const int32_t* __restrict__ lists, int64_t stride,
                                              uint32_t* counts, int32_t* sm, uint32_t* s_next) {
#define YGX_ROWS(R, W, C)                                                                    \
  {                                                                                          \
    const int q = threadIdx.x / (32 * W);                                                    \
    sort_rows<R, W, Idx>(ta, tb, lists, stride, counts, C, 0, 0,                             \
                         counts + kRowWork + 1 + (C - kWarpClasses), s_next + q,             \
                         threadIdx.x % (32 * W), 1 + q, sm + q * (W * 33 * 16));             \
    __syncthreads();                                                                         \
  }
  YGX_ROWS(16, 16, 15)
  YGX_ROWS(12, 16, 14)
  YGX_ROWS(16, 8, 13)
  YGX_ROWS(12, 8, 12)
  YGX_ROWS(16, 4, 11)
  YGX_ROWS(12, 4, 10)
#undef YGX_ROWS
}

}  // namespace
}  // namespace ygx
