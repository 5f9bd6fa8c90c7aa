// Dense level-major M2L buffers (yggdrax/dense_interactions.py:34-254,
// yggdrax/_geometry_impl.py:342-420) and class-major grouped far pairs
// (yggdrax/grouped_interactions.py:75-200).
//
// Dense: one thread per (level, slot, interaction) writes the padded source
// id, mask, count and target-minus-source displacement; the level-major
// geometry is one thread per (level, slot).  Grouped: the class key of every
// pair (target level, source level, displacement in target-level cells, in
// float64 exactly as the reference's NumPy code computes it) is packed
// into a <= 128-bit unsigned key (fields shifted to be non-negative, widths
// from their ranges), sorted stably, and the classes are the runs of equal
// keys.
//
// The sort is what this costs.  A key of more than 64 bits is sorted by its
// top 64 alone (8 passes of the onesweep sort); the pairs that tie there out of
// order are ordered by their remaining bits in place (2% of a Plummer tree's
// pairs, most of a lattice's: GroupTies).  A few bits more than 64 are sorted first.
// Beside the sort, the fields are recomputed where they are needed instead of
// stored (two 62-byte passes over the pairs became one of 24 bytes), each pair
// travels as one 16-byte record, and the class tables are decoded from the
// sorted keys.  12,410,462 pairs, 97-bit keys (the far list of 1,048,576
// Plummer particles): 3.1 -> 2.1 ms.
#include "common.cuh"
#include "scan_seg.cuh"
#include "sort.cuh"

namespace ygx {

namespace {

__global__ void k_level_major(const int32_t* __restrict__ nbl32, const void* level_offsets,
                              int index_bits, int num_levels, int64_t max_nodes,
                              const float* __restrict__ center,
                              const float* __restrict__ half_extent,
                              const float* __restrict__ radius,
                              const float* __restrict__ max_extent, float* __restrict__ o_center,
                              float* __restrict__ o_half, float* __restrict__ o_radius,
                              float* __restrict__ o_max, void* o_nodes) {
  const int64_t n = (int64_t)num_levels * max_nodes;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t l = q / max_nodes, m = q % max_nodes;
    const int64_t start = load_idx(level_offsets, index_bits, l);
    const int64_t count = load_idx(level_offsets, index_bits, l + 1) - start;
    const int64_t node = m < count ? (int64_t)nbl32[start + m] : -1;
    if (node >= 0) {
      for (int a = 0; a < 3; ++a) {
        o_center[3 * q + a] = center[3 * node + a];
        o_half[3 * q + a] = half_extent[3 * node + a];
      }
      o_radius[q] = radius[node];
      o_max[q] = max_extent[node];
    } else {
      for (int a = 0; a < 3; ++a) o_center[3 * q + a] = o_half[3 * q + a] = 0.0f;
      o_radius[q] = o_max[q] = 0.0f;
    }
    store_idx(o_nodes, index_bits, q, node);
  }
}

__global__ void k_dense_m2l(const void* node_idx, int index_bits, int64_t slots, int64_t K,
                            const void* counts, const void* offsets, const void* sources,
                            const float* __restrict__ center, int64_t total, void* o_src,
                            bool* __restrict__ o_mask, void* o_counts, float* __restrict__ o_disp) {
  const int64_t n = slots * K;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t sl = q / K, k = q % K;
    const int64_t node = load_idx(node_idx, index_bits, sl);
    int64_t src = -1, cnt = 0;
    float d[3] = {0.0f, 0.0f, 0.0f};
    if (node >= 0 && node < total) {
      cnt = load_idx(counts, index_bits, node);
      if (k < cnt) {
        src = load_idx(sources, index_bits, load_idx(offsets, index_bits, node) + k);
        const int64_t s = src < 0 ? 0 : (src >= total ? total - 1 : src);
        for (int a = 0; a < 3; ++a) d[a] = __fsub_rn(center[3 * node + a], center[3 * s + a]);
      }
    }
    store_idx(o_src, index_bits, q, src);
    o_mask[q] = node >= 0 && k < cnt;
    for (int a = 0; a < 3; ++a) o_disp[3 * q + a] = d[a];
    if (k == 0) store_idx(o_counts, index_bits, sl, node >= 0 ? cnt : 0);
  }
}

// cell size of a level: max(extent / max(2^level, 1), 1e-12) in float64
__device__ __forceinline__ double cell_of(double extent, int level) {
  const double denom = ldexp(1.0, level);
  const double c = extent / (denom > 1.0 ? denom : 1.0);
  return c > 1e-12 ? c : 1e-12;
}

// The cell sizes of levels 0..63 (a CTA's copy: a division and a scaling less
// per axis and pair); deeper levels, which tied codes can make, compute theirs.
struct CellTable {
  double cell[64][3];
  __device__ void fill(const double ext[3]) {
    for (int k = threadIdx.x; k < 64 * 3; k += blockDim.x)
      cell[k / 3][k % 3] = cell_of(ext[k % 3], k / 3);
    __syncthreads();
  }
  __device__ __forceinline__ double at(int level, int a, const double ext[3]) const {
    return (unsigned)level < 64u ? cell[level][a] : cell_of(ext[a], level);
  }
};

// Fields of a pair: target level, source level, displacement index
// rint((c_t - c_s) / cell(target level)) per axis, in float64.
struct GroupPairs {
  const void *src, *tgt;
  int index_bits;
  int64_t P;
  const int32_t* level32;
  const float* center;
  double ext[3];
};
__device__ __forceinline__ void group_fields(const GroupPairs& g, const CellTable& cells,
                                             int64_t s, int64_t t, int v[5]) {
  v[0] = g.level32[t];
  v[1] = g.level32[s];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double delta = (double)g.center[3 * t + a] - (double)g.center[3 * s + a];
    v[2 + a] = (int)rint(delta / cells.at(v[0], a, g.ext));
  }
}

// Minima / maxima of the fields (for the key widths), a CTA's in shared memory
// first: with an atomic per warp on the same ten words the kernel waited for them
// (3.5 M pairs 92 -> 62 us).
__global__ void k_group_ranges(const GroupPairs g, int* __restrict__ fmin,
                               int* __restrict__ fmax) {
  __shared__ CellTable cells;
  __shared__ int s_lo[5], s_hi[5];
  if (threadIdx.x < 5) {
    s_lo[threadIdx.x] = INT_MAX;
    s_hi[threadIdx.x] = INT_MIN;
  }
  cells.fill(g.ext);
  int lo[5], hi[5];
  for (int f = 0; f < 5; ++f) {
    lo[f] = INT_MAX;
    hi[f] = INT_MIN;
  }
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < g.P;
       p += (int64_t)gridDim.x * blockDim.x) {
    int v[5];
    group_fields(g, cells, load_idx(g.src, g.index_bits, p), load_idx(g.tgt, g.index_bits, p), v);
    for (int f = 0; f < 5; ++f) {
      lo[f] = v[f] < lo[f] ? v[f] : lo[f];
      hi[f] = v[f] > hi[f] ? v[f] : hi[f];
    }
  }
  for (int f = 0; f < 5; ++f) {
    for (int o = 16; o > 0; o >>= 1) {
      const int a = __shfl_xor_sync(0xffffffffu, lo[f], o);
      const int b = __shfl_xor_sync(0xffffffffu, hi[f], o);
      lo[f] = a < lo[f] ? a : lo[f];
      hi[f] = b > hi[f] ? b : hi[f];
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&s_lo[f], lo[f]);
      atomicMax(&s_hi[f], hi[f]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    atomicMin(&fmin[threadIdx.x], s_lo[threadIdx.x]);
    atomicMax(&fmax[threadIdx.x], s_hi[threadIdx.x]);
  }
}

// The key: fields from most (0) to least (4) significant; `top` is its upper
// 64 bits (all of it, if it has no more), `low` the `cut` bits below.
struct KeyLayout {
  int shift[5];  // bit position of each field in the 128-bit key
  int width[5];
  int fmin[5];
  int cut;
};
struct __align__(16) GroupRec {
  uint64_t low;
  int32_t s, t;
};

__global__ void k_group_pack(const GroupPairs g, KeyLayout kl, KeyLayout* __restrict__ kl_out,
                             uint64_t* __restrict__ top, GroupRec* __restrict__ rec) {
  __shared__ CellTable cells;
  cells.fill(g.ext);
  if (blockIdx.x == 0 && threadIdx.x == 0) *kl_out = kl;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < g.P;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = load_idx(g.src, g.index_bits, p), t = load_idx(g.tgt, g.index_bits, p);
    int v[5];
    group_fields(g, cells, s, t, v);
    unsigned __int128 k = 0;
    for (int f = 0; f < 5; ++f)
      k |= (unsigned __int128)(uint64_t)((int64_t)v[f] - (int64_t)kl.fmin[f]) << kl.shift[f];
    top[p] = (uint64_t)(k >> kl.cut);
    GroupRec r;
    r.low = kl.cut > 0 ? (uint64_t)k & (~0ull >> (64 - kl.cut)) : 0ull;
    r.s = (int32_t)s;
    r.t = (int32_t)t;
    rec[p] = r;
  }
}

// Pairs sorted by `top` whose runs of equal words are not yet in the order of
// `low`.  Three kernels, since runs differ: a Plummer tree's hold two to a few
// hundred pairs of different classes, a lattice's thousands of one or a few.
//  * k_group_ties copies the order, ranks the runs that lie within a warp's 32
//    positions, and lists descents of the others (a pair whose `low` is below that
//    of the pair before it): every run that has any gets one listed, a long one
//    once in a while.  A run without, such as one class of any size, is in order.
//  * k_group_short takes the descents, a warp each: the first listed of a run of at
//    most kTieMax pairs ranks the run against itself; longer runs are listed.
//  * k_group_long sorts those, a CTA per run, by 8-bit digits of `low`.  Runs
//    longer than 1/64 of the list (fewer than 64 there are) go through the onesweep
//    sort one by one: a CTA's sort of so many pairs costs what the passes over the
//    whole list do.
// Ranking every run, and sorting the whole list twice more if one was longer than
// 1,024 pairs, took the grouping of a lattice of 128^3 points, leaf 4 (55.8 M pairs,
// 76 bits), to 23.0 ms; 13.4 so.
constexpr int kTieMax = 256;
struct GroupTies {
  const uint64_t* top;
  const GroupRec* rec;
  int64_t P;
  uint32_t* perm;     // sorted position -> pair, read only until k_group_long
  uint32_t* out;      // the same in order
  uint32_t* descents;
  uint2* runs;        // first position, pairs
  // one per kTieMax positions, zeroed: no two longer runs start in one (claims),
  // or reach into it by more than that (seen)
  uint32_t *claims, *seen;
  int* count;         // huge runs; descents; long runs; long runs taken
  uint2* huge;        // kHugeRuns: runs of more than `longest` pairs
  int64_t longest;
};
constexpr int kHugeRuns = 64;
// Up to this many bits below the top word, one pass, are sorted first instead: the
// pass, its keys and the gather of the top words cost what a look at the ties does
// (37 M jittered lattice pairs, 71 bits: 7.0 ms the call, 6.4 with the ties) and
// nothing more where many tie (11 M pairs of 60,000 points of which a third coincide,
// 67 bits: 2.1 and 2.5).  Two passes cost a Plummer tree twice its ties.
constexpr int kLowFirst = 8;

__global__ void k_group_ties(const GroupTies g) {
  const int lane = threadIdx.x & 31;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < g.P;
       i0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = i0 + lane;
    const bool live = i < g.P;
    const uint64_t t = live ? g.top[i] : 0ull;
    const uint32_t p = live ? g.perm[i] : 0u;
    uint64_t before = __shfl_up_sync(0xffffffffu, t, 1);
    if (lane == 0 && live && i > 0) before = g.top[i - 1];
    const bool tied = live && i > 0 && before == t;
    const unsigned ties = __ballot_sync(0xffffffffu, tied);
    const bool next = (ties >> lane) & 2u;  // the pair after this one is tied to it
    const uint64_t low = tied || next ? g.rec[p].low : 0ull;
    uint64_t low_before = __shfl_up_sync(0xffffffffu, low, 1);
    if (lane == 0 && tied) low_before = g.rec[g.perm[i - 1]].low;
    const bool descent = tied && low < low_before;
    const unsigned m = __ballot_sync(0xffffffffu, descent);
    int64_t at = i;
    if (m) {
      // a run within these 32 positions is ranked here
      const bool on = lane == 31 && i + 1 < g.P && g.top[i + 1] == t;
      const unsigned open = __ballot_sync(0xffffffffu, on) ? ~0u : 0u;
      const unsigned heads = ~ties, upto = heads & (2u * (1u << lane) - 1u);
      const int start = upto ? 31 - __clz(upto) : -1;  // -1: it comes from before
      const bool inside = start >= 0 && (!open || (heads & ~(2u * (1u << lane) - 1u)));
      int rank = 0;
      for (int j = 0; j < 32; ++j) {
        const uint64_t v = __shfl_sync(0xffffffffu, low, j);
        const int s = __shfl_sync(0xffffffffu, start, j);
        rank += s == start && (v < low || (v == low && j < lane));
      }
      if (inside) at = i0 + start + rank;
      // of the others, one descent a run, and one per kTieMax positions further
      // than that from its run's start
      const unsigned same = __match_any_sync(0xffffffffu, descent && !inside ? start : 32 + lane);
      bool list = descent && !inside && lane == __ffs(same) - 1;
      if (list && i >= kTieMax && g.top[i - kTieMax] == t)
        list = atomicExch(&g.seen[i / kTieMax], 1u) == 0u;
      const unsigned ml = __ballot_sync(0xffffffffu, list);
      int base = 0;
      if (lane == 0 && ml) base = atomicAdd(&g.count[1], __popc(ml));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (list) g.descents[(uint32_t)base + __popc(ml & ((1u << lane) - 1u))] = (uint32_t)i;
    }
    if (live) g.out[at] = p;
  }
}

// The end of the run that holds position d: how far its word goes on in
// direction `dir`, found by 31 doublings at once, then by 32 probes a step.
__device__ __forceinline__ int64_t group_reach(const GroupTies& g, int64_t d, int dir, int lane) {
  const uint64_t w = g.top[d];
  auto in = [&](int64_t k) {
    const int64_t q = d + dir * k;
    return q >= 0 && q < g.P && g.top[q] == w;
  };
  const unsigned m = __ballot_sync(0xffffffffu, lane < 31 && in((int64_t)1 << lane));
  const int n = __ffs(~m) - 1;  // 2^0 .. 2^(n-1) are in the run
  int64_t lo = n > 0 ? (int64_t)1 << (n - 1) : 0, hi = (int64_t)1 << n;  // in, out
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 31) / 32, k = lo + step * (lane + 1);
    const unsigned q = __ballot_sync(0xffffffffu, k < hi && in(k));
    const int c = __ffs(~q) - 1;  // (bit 31 clear: lo + 32 step >= hi)
    const int64_t at = lo + step * c;
    hi = at + step < hi ? at + step : hi;
    lo = at;
  }
  return lo;
}

__global__ void k_group_short(const GroupTies g) {
  const int lane = threadIdx.x & 31;
  const int warps = (int)(gridDim.x * blockDim.x) >> 5;
  const uint32_t n_desc = (uint32_t)g.count[1];
  for (uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < n_desc; e += warps) {
    const int64_t d = g.descents[e];
    const int64_t a = d - group_reach(g, d, -1, lane), n = d - a + group_reach(g, d, 1, lane) + 1;
    if (n > kTieMax) {
      if (lane == 0 && atomicExch(&g.claims[a / kTieMax], 1u) == 0u) {
        if (n > g.longest) g.huge[atomicAdd(&g.count[0], 1)] = make_uint2((uint32_t)a, (uint32_t)n);
        else g.runs[atomicAdd(&g.count[2], 1)] = make_uint2((uint32_t)a, (uint32_t)n);
      }
      continue;
    }
    // the run's first descent?  (the first is listed: it is its warp's first of
    // the run, and less than kTieMax behind the run's start)
    bool first = true;
    for (int64_t q0 = a; q0 + 1 < d && first; q0 += 31) {
      const int64_t q = q0 + lane;
      const uint64_t low = q < d ? g.rec[g.perm[q]].low : ~0ull;
      const uint64_t next = __shfl_down_sync(0xffffffffu, low, 1);
      first = !__any_sync(0xffffffffu, lane < 31 && next < low);
    }
    if (!first) continue;
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int k = e0 + lane;
      const uint32_t mine = k < n ? g.perm[a + k] : 0u;
      const uint64_t low = k < n ? g.rec[mine].low : 0ull;
      int rank = 0;
      for (int j0 = 0; j0 < n; j0 += 32) {
        const uint64_t theirs = j0 + lane < n ? g.rec[g.perm[a + j0 + lane]].low : 0ull;
        const int m = n - j0 < 32 ? (int)(n - j0) : 32;
        for (int j = 0; j < m; ++j) {
          const uint64_t v = __shfl_sync(0xffffffffu, theirs, j);
          rank += v < low || (v == low && j0 + j < k);
        }
      }
      if (k < n) g.out[a + rank] = mine;
    }
  }
}

// Least digit first, stable: the run's histogram, then its pairs 4,096 at a time --
// 256 a warp, eight of its lanes' in flight --, each at its digit's place plus its
// rank among the chunk's.  A digit that all pairs share moves nothing.  Bound by the
// gathers of `low` and the chunks' barriers: 140,000 pairs, one digit, 409 us with
// 512 at a time, 234 so.
constexpr int kLongThreads = 512;
constexpr int kLongWarps = kLongThreads / 32;
constexpr int kLongItems = 8;
__global__ void __launch_bounds__(kLongThreads) k_group_long(const GroupTies g, int cut) {
  __shared__ uint32_t s_bin[256], s_all[256];
  __shared__ uint16_t s_warp[kLongWarps][256];
  __shared__ uint32_t s_run;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t n_runs = (uint32_t)g.count[2];
  while (true) {
    if (tid == 0) s_run = (uint32_t)atomicAdd(&g.count[3], 1);
    __syncthreads();
    if (s_run >= n_runs) break;
    const uint2 run = g.runs[s_run];
    const uint32_t n = run.y;
    uint32_t *src = g.perm + run.x, *dst = g.out + run.x;
    for (int shift = 0; shift < cut; shift += 8) {
      auto digit = [&](uint32_t p) { return (int)(g.rec[p].low >> shift) & 255; };
      if (tid < 256) s_bin[tid] = 0u;
      __syncthreads();
      for (uint32_t k = tid; k < n; k += kLongThreads * 4) {
        uint32_t p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          p[u] = k + u * kLongThreads < n ? __ldcg(src + k + u * kLongThreads) : 0u;
        int d[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = digit(p[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k + u * kLongThreads < n) atomicAdd(&s_bin[d[u]], 1u);
      }
      __syncthreads();
      if (__syncthreads_or(tid < 256 && s_bin[tid] == n)) continue;
      if (warp == 0) {  // exclusive sums, 8 digits a lane
        uint32_t v[8], sum = 0;
        for (int j = 0; j < 8; ++j) {
          v[j] = sum;
          sum += s_bin[8 * lane + j];
        }
        uint32_t incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t w = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += w;
        }
        for (int j = 0; j < 8; ++j) s_bin[8 * lane + j] = incl - sum + v[j];
      }
      for (uint32_t c0 = 0; c0 < n; c0 += kLongThreads * kLongItems) {
        for (int k = tid; k < kLongWarps * 256; k += kLongThreads) (&s_warp[0][0])[k] = 0;
        const uint32_t k0 = c0 + warp * (32 * kLongItems) + lane;
        uint32_t p[kLongItems];
        int d[kLongItems];
        uint16_t rank[kLongItems];
#pragma unroll
        for (int u = 0; u < kLongItems; ++u) p[u] = k0 + 32 * u < n ? __ldcg(src + k0 + 32 * u) : 0u;
#pragma unroll
        for (int u = 0; u < kLongItems; ++u) d[u] = k0 + 32 * u < n ? digit(p[u]) : 256;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kLongItems; ++u) {
          const unsigned peers = __match_any_sync(0xffffffffu, d[u]);
          const int before = __popc(peers & ((1u << lane) - 1u));
          const uint16_t held = d[u] < 256 ? s_warp[warp][d[u]] : (uint16_t)0;
          rank[u] = (uint16_t)(held + before);
          __syncwarp();
          if (d[u] < 256 && before == 0) s_warp[warp][d[u]] = (uint16_t)(held + __popc(peers));
          __syncwarp();
        }
        __syncthreads();
        if (tid < 256) {
          uint32_t sum = 0;  // counts of the warps before, and the chunk's
          for (int w = 0; w < kLongWarps; ++w) {
            const uint32_t c = s_warp[w][tid];
            s_warp[w][tid] = (uint16_t)sum;
            sum += c;
          }
          s_all[tid] = sum;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kLongItems; ++u)
          if (d[u] < 256) dst[s_bin[d[u]] + s_warp[warp][d[u]] + rank[u]] = p[u];
        __syncthreads();
        if (tid < 256) s_bin[tid] += s_all[tid];
      }
      __syncthreads();
      uint32_t* x = src;
      src = dst;
      dst = x;
    }
    if (src == g.perm + run.x)  // nothing moved (out holds the copy), or an even number of times
      for (uint32_t k = tid; k < n; k += kLongThreads) dst[k] = __ldcg(src + k);
    __syncthreads();
  }
}

__global__ void k_group_low_keys(const GroupRec* __restrict__ rec, int64_t P,
                                 uint64_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = rec[i].low;
}
__global__ void k_gather_u64(const uint64_t* __restrict__ in, const uint32_t* __restrict__ perm,
                             int64_t n, uint64_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[perm[i]];
}
__global__ void k_group_run_keys(const GroupRec* __restrict__ rec,
                                 const uint32_t* __restrict__ perm, int64_t n,
                                 uint64_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = rec[perm[i]].low;
}

// Records in sorted order and the run starts (classes), with the number of
// runs that start in each tile.
__global__ void __launch_bounds__(kScanThreads)
    k_group_heads(const uint64_t* __restrict__ top, const uint32_t* __restrict__ perm,
                  const GroupRec* __restrict__ rec, int64_t P, GroupRec* __restrict__ sorted,
                  uint8_t* __restrict__ head, int64_t* __restrict__ tile_heads,
                  const int* __restrict__ skip) {
  // a huge run is not in order yet
  if (skip && *skip) return;
  __shared__ int64_t s_warp[kScanThreads / 32];
  const int lane = threadIdx.x & 31;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  int64_t heads = 0;
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
    GroupRec r{0ull, 0, 0};
    uint64_t t = 0;
    if (i < P) {
      r = rec[perm[i]];
      t = top[i];
      sorted[i] = r;
    }
    uint64_t pl = __shfl_up_sync(0xffffffffu, r.low, 1);
    if (lane == 0 && i > 0 && i < P) pl = rec[perm[i - 1]].low;
    if (i < P) {
      const bool h = i == 0 || top[i - 1] != t || pl != r.low;
      head[i] = h;
      heads += h;
    }
  }
  heads = seg_block_sum(heads, s_warp);
  if (threadIdx.x == 0) tile_heads[blockIdx.x] = heads;
}

__global__ void __launch_bounds__(kScanThreads)
    k_group_emit(const uint64_t* __restrict__ top, const uint32_t* __restrict__ perm,
                 const GroupRec* __restrict__ sorted, const uint8_t* __restrict__ head,
                 const int64_t* __restrict__ tile_off, int64_t P, int index_bits, double ex,
                 double ey, double ez, const KeyLayout* __restrict__ layout,
                 int32_t* __restrict__ class_keys, float* __restrict__ class_disp,
                 void* class_offsets, void* class_sources, void* class_targets,
                 void* class_ids) {
  __shared__ KeyLayout kl;
  __shared__ int s_warp[kScanThreads / 32];
  if (threadIdx.x == 0) kl = *layout;
  __syncthreads();
  const double ext[3] = {ex, ey, ez};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  int64_t before = tile_off[blockIdx.x];
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
    const bool h = i < P && head[i];
    const unsigned mask = __ballot_sync(0xffffffffu, h);
    if (lane == 0) s_warp[warp] = __popc(mask);
    __syncthreads();
    int mine = 0, all = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) {
      if (w < warp) mine += s_warp[w];
      all += s_warp[w];
    }
    __syncthreads();
    if (i < P) {
      // the class that this pair belongs to: heads up to and including it
      const int64_t cls =
          before + mine + __popc(mask & ((2u << lane) - 1u)) - 1;
      const GroupRec r = sorted[i];
      store_idx(class_sources, index_bits, i, r.s);
      store_idx(class_targets, index_bits, i, r.t);
      // class ids as np.searchsorted(class_starts, arange(n)) (side "left",
      // grouped_interactions.py:163) gives them: a pair that is not the first
      // of its class gets the next class's id (a quirk kept for parity)
      store_idx(class_ids, index_bits, perm[i], h ? cls : cls + 1);
      if (h) {
        store_idx(class_offsets, index_bits, cls, i);
        const unsigned __int128 key = ((unsigned __int128)top[i] << kl.cut) | r.low;
        int v[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
          const uint64_t w = (uint64_t)(key >> kl.shift[f]);
          v[f] = (int)((int64_t)(kl.width[f] > 0 ? w & (~0ull >> (64 - kl.width[f])) : 0ull) +
                       (int64_t)kl.fmin[f]);
          class_keys[5 * cls + f] = v[f];
        }
#pragma unroll
        for (int a = 0; a < 3; ++a)
          class_disp[3 * cls + a] = __double2float_rn((double)v[2 + a] * cell_of(ext[a], v[0]));
      }
      if (i == P - 1) store_idx(class_offsets, index_bits, cls + 1, P);
    }
    before += all;
    if (base + (int64_t)(k + 1) * kScanThreads >= P) break;
  }
}

struct GroupScratch {
  int* fmin;
  int* fmax;
  int* counts;           // GroupTies::count
  uint2* huge;           // GroupTies::huge
  KeyLayout* layout;
  uint64_t* top;         // pair order
  uint64_t* top_sorted;
  GroupRec* rec;         // pair order
  GroupRec* rec_sorted;
  uint32_t* perm_a;      // sorted position -> pair
  uint32_t* perm_b;
  uint8_t* head;
  int64_t* tile_heads;
  SortScratch sort;
};

GroupScratch carve_group(Arena& a, int64_t P) {
  GroupScratch g;
  const int64_t n = P > 0 ? P : 1;
  g.fmin = a.take<int>(8);
  g.fmax = a.take<int>(8);
  g.counts = a.take<int>(8);
  g.huge = a.take<uint2>(kHugeRuns);
  g.layout = a.take<KeyLayout>(1);
  g.top = a.take<uint64_t>(n);
  g.top_sorted = a.take<uint64_t>(n);
  g.rec = a.take<GroupRec>(n);
  g.rec_sorted = a.take<GroupRec>(n);
  g.perm_a = a.take<uint32_t>(n);
  g.perm_b = a.take<uint32_t>(n);
  g.head = a.take<uint8_t>(n);
  g.tile_heads = a.take<int64_t>(scan_tiles(n) + 1);
  g.sort = carve_sort_scratch(a, n);
  return g;
}

__global__ void k_init_minmax(int* fmin, int* fmax, int* counts) {
  if (threadIdx.x < 4) counts[threadIdx.x] = 0;
  if (threadIdx.x < 5) {
    fmin[threadIdx.x] = INT_MAX;
    fmax[threadIdx.x] = INT_MIN;
  }
}

int bit_length(uint64_t x) {
  int b = 0;
  while (x) {
    ++b;
    x >>= 1;
  }
  return b;
}

}  // namespace

}  // namespace ygx

extern "C" {

int ygx_level_major_geometry(const int32_t* nbl32, const void* level_offsets, int index_bits,
                             int num_levels, int64_t max_nodes, const float* center,
                             const float* half_extent, const float* radius,
                             const float* max_extent, float* o_center, float* o_half,
                             float* o_radius, float* o_max, void* o_nodes, cudaStream_t stream) {
  if (num_levels < 1 || max_nodes < 1 || (index_bits != 32 && index_bits != 64) || !nbl32 ||
      !level_offsets)
    return YGX_ERR_ARG;
  ygx::k_level_major<<<ygx::grid_for((int64_t)num_levels * max_nodes, 256), 256, 0, stream>>>(
      nbl32, level_offsets, index_bits, num_levels, max_nodes, center, half_extent, radius,
      max_extent, o_center, o_half, o_radius, o_max, o_nodes);
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

int ygx_dense_m2l(const void* node_idx, int index_bits, int64_t slots, int64_t max_interactions,
                  const void* counts, const void* offsets, const void* sources,
                  const float* center, int64_t total, void* o_src, bool* o_mask, void* o_counts,
                  float* o_disp, cudaStream_t stream) {
  if (slots < 1 || max_interactions < 1 || total < 1 || (index_bits != 32 && index_bits != 64))
    return YGX_ERR_ARG;
  ygx::k_dense_m2l<<<ygx::grid_for(slots * max_interactions, 256), 256, 0, stream>>>(
      node_idx, index_bits, slots, max_interactions, counts, offsets, sources, center, total,
      o_src, o_mask, o_counts, o_disp);
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

size_t ygx_grouped_workspace_size(int64_t num_pairs) {
  ygx::Arena a{nullptr, 0, 0};
  ygx::carve_group(a, num_pairs);
  return a.used + 256;
}

// Phase 1: fields of every pair and their ranges; *num_classes_out is set by
// ygx_grouped_classes.  Synchronizes (the key widths come from the ranges).
int ygx_grouped_classes(const void* sources, const void* targets, int index_bits,
                        int64_t num_pairs, const int32_t* level32, const float* center,
                        const double* root_extent, int64_t* num_classes_out, void* ws,
                        size_t ws_bytes, cudaStream_t stream) {
  if (num_pairs < 1 || num_pairs >= (int64_t)UINT32_MAX - 1 || !root_extent ||
      !num_classes_out || (index_bits != 32 && index_bits != 64))
    return YGX_ERR_ARG;
  if (ws_bytes < ygx_grouped_workspace_size(num_pairs)) return YGX_ERR_ARG;
  ygx::Arena a{(char*)ws, 0, ws_bytes};
  ygx::GroupScratch g = ygx::carve_group(a, num_pairs);
  const int64_t P = num_pairs;
  const ygx::GroupPairs pairs{sources, targets, index_bits,
                              P,       level32, center,
                              {root_extent[0], root_extent[1], root_extent[2]}};
  ygx::k_init_minmax<<<1, 32, 0, stream>>>(g.fmin, g.fmax, g.counts);
  YGX_CHECK_LAUNCH();
  ygx::k_group_ranges<<<ygx::grid_for(P, 256), 256, 0, stream>>>(pairs, g.fmin, g.fmax);
  YGX_CHECK_LAUNCH();
  struct {
    int lo[64], hi[64];  // fmin and fmax lie one arena step apart
  } range;
  static_assert(sizeof(range) == 512, "two arena steps");
  if ((char*)g.fmax - (char*)g.fmin != 256 ||
      cudaMemcpyAsync(&range, g.fmin, 256 + 5 * sizeof(int), cudaMemcpyDeviceToHost, stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess)
    return YGX_ERR_CUDA;
  // fields from most to least significant: target level, source level, dx, dy, dz
  ygx::KeyLayout kl;
  int bits = 0;
  for (int f = 4; f >= 0; --f) {
    kl.fmin[f] = range.lo[f];
    kl.width[f] = ygx::bit_length((uint64_t)((int64_t)range.hi[f] - (int64_t)range.lo[f]));
    kl.shift[f] = bits;
    bits += kl.width[f];
  }
  if (bits > 128) return YGX_ERR_TOO_LARGE;
  kl.cut = bits > 64 ? bits - 64 : 0;
  ygx::k_group_pack<<<ygx::grid_for(P, 256), 256, 0, stream>>>(pairs, kl, g.layout, g.top, g.rec);
  YGX_CHECK_LAUNCH();
  uint32_t* status = reinterpret_cast<uint32_t*>(g.fmin + 6);
  const int64_t tiles = ygx::scan_tiles(P);
  struct {
    int64_t classes;
    int huge;
  } h{0, 0};
  // sorted by `top` (one class: the identity order), ties resolved into perm_b;
  // then, if there are huge runs, again after those
  const bool ties_later = kl.cut > ygx::kLowFirst;
  for (int attempt = 0; attempt < 2; ++attempt) {
    int rc;
    if (attempt == 0 && kl.cut > 0 && !ties_later) {
      uint64_t* keys = reinterpret_cast<uint64_t*>(g.rec_sorted);  // free until the heads
      ygx::k_group_low_keys<<<ygx::grid_for(P, 256), 256, 0, stream>>>(g.rec, P, keys);
      YGX_CHECK_LAUNCH();
      rc = ygx::onesweep_sort(keys, nullptr, P, 0, kl.cut, g.top_sorted, g.perm_a, g.sort, false,
                              status, stream);
      if (rc) return rc;
      ygx::k_gather_u64<<<ygx::grid_for(P, 256), 256, 0, stream>>>(g.top, g.perm_a, P, keys);
      YGX_CHECK_LAUNCH();
      rc = ygx::onesweep_sort(keys, g.perm_a, P, 0, 64, g.top_sorted, g.perm_b, g.sort, false,
                              status, stream);
      if (rc) return rc;
    } else if (attempt == 0) {
      rc = ygx::onesweep_sort(g.top, nullptr, P, 0, bits == 0 ? 1 : (bits > 64 ? 64 : bits),
                              g.top_sorted, ties_later ? g.perm_a : g.perm_b, g.sort, false,
                              status, stream);
      if (rc) return rc;
      if (ties_later) {
        // the lists lie where the heads' records come, 16 bytes a pair: at most P
        // descents, P / kTieMax runs, twice P / kTieMax + 1 words (P > 1 here: one
        // pair's key has no bits)
        char* lists = reinterpret_cast<char*>(g.rec_sorted);
        uint32_t* claims = reinterpret_cast<uint32_t*>(lists + 12 * P);
        const int64_t blocks = P / ygx::kTieMax + 1;
        if (cudaMemsetAsync(claims, 0, 2 * sizeof(uint32_t) * blocks, stream) != cudaSuccess)
          return YGX_ERR_CUDA;
        const ygx::GroupTies ties{g.top_sorted, g.rec, P, g.perm_a, g.perm_b,
                                  reinterpret_cast<uint32_t*>(lists),
                                  reinterpret_cast<uint2*>(lists + 4 * (P + P % 2)),
                                  claims, claims + blocks, g.counts, g.huge,
                                  P / 64 > 16384 ? P / 64 : 16384};
        ygx::k_group_ties<<<ygx::grid_for(P, 256), 256, 0, stream>>>(ties);
        YGX_CHECK_LAUNCH();
        ygx::k_group_short<<<ygx::grid_for(P, 256), 256, 0, stream>>>(ties);
        YGX_CHECK_LAUNCH();
        if (P > ygx::kTieMax) {
          ygx::k_group_long<<<ygx::kNumSMs * 2, ygx::kLongThreads, 0, stream>>>(ties, kl.cut);
          YGX_CHECK_LAUNCH();
        }
      }
    } else {
      uint2 runs[ygx::kHugeRuns];
      if (h.huge > ygx::kHugeRuns ||
          cudaMemcpyAsync(runs, g.huge, sizeof(uint2) * h.huge, cudaMemcpyDeviceToHost, stream) !=
              cudaSuccess ||
          cudaStreamSynchronize(stream) != cudaSuccess)
        return YGX_ERR_CUDA;
      uint64_t* keys = reinterpret_cast<uint64_t*>(g.rec_sorted);  // free until the heads
      for (int k = 0; k < h.huge; ++k) {
        const int64_t n = runs[k].y;
        const uint32_t* in = g.perm_a + runs[k].x;
        ygx::k_group_run_keys<<<ygx::grid_for(n, 256), 256, 0, stream>>>(g.rec, in, n, keys);
        YGX_CHECK_LAUNCH();
        rc = ygx::onesweep_sort(keys, in, n, 0, kl.cut, keys + P, g.perm_b + runs[k].x, g.sort,
                                false, status, stream);
        if (rc) return rc;
      }
    }
    ygx::k_group_heads<<<(unsigned)tiles, ygx::kScanThreads, 0, stream>>>(
        g.top_sorted, g.perm_b, g.rec, P, g.rec_sorted, g.head, g.tile_heads,
        attempt == 0 ? g.counts : nullptr);
    YGX_CHECK_LAUNCH();
    // exclusive over the tiles and, as one more "tile", the total
    if (cudaMemsetAsync(g.tile_heads + tiles, 0, sizeof(int64_t), stream) != cudaSuccess)
      return YGX_ERR_CUDA;
    ygx::k_seg_mid<<<1, 1024, 0, stream>>>(g.tile_heads, tiles + 1);
    YGX_CHECK_LAUNCH();
    if (cudaMemcpyAsync(&h.classes, g.tile_heads + tiles, sizeof(int64_t), cudaMemcpyDeviceToHost,
                        stream) != cudaSuccess ||
        (ties_later && attempt == 0 &&
         cudaMemcpyAsync(&h.huge, g.counts, sizeof(int), cudaMemcpyDeviceToHost, stream) !=
             cudaSuccess) ||
        cudaStreamSynchronize(stream) != cudaSuccess)
      return YGX_ERR_CUDA;
    if (attempt > 0 || !h.huge) break;
  }
  *num_classes_out = h.classes;
  return YGX_OK;
}

// Phase 2 (same workspace, after ygx_grouped_classes): class keys (C x 5
// int32), class displacements (C x 3 float), class offsets (C + 1), sources /
// targets in class order and each pair's class in the input order.
int ygx_grouped_emit(const void* sources, const void* targets, int index_bits, int64_t num_pairs,
                     const double* root_extent, int32_t* class_keys, float* class_disp,
                     void* class_offsets, void* class_sources, void* class_targets,
                     void* class_ids, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if (num_pairs < 1 || !root_extent || (index_bits != 32 && index_bits != 64)) return YGX_ERR_ARG;
  if (ws_bytes < ygx_grouped_workspace_size(num_pairs)) return YGX_ERR_ARG;
  ygx::Arena a{(char*)ws, 0, ws_bytes};
  ygx::GroupScratch g = ygx::carve_group(a, num_pairs);
  ygx::k_group_emit<<<(unsigned)ygx::scan_tiles(num_pairs), ygx::kScanThreads, 0, stream>>>(
      g.top_sorted, g.perm_b, g.rec_sorted, g.head, g.tile_heads, num_pairs, index_bits,
      root_extent[0], root_extent[1], root_extent[2], g.layout, class_keys, class_disp,
      class_offsets, class_sources, class_targets, class_ids);
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

}  // extern "C"
