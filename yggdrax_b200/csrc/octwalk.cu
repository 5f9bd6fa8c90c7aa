// Native octree walk: the dual-tree walk in explicit octree cell space
// (_dual_tree_walk_octree_impl, yggdrax/_interactions_impl.py:1908-2597),
// behind build_octree_native_far_pairs (:5556-5634) and
// build_octree_native_neighbor_lists (:5637-5717); and the cell box geometry
// those walks use (compute_explicit_octree_box_geometry,
// yggdrax/octree.py:422-476).
//
// The walk is breadth first from (root, root).  Each generation is a stable
// compaction (as the reference's cumsum pushes): every pair is evaluated (MAC
// on the box centres and extents, accept / near / refine, split rule, number
// of children), prefix sums give every child and every accepted / near pair
// its slot, and the next wavefront and the pair log are written there.  All
// generations run in one cooperative launch (genwalk.cuh), which also follows
// the counters.  The log of a generation holds its accepted pairs twice: first
// every pair as (row of the first cell, second cell) in wavefront order,
// then every pair as (row of the second cell, first cell) -- the
// reference's fwd and bwd blocks (:2243-2394).  A stable sort of the whole
// log by row therefore yields every row in (generation, block, wavefront)
// order, the reference's row order up to the order inside one block, which
// the reference leaves to an unstable argsort (:813-873).
#include "genwalk.cuh"

namespace ygx {

namespace {

constexpr uint32_t kOctFarOver = 1u << 0;    // a far row exceeded its capacity
constexpr uint32_t kOctNearOver = 1u << 1;   // a near row exceeded its capacity
constexpr uint32_t kOctQueueOver = 1u << 2;  // more children than the queue holds
constexpr uint32_t kOctBadInput = 1u << 3;   // a cell id out of range
constexpr uint32_t kOctWfShort = 1u << 4;    // children exceed the wavefront buffer
constexpr uint32_t kOctLogShort = 1u << 5;   // the pair log was too short (walk continues)
constexpr int kOctMaxGens = 1 << 16;

struct OctCtl {
  long long far_n;     // far log entries so far (2 per accepted pair)
  long long near_n;    // near log entries so far (2 per near pair)
  unsigned long long accept;  // decisions
  unsigned long long nearc;
  unsigned long long refine;
  long long wf_need;   // largest number of children of a generation
  // raised while a generation is evaluated (read after its first barrier) and
  // while it is written (read after its second): a CTA that is ahead writes
  // the other word
  unsigned int flags_eval, flags_emit;
  unsigned int flags;    // at the end
  unsigned int gens;
  unsigned int arrived;  // grid barrier
  unsigned int timeout;
};

struct OctArgs {
  const int32_t* kids;         // [M][8] the octant slots below child_count that hold a
                               // cell, moved to the front
  const float4* rec;           // [M] centre, MAC extent
  const uint8_t* info;         // [M] cells in kids (4 bits) | leaf test << 4
  const int32_t* far_row;      // [M] row key of a cell in the far log, or null
  const int32_t* near_row;     // [M] row key of a cell in the near log (-1: none), or null
  int32_t* far_cnt;            // [M]
  int32_t* near_cnt;           // [near rows]
  int64_t M;
  float theta_sq;
  float theta;
  int mac;                     // 0 bh, 1 dehnen, 2 engblom
  int64_t far_cap;             // per-row capacities
  int64_t near_cap;
  int2* wf[2];                 // wavefronts (first cell, second cell)
  uint8_t* kind;               // per pair of the current wavefront
  int64_t wf_room, queue, log_cap;
  uint64_t *far_key, *near_key;
  uint32_t *far_val, *near_val;
  GenTotals* totals;
  OctCtl* ctl;
  uint32_t spin_limit;
};

// Node records of the walk.  Refined pairs push the first child_count octant
// slots of the split side, empty (-1) slots skipped
// (_octree_refine_pairs_single, :106-165): those are gathered once here.
__global__ void k_oct_prepare(const void* __restrict__ children, const void* __restrict__ counts,
                              int index_bits, int64_t M, const float* __restrict__ centers,
                              const float* __restrict__ radii,
                              const float* __restrict__ max_extents,
                              const uint8_t* __restrict__ leaf, int mac, float scale,
                              int32_t root, int32_t* __restrict__ kids, float4* __restrict__ rec,
                              uint8_t* __restrict__ info, int2* __restrict__ wf0,
                              OctCtl* __restrict__ ctl) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x) {
    // dehnen / engblom: box radius (dehnen scaled); bh: box max extent
    const float e = mac == 0 ? max_extents[k] : mac == 1 ? __fmul_rn(scale, radii[k]) : radii[k];
    rec[k] = make_float4(centers[3 * k], centers[3 * k + 1], centers[3 * k + 2], e);
    const int64_t cc = (int32_t)load_idx(counts, index_bits, k);
    int n = 0;
    for (int j = 0; j < 8 && j < cc; ++j) {
      const int32_t c = (int32_t)load_idx(children, index_bits, 8 * k + j);
      if (c >= 0) kids[8 * k + n++] = c;
    }
    info[k] = (uint8_t)(n | (leaf[k] != 0 ? 16 : 0));
    if (k == 0) {
      wf0[0] = make_int2(root, root);
      *ctl = OctCtl{0, 0, 0, 0, 0, 1, 0u, 0u, 0u, 0u, 0u, 0u};
    }
  }
}

// What becomes of a pair (kind): 1 the children of both sides of the diagonal
// (a <= b), 3 the target's children, 4 the source's -- the split rule never
// splits both sides of an off-diagonal pair -- or accepted / near, or 0.
constexpr uint8_t kOctFar = 8, kOctNear = 16;

__device__ __forceinline__ uint8_t oct_evaluate(const OctArgs& p, int2 w, int* children,
                                                bool* refine) {
  const int32_t t = w.x, s = w.y;
  const float4 T = p.rec[t], S = p.rec[s];
  const int ti = p.info[t], si = p.info[s];
  // delta = centers[t] - centers[s]; squares summed in written order
  const float dx = __fsub_rn(T.x, S.x), dy = __fsub_rn(T.y, S.y), dz = __fsub_rn(T.z, S.z);
  const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
  const float et = T.w, es = S.w;
  float lhs;
  if (p.mac == 2) lhs = __fadd_rn(fmaxf(et, es), __fmul_rn(p.theta, fminf(et, es)));
  else lhs = __fadd_rn(et, es);
  const bool ok = __fmul_rn(lhs, lhs) <= __fmul_rn(p.theta_sq, d2);
  const bool same = t == s, tl = ti >> 4, sl = si >> 4;
  *children = 0;
  *refine = false;
  if (!same && d2 > 0.0f && ok) return kOctFar;
  if (tl && sl && !same) return kOctNear;
  *refine = true;
  const int nt = ti & 15, ns = si & 15;
  const bool split_t = !tl && (same || sl || et >= es);
  const bool split_s = !sl && (same || tl || es > et);
  if (split_t && split_s) {  // the diagonal
    *children = nt * (nt + 1) / 2;
    return 1;
  }
  if (split_t) {
    *children = nt;
    return 3;
  }
  if (split_s) {
    *children = ns;
    return 4;
  }
  return 0;
}
__device__ __forceinline__ int oct_child_count(const OctArgs& p, uint8_t kind, int2 w) {
  const int n = p.info[kind == 4 ? w.y : w.x] & 15;
  return kind == 1 ? n * (n + 1) / 2 : kind == 3 || kind == 4 ? n : 0;
}

// Writes one accepted / near pair to both blocks of its log and counts both
// rows, at counter n.x and n.y.  A row past its capacity and a log that is too
// short are flagged.
__device__ __forceinline__ unsigned oct_log(uint64_t* key, uint32_t* val, int64_t log_cap,
                                            long long fwd, long long bwd, int32_t row_t,
                                            int32_t row_s, int2 w, int32_t* cnt, int2 n,
                                            int64_t cap, unsigned over) {
  unsigned f = 0;
  if (bwd < log_cap) {
    key[fwd] = (uint64_t)(uint32_t)row_t;
    val[fwd] = (uint32_t)w.y;
    key[bwd] = (uint64_t)(uint32_t)row_s;
    val[bwd] = (uint32_t)w.x;
  } else {
    f |= kOctLogShort;
  }
  if ((int64_t)atomicAdd(&cnt[n.x], 1) >= cap) f |= over;
  if ((int64_t)atomicAdd(&cnt[n.y], 1) >= cap) f |= over;
  return f;
}

// The whole walk.  The log grows by both blocks of a generation, the wavefront
// keeps its first `queue` children (flagged when there were more), and a
// generation with more children than the wavefront buffer holds ends the walk
// to ask for a larger one.  Every CTA follows the same counters.  The far and
// near walks of 1,048,576 clumped particles (12 generations each): 0.71 ms
// together, against 1.4 ms of kernels in nine launches per generation and the
// host's read-back between them (tree and both lists: 4.6 -> 3.2 ms).
__global__ void __launch_bounds__(kGenThreads, 2) k_oct_walk(const OctArgs a) {
  constexpr unsigned kStop =
      kOctFarOver | kOctNearOver | kOctQueueOver | kOctBadInput | kOctWfShort;
  long long size = 1, far_n = 0, near_n = 0, wf_need = 1;
  unsigned long long n_acc = 0, n_near = 0, n_ref = 0;
  unsigned flags = 0, gens = 0, target = 0;
  int cur = 0;
  bool ok = true;
  while (size > 0 && (flags & kStop) == 0 && gens < (unsigned)kOctMaxGens) {
    const int2* wf = a.wf[cur];
    int2* next = a.wf[cur ^ 1];
    const int64_t slice = gen_slice(size);
    const int64_t lo = blockIdx.x * slice, hi = lo + slice < size ? lo + slice : size;
    unsigned long long nc = 0, nf = 0, nn = 0;
    bool bad = false;
    for (int64_t i = lo + threadIdx.x; i < hi; i += kGenThreads) {
      const int2 w = __ldcg(wf + i);
      uint8_t kd = 0;
      if (w.x >= 0 && w.y >= 0 && w.x < a.M && w.y < a.M) {
        int c;
        bool refine;
        kd = oct_evaluate(a, w, &c, &refine);
        // all three decisions are counted, collected or not
        n_acc += kd == kOctFar;
        n_near += kd == kOctNear;
        n_ref += refine;
        if ((kd == kOctFar && !a.far_row) || (kd == kOctNear && !a.near_row)) kd = 0;
        nc += c;
        nf += kd == kOctFar;
        nn += kd == kOctNear;
      } else {
        bad = true;
      }
      a.kind[i] = kd;
    }
    if (bad) atomicOr(&a.ctl->flags_eval, kOctBadInput);
    gen_publish(nc, nf, nn, a.totals);
    if (!(ok = gen_barrier(&a.ctl->arrived, &target, a.spin_limit))) break;
    GenTotals pre, all;
    gen_prefix(a.totals, &pre, &all);
    flags |= __ldcg(&a.ctl->flags_eval);
    unsigned raise = 0;
    for (int64_t c0 = lo; c0 < hi; c0 += kGenThreads) {
      const int64_t i = c0 + threadIdx.x;
      const uint8_t kd = i < hi ? a.kind[i] : 0;
      const int2 w = kd ? __ldcg(wf + i) : make_int2(0, 0);
      // children (at most 36 x 512) | far << 32 | near << 48
      const unsigned long long v =
          (unsigned long long)(kd && kd < kOctFar ? oct_child_count(a, kd, w) : 0) |
          (kd == kOctFar ? 1ull << 32 : 0ull) | (kd == kOctNear ? 1ull << 48 : 0ull);
      unsigned long long sum;
      const unsigned long long at = gen_block_scan(v, &sum);
      if (kd == kOctFar) {
        // counted by cell: a cell's row key is the caller's and only sorted by
        const long long r = far_n + (long long)pre.x + (long long)((at >> 32) & 0xffffull);
        raise |= oct_log(a.far_key, a.far_val, a.log_cap, r, r + (long long)all.x,
                         a.far_row[w.x], a.far_row[w.y], w, a.far_cnt, w, a.far_cap, kOctFarOver);
      } else if (kd == kOctNear) {
        const long long r = near_n + (long long)pre.y + (long long)(at >> 48);
        const int32_t rt = a.near_row[w.x], rs = a.near_row[w.y];
        if (rt < 0 || rs < 0) raise |= kOctBadInput;
        else
          raise |= oct_log(a.near_key, a.near_val, a.log_cap, r, r + (long long)all.y, rt, rs, w,
                           a.near_cnt, make_int2(rt, rs), a.near_cap, kOctNearOver);
      } else if (kd) {
        int64_t slot = (int64_t)pre.child + (int64_t)(at & 0xffffffffull);
        auto put = [&](int x, int y) {
          if (slot < a.wf_room) next[slot] = x < y ? make_int2(x, y) : make_int2(y, x);
          ++slot;
        };
        const int32_t split = kd == 4 ? w.y : w.x, other = kd == 4 ? w.x : w.y;
        const int32_t* c = a.kids + (int64_t)split * 8;
        const int n = a.info[split] & 15;
        for (int i0 = 0; i0 < n; ++i0) {
          if (kd == 1)
            for (int i1 = i0; i1 < n; ++i1) put(c[i0], c[i1]);
          else
            put(c[i0], other);
        }
      }
      pre.child += sum & 0xffffffffull;
      pre.x += (sum >> 32) & 0xffffull;
      pre.y += sum >> 48;
    }
    if (raise) atomicOr(&a.ctl->flags_emit, raise);
    const long long children = (long long)all.child;
    const long long kept = children < a.queue ? children : a.queue;
    if (children > a.queue) flags |= kOctQueueOver;
    if (kept > a.wf_room) flags |= kOctWfShort;
    if (kept > wf_need) wf_need = kept;
    far_n += 2 * (long long)all.x;
    near_n += 2 * (long long)all.y;
    size = kept;
    cur ^= 1;
    ++gens;
    if (!(ok = gen_barrier(&a.ctl->arrived, &target, a.spin_limit))) break;
    flags |= __ldcg(&a.ctl->flags_emit);
  }
  for (int o = 16; o > 0; o >>= 1) {
    n_acc += __shfl_xor_sync(0xffffffffu, n_acc, o);
    n_near += __shfl_xor_sync(0xffffffffu, n_near, o);
    n_ref += __shfl_xor_sync(0xffffffffu, n_ref, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (n_acc) atomicAdd(&a.ctl->accept, n_acc);
    if (n_near) atomicAdd(&a.ctl->nearc, n_near);
    if (n_ref) atomicAdd(&a.ctl->refine, n_ref);
  }
  if (threadIdx.x == 0) {
    if (!ok) a.ctl->timeout = 1u;
    if (blockIdx.x == 0) {
      a.ctl->far_n = far_n;
      a.ctl->near_n = near_n;
      a.ctl->wf_need = wf_need;
      a.ctl->gens = size > 0 && (flags & kStop) == 0 ? (unsigned)kOctMaxGens + 1u : gens;
      a.ctl->flags = flags;
    }
  }
}

// Every third bit of a 64-bit word (the inverse of the Morton spread), by
// the standard mask-and-shift compaction.
__device__ __forceinline__ uint64_t compact3(uint64_t x) {
  x &= 0x1249249249249249ull;
  x = (x ^ (x >> 2)) & 0x10C30C30C30C30C3ull;
  x = (x ^ (x >> 4)) & 0x100F00F00F00F00Full;
  x = (x ^ (x >> 8)) & 0x001F0000FF0000FFull;
  x = (x ^ (x >> 16)) & 0x001F00000000FFFFull;
  x = (x ^ (x >> 32)) & 0x00000000001FFFFFull;
  return x;
}

// Box of a cell from its code and depth (compute_explicit_octree_box_geometry,
// octree.py:422-476), fp32 with every operation rounded: cell = domain /
// 2^depth, mins = bmin + cell * index, maxs = mins + cell, centre 0.5 (mins +
// maxs), half 0.5 (maxs - mins), radius sqrt((h0^2 + h1^2) + h2^2), max extent
// max(h); zeros on invalid cells.
struct OctBoxOut {
  float *centers, *half, *radii, *max_extents;
};
__device__ __forceinline__ void oct_box(int64_t k, bool valid, uint64_t code, int64_t d,
                                        const float b0[3], const float dom[3],
                                        const OctBoxOut& o) {
  float c[3] = {0.f, 0.f, 0.f}, h[3] = {0.f, 0.f, 0.f}, r = 0.f, mx = 0.f;
  if (valid) {
    d = d < 0 ? 0 : (d > 21 ? 21 : d);
    const uint64_t sh = (uint64_t)(21 - d);
    const uint64_t q[3] = {compact3(code) >> sh, compact3(code >> 1) >> sh,
                           compact3(code >> 2) >> sh};
    const float cnt = (float)(1ull << d);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float cell = __fdiv_rn(dom[a], cnt);
      const float lo = __fadd_rn(b0[a], __fmul_rn(cell, (float)q[a]));
      const float hi = __fadd_rn(lo, cell);
      c[a] = __fmul_rn(0.5f, __fadd_rn(lo, hi));
      h[a] = __fmul_rn(0.5f, __fsub_rn(hi, lo));
    }
    const float s = __fadd_rn(__fadd_rn(__fmul_rn(h[0], h[0]), __fmul_rn(h[1], h[1])),
                              __fmul_rn(h[2], h[2]));
    r = __fsqrt_rn(s);
    mx = fmaxf(fmaxf(h[0], h[1]), h[2]);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o.centers[3 * k + a] = c[a];
    o.half[3 * k + a] = h[a];
  }
  o.radii[k] = r;
  o.max_extents[k] = mx;
}

__global__ void k_oct_box(const uint8_t* __restrict__ valid, const uint64_t* __restrict__ codes,
                          const void* __restrict__ depths, int index_bits, int64_t M,
                          float bx0, float by0, float bz0, float dx, float dy, float dz,
                          const OctBoxOut o) {
  const float b0[3] = {bx0, by0, bz0}, dom[3] = {dx, dy, dz};
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x)
    oct_box(k, valid[k] != 0, codes[k], load_idx(depths, index_bits, k), b0, dom, o);
}

// The traversal view of an octree (octree.py:577-704): per cell the smallest
// radix node and radix leaf mapped to it (-1: none, or the cell is not valid /
// not a leaf), the box, and the numbers of valid and leaf cells.  As tensor
// operations (two scatters with their index ranges, masks and sums, the bounds
// read back to the host for the boxes) a view took a quarter of a millisecond;
// with two launches the octree-native step of 1,048,576 particles (two views)
// takes 2.61 ms instead of 3.09.
__global__ void k_oct_view_min(const void* __restrict__ node_to_oct, int64_t nodes,
                               const void* __restrict__ leaf_to_oct, int64_t leaves,
                               int64_t first_leaf, int index_bits, int64_t M,
                               uint32_t* __restrict__ min_node, uint32_t* __restrict__ min_leaf) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nodes + leaves;
       k += (int64_t)gridDim.x * blockDim.x) {
    const bool node = k < nodes;
    const int64_t c = node ? load_idx(node_to_oct, index_bits, k)
                           : load_idx(leaf_to_oct, index_bits, k - nodes);
    if (c < 0 || c >= M) continue;
    if (node) atomicMin(min_node + c, (uint32_t)k);
    else atomicMin(min_leaf + c, (uint32_t)(first_leaf + k - nodes));
  }
}
__global__ void k_oct_view(const uint8_t* __restrict__ valid, const uint8_t* __restrict__ leaf,
                           const uint64_t* __restrict__ codes, const void* __restrict__ depths,
                           int index_bits, int64_t M, const float* __restrict__ bmin,
                           const float* __restrict__ bmax, const uint32_t* __restrict__ min_node,
                           const uint32_t* __restrict__ min_leaf, void* node_of, void* leaf_of,
                           unsigned long long* __restrict__ counts, const OctBoxOut o) {
  float b0[3], dom[3];
  for (int a = 0; a < 3; ++a) {
    b0[a] = bmin[a];
    dom[a] = __fsub_rn(bmax[a], bmin[a]);
  }
  unsigned long long nv = 0, nl = 0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M;
       k += (int64_t)gridDim.x * blockDim.x) {
    const bool v = valid[k] != 0, l = leaf[k] != 0;
    const uint32_t n = min_node[k], f = min_leaf[k];
    store_idx(node_of, index_bits, k, v && n != 0xffffffffu ? (int64_t)n : -1);
    store_idx(leaf_of, index_bits, k, l && f != 0xffffffffu ? (int64_t)f : -1);
    oct_box(k, v, codes[k], load_idx(depths, index_bits, k), b0, dom, o);
    nv += v;
    nl += l;
  }
  for (int s = 16; s > 0; s >>= 1) {
    nv += __shfl_xor_sync(0xffffffffu, nv, s);
    nl += __shfl_xor_sync(0xffffffffu, nl, s);
  }
  if ((threadIdx.x & 31) == 0) {
    if (nv) atomicAdd(counts, nv);
    if (nl) atomicAdd(counts + 1, nl);
  }
}

struct OctScratch {
  OctCtl* ctl;
  int32_t* kids;
  float4* rec;
  uint8_t* info;
  int2* wf[2];
  uint8_t* kind;
  GenTotals* totals;
};

OctScratch carve_oct(Arena& a, int64_t M, int64_t wf) {
  OctScratch s;
  s.ctl = a.take<OctCtl>(1);
  s.kids = a.take<int32_t>(8 * M);
  s.rec = a.take<float4>(M);
  s.info = a.take<uint8_t>(M);
  for (int k = 0; k < 2; ++k) s.wf[k] = a.take<int2>(wf);
  s.kind = a.take<uint8_t>(wf);
  s.totals = a.take<GenTotals>(kGenMaxBlocks);
  return s;
}

}  // namespace

}  // namespace ygx

extern "C" {

int ygx_octree_box_geometry(const uint8_t* valid, const uint64_t* codes, const void* depths,
                            int index_bits, int64_t M, const float* bounds_min,
                            const float* bounds_max, float* centers, float* half_extents,
                            float* radii, float* max_extents, cudaStream_t stream) {
  if (M < 0 || (index_bits != 32 && index_bits != 64) || !bounds_min || !bounds_max)
    return YGX_ERR_ARG;
  if (M == 0) return YGX_OK;
  if (!valid || !codes || !depths || !centers || !half_extents || !radii || !max_extents)
    return YGX_ERR_ARG;
  // domain = bounds_max - bounds_min in fp32 (host values)
  const float d0 = bounds_max[0] - bounds_min[0], d1 = bounds_max[1] - bounds_min[1],
              d2 = bounds_max[2] - bounds_min[2];
  ygx::k_oct_box<<<ygx::grid_for(M, 256), 256, 0, stream>>>(
      valid, codes, depths, index_bits, M, bounds_min[0], bounds_min[1], bounds_min[2], d0, d1,
      d2, ygx::OctBoxOut{centers, half_extents, radii, max_extents});
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

size_t ygx_octree_view_workspace_size(int64_t M) {
  return 2 * ygx::align_up(sizeof(uint32_t) * (size_t)(M > 0 ? M : 1)) + 256;
}

int ygx_octree_view(const uint8_t* valid, const uint8_t* leaf, const uint64_t* codes,
                    const void* depths, const void* node_to_oct, int64_t nodes,
                    const void* leaf_to_oct, int64_t leaves, int64_t num_internal, int index_bits,
                    int64_t M, const float* bounds_min, const float* bounds_max, void* node_of,
                    void* leaf_of, uint64_t* counts, float* centers, float* half_extents,
                    float* radii, float* max_extents, void* ws, size_t ws_bytes,
                    cudaStream_t stream) {
  if (M < 1 || M > INT32_MAX || nodes < 0 || nodes > INT32_MAX || leaves < 0 ||
      num_internal < 0 || num_internal + leaves > INT32_MAX ||
      (index_bits != 32 && index_bits != 64) || !valid || !leaf || !codes || !depths ||
      (nodes > 0 && !node_to_oct) || (leaves > 0 && !leaf_to_oct) || !bounds_min ||
      !bounds_max || !node_of || !leaf_of || !counts || !centers || !half_extents || !radii ||
      !max_extents || !ws || ws_bytes < ygx_octree_view_workspace_size(M))
    return YGX_ERR_ARG;
  ygx::Arena a{(char*)ws, 0, ws_bytes};
  uint32_t* min_node = a.take<uint32_t>(M);
  uint32_t* min_leaf = a.take<uint32_t>(M);
  if (cudaMemsetAsync(min_node, 0xff, (size_t)((char*)(min_leaf + M) - (char*)min_node), stream) !=
          cudaSuccess ||
      cudaMemsetAsync(counts, 0, 2 * sizeof(uint64_t), stream) != cudaSuccess)
    return YGX_ERR_CUDA;
  ygx::k_oct_view_min<<<ygx::grid_for(nodes + leaves, 256), 256, 0, stream>>>(
      node_to_oct, nodes, leaf_to_oct, leaves, num_internal, index_bits, M, min_node, min_leaf);
  YGX_CHECK_LAUNCH();
  ygx::k_oct_view<<<ygx::grid_for(M, 256), 256, 0, stream>>>(
      valid, leaf, codes, depths, index_bits, M, bounds_min, bounds_max, min_node, min_leaf,
      node_of, leaf_of, reinterpret_cast<unsigned long long*>(counts),
      ygx::OctBoxOut{centers, half_extents, radii, max_extents});
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

size_t ygx_octree_walk_workspace_size(int64_t M, int64_t wf_capacity) {
  ygx::Arena a{nullptr, 0, 0};
  ygx::carve_oct(a, M > 0 ? M : 1, wf_capacity > 0 ? wf_capacity : 1);
  return a.used + 256;
}

int ygx_octree_walk(const void* children, const void* child_counts, int index_bits, int64_t M,
                    const float* centers, const float* radii, const float* max_extents,
                    const uint8_t* leaf_mask, const int32_t* far_row, const int32_t* near_row,
                    int64_t near_rows, int64_t root, int mac, float theta,
                    float dehnen_radius_scale, int64_t max_pair_queue, int64_t wf_capacity,
                    int64_t far_row_cap, int64_t near_row_cap, int64_t log_capacity,
                    uint64_t* far_key, uint32_t* far_val, uint64_t* near_key,
                    uint32_t* near_val, int32_t* far_cnt, int32_t* near_cnt,
                    int64_t* stats_out, uint32_t* flags_out, void* ws, size_t ws_bytes,
                    cudaStream_t stream) {
  if (M < 1 || M > INT32_MAX || root < 0 || root >= M || mac < 0 || mac > 2 ||
      max_pair_queue < 1 || wf_capacity < 1 || log_capacity < 1 ||
      (index_bits != 32 && index_bits != 64) || !children || !child_counts || !centers ||
      !radii || !max_extents || !leaf_mask || !stats_out || !flags_out || !ws ||
      (!far_row && !near_row) || (far_row && (!far_key || !far_val || !far_cnt)) ||
      (near_row && (near_rows < 1 || !near_key || !near_val || !near_cnt)))
    return YGX_ERR_ARG;
  if (ws_bytes < ygx_octree_walk_workspace_size(M, wf_capacity)) return YGX_ERR_ARG;
  ygx::Arena a{(char*)ws, 0, ws_bytes};
  ygx::OctScratch s = ygx::carve_oct(a, M, wf_capacity);
  ygx::k_oct_prepare<<<ygx::grid_for(M, 256), 256, 0, stream>>>(
      children, child_counts, index_bits, M, centers, radii, max_extents, leaf_mask, mac,
      dehnen_radius_scale, (int32_t)root, s.kids, s.rec, s.info, s.wf[0], s.ctl);
  YGX_CHECK_LAUNCH();
  if ((far_cnt && cudaMemsetAsync(far_cnt, 0, sizeof(int32_t) * M, stream) != cudaSuccess) ||
      (near_cnt && cudaMemsetAsync(near_cnt, 0, sizeof(int32_t) * near_rows, stream) !=
                       cudaSuccess))
    return YGX_ERR_CUDA;
  ygx::OctArgs p;
  p.kids = s.kids;
  p.rec = s.rec;
  p.info = s.info;
  p.far_row = far_row;
  p.near_row = near_row;
  p.far_cnt = far_cnt;
  p.near_cnt = near_cnt;
  p.M = M;
  // theta^2 in fp32 (jnp.asarray(theta, centers.dtype) ** 2); engblom's theta
  // is sqrt(theta^2)
  const float th = theta;
  p.theta_sq = th * th;
  p.theta = sqrtf(p.theta_sq);
  p.mac = mac;
  p.far_cap = far_row_cap;
  p.near_cap = near_row_cap;
  p.wf[0] = s.wf[0];
  p.wf[1] = s.wf[1];
  p.kind = s.kind;
  p.wf_room = wf_capacity;
  p.queue = max_pair_queue < 4 ? 4 : max_pair_queue;
  p.log_cap = log_capacity;
  p.far_key = far_key;
  p.far_val = far_val;
  p.near_key = near_key;
  p.near_val = near_val;
  p.totals = s.totals;
  p.ctl = s.ctl;
  p.spin_limit = (uint32_t)ygx::g_tune.spin_limit;
  const int grid = ygx::gen_grid(ygx::k_oct_walk);
  void* params[] = {&p};
  if (grid < 1 || cudaLaunchCooperativeKernel((const void*)ygx::k_oct_walk, dim3((unsigned)grid),
                                              dim3(ygx::kGenThreads), params, 0,
                                              stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return YGX_ERR_CUDA;
  }
  YGX_CHECK_LAUNCH();
  ygx::OctCtl h;
  if (cudaMemcpyAsync(&h, s.ctl, sizeof(h), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess)
    return YGX_ERR_CUDA;
  if (h.timeout) return YGX_ERR_TIMEOUT;
  int rc = YGX_OK;
  if (h.gens > (unsigned)ygx::kOctMaxGens) {
    rc = YGX_ERR_QUEUE_OVERFLOW;
    h.gens = (unsigned)ygx::kOctMaxGens;
  }
  stats_out[0] = h.far_n;
  stats_out[1] = h.near_n;
  stats_out[2] = (int64_t)h.accept;
  stats_out[3] = (int64_t)h.nearc;
  stats_out[4] = (int64_t)h.refine;
  stats_out[5] = (int64_t)h.gens;
  stats_out[6] = h.wf_need;
  flags_out[0] = h.flags;
  if (h.flags & ygx::kOctBadInput) return YGX_ERR_ARG;
  return rc;
}

}  // extern "C"
