// The unordered per-target walk over sibling pairs (schedules "target" and
// "learned" of trees below 2^24 nodes).  Included by target_walk.cu, whose
// header says why the pairs of one target follow from its parent's "split on
// my side" list alone; this file is the same walk with cheaper steps.
//
// What bounds it: the steps' own instructions and the latency of the record
// gathers (a step evaluates 32 candidates of one target; nothing is read
// twice from DRAM).  So the layout serves the step:
//  * Nodes are addressed by slot 2 * parent + side.  A refined candidate
//    pushes ONE 4-byte stack word for both children, the next window reads 16
//    words for 32 lanes, and the records of two siblings are one 32-byte
//    sector.
//  * A candidate is slot | generation << 24 (a slot below 2^24, a generation
//    below 256: twice the deepest level), half of the ordered walk's entry.
//  * A leaf target can never split on its own side and an internal target
//    never has a near pair, so the step has three outcomes (far, "kept":
//    near or split list, refine) in two specialisations and two ballots.
//  * A target that one warp runs from start to end (most of them) counts its
//    rows and appends its split list with no atomics; only a target that is
//    handed off uses the shared counters.
//  * A finished target's warp goes on with its left child and queues the
//    right one, so half of the dependent hops need no queue round trip.
// Measured, kernel time, against the walk over single 64-bit candidates with
// its level-order claims (k_tw_walk<mac, false>, kept for trees past 2^24
// nodes), and the steps it takes:
//   16,777,216 Plummer, leaf 32, dehnen 0.6   13.3 -> 7.2 ms   36.0 -> 19.6 M
//    4,194,304 Plummer, leaf 32, bh 0.5        3.05 -> 1.47 ms   5.8 -> 3.3 M
//    4,194,304 clumps, fixed depth             2.51 -> 1.31 ms   5.1 -> 2.9 M
//    1,000,003 Plummer, leaf 32                1.50 -> 0.78 ms   2.0 -> 1.1 M
//       65,536 cube, leaf 16                   0.37 -> 0.19 ms
//        4,000 cube, leaf 8, bh 0.5            0.18 -> 0.08 ms
// A forest of 512 sets of 256 to 65,536 particles (leaf 16, dehnen 0.6)
// walks in 2.64 ms and its rows are copied in 0.49, where the generation walk took 2.93 and its log's scatter
// 1.70.
// The large trees are bound by instruction issue, the small ones by the chain
// of dependent gathers down the tree's levels.  Pairs evaluated 32 wide with
// the next window prefetched took 8.3 ms at 16M; 5 CTAs per SM spill (8.0).
#pragma once

namespace ygx {
namespace {

constexpr int kPwWarps = 8;
constexpr int kPwThreads = kPwWarps * 32;
constexpr int kPwBlocksPerSM = 4;
constexpr int kPwStk = 320;        // stack words (sibling pairs) per warp
constexpr int kPwStg = 192;        // staged entries per stream; flushed above kPwStg - 64
constexpr int kPwSpillGroup = 8;   // sibling pairs per continuation piece
constexpr int kPwInhGroup = 64;    // inherited candidates per continuation piece
constexpr uint32_t kPwSlotMask = 0xffffffu;
constexpr uint32_t kPwGen = 0x1000000u;
constexpr int64_t kPwMaxNodes = 1 << 24;  // slots are 24 bits
// A forest's nodes are not internal nodes first, so a slot's id says itself
// whether it is a leaf: its sign bit, which the lists' copies drop.
constexpr uint32_t kPwLeaf = 0x80000000u;
constexpr uint32_t kPwId = 0x7fffffffu;

enum PwFlag : uint32_t { kPwSibling = 1u, kPwShared = 2u };

// A queue entry: a target whose parent is done, or a part of a target.
struct __align__(16) PwPiece {
  uint32_t et;       // the target's slot | depth << 24
  uint32_t flags;    // kPwSibling: the sibling is a candidate; kPwShared: a part
  uint32_t n_spill;  // sibling pairs at spill_off
  uint32_t n_inh;    // split-list entries at inh_off
  unsigned long long spill_off, inh_off;
};

// One output row (device table, far rows by node, near rows by leaf id).
struct __align__(16) PwRow {
  long long pad;  // its slot in the raw array (predicted rows)
  int32_t rcap;   // the slot's capacity (0: no prediction, all to the pool)
  int32_t row;    // node id / leaf position
};

struct PwWarpSmem {
  TwBlkSet al;
  TwWarpStats st;
  long long t_mark;
  unsigned long long s_off;  // this target's split list (run by one warp)
  int32_t s_len;
  int32_t cnt[2];  // far / near entries so far (targets run by one warp)
  PwRow row[2];    // the current target's far / near row
  uint32_t stk[kPwStk];
  uint32_t stg_a[kPwStg];  // far
  uint32_t stg_b[kPwStg];  // near (leaf targets) or split list
};
struct PwSmem {
  PwWarpSmem w[kPwWarps];
  unsigned int hist[kTwHist];
  unsigned long long sums[8];
};

struct PwArgs {
  const float4* sc;        // per slot: centre x, y, z and MAC extent
  const int32_t* sid;      // per slot: node id, kPwLeaf set on leaves
  const PwRow* rows;       // far rows per node
  const PwRow* near_rows;  // near rows per node (leaves only)
  int32_t n_targets;
  float theta_sq, theta;
  // per node, zeroed; used only by targets that were handed off
  int32_t* s_cnt;
  int32_t* s_nch;
  int32_t* s_head;
  int32_t* pieces_left;
  int32_t* far_cnt;   // per node
  int32_t* near_cnt;  // per leaf position
  int32_t* far_pool;
  int32_t* near_pool;
  uint32_t* s_pool;
  uint32_t* spill;
  unsigned long long far_cap, near_cap, s_cap, spill_cap;
  unsigned long long* far_keys;
  TwChunk* far_recs;
  unsigned long long* near_keys;
  TwChunk* near_recs;
  TwSChunk* s_recs;
  unsigned int far_rec_cap, near_rec_cap, s_rec_cap, q_cap;
  PwPiece* queue;
  unsigned int* q_ready;
  unsigned int* gen_hist;
  TwCtl* ctl;
  uint32_t* status;
  uint32_t spin_limit;
  int budget;
  int hungry;  // waiting warps above which a long piece is split early
  unsigned long long blk_entries;
  unsigned int blk_records;
  int32_t* far_raw;
  int32_t* near_raw;
  unsigned* first_ovf_far;
  unsigned* first_ovf_near;
};

__device__ __forceinline__ uint32_t pw_load_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t pw_load_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void pw_store_release(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void pw_copy16(void* smem, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(smem)),
               "l"(global)
               : "memory");
}
__device__ __forceinline__ void pw_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Slot records of both children of every internal node, the rows' places,
// and the two pieces
// that start the walk (the root's children: nothing inherited, each the
// other's sibling).
__global__ void k_pw_slots(const float* __restrict__ center, const float* __restrict__ radius,
                           const float* __restrict__ max_extent,
                           const int32_t* __restrict__ left32, const int32_t* __restrict__ right32,
                           int32_t ni, int32_t total, int32_t root, int mac, float dehnen_scale,
                           float4* __restrict__ sc, int32_t* __restrict__ sid,
                           PwPiece* __restrict__ queue, unsigned int* __restrict__ q_ready,
                           TwCtl* __restrict__ ctl, const int32_t* __restrict__ leafpos,
                           const int32_t* __restrict__ far_rcap,
                           const int32_t* __restrict__ near_rcap,
                           const int64_t* __restrict__ pad_far,
                           const int64_t* __restrict__ pad_near, PwRow* __restrict__ rows,
                           unsigned* __restrict__ first_ovf_far,
                           unsigned* __restrict__ first_ovf_near,
                           uint32_t* __restrict__ status) {
  for (int32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < total;
       s += gridDim.x * blockDim.x) {
    PwRow f{0, 0, s};
    if (far_rcap) {
      f.pad = pad_far[s];
      f.rcap = far_rcap[s];
      first_ovf_far[s] = 0xffffffffu;
    }
    rows[s] = f;
    if (s >= ni) {
      const int32_t lp = leafpos[s];
      PwRow q{0, 0, lp};
      if (far_rcap) {
        q.pad = pad_near[lp];
        q.rcap = near_rcap[lp];
        first_ovf_near[lp] = 0xffffffffu;
      }
      rows[total + s - ni] = q;
    }
    if (s >= 2 * ni) continue;
    const int32_t c = (s & 1) ? right32[s >> 1] : left32[s >> 1];
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((unsigned)c < (unsigned)total) {
      // _build_mac_extents (_interactions_impl.py:993-1061)
      float e = mac == kTwBH ? max_extent[c] : radius[c];
      if (mac == kTwDehnen) e = __fmul_rn(dehnen_scale, e);
      r = make_float4(center[3 * c], center[3 * c + 1], center[3 * c + 2], e);
    }
    // an id outside the tree has extent 0 here: reported, and it is never
    // dereferenced as a node (a leaf id ends the walk there)
    if (!(r.w > 0.0f)) raise_flag(status, kFlagBadInput);
    sc[s] = r;
    const int32_t id = (unsigned)c < (unsigned)total ? c : total - 1;
    sid[s] = id >= ni ? (int32_t)((uint32_t)id | kPwLeaf) : id;
    if (s < 2) {
      if (s == 0) {
        float e = mac == kTwBH ? max_extent[root] : radius[root];
        if (mac == kTwDehnen) e = __fmul_rn(dehnen_scale, e);
        if (!(e > 0.0f)) raise_flag(status, kFlagBadInput);
        ctl->q_tail = 2u;
      }
      PwPiece p;
      p.et = (uint32_t)(2 * root + s) | kPwGen;
      p.flags = kPwSibling;
      p.n_spill = p.n_inh = 0;
      p.spill_off = p.inh_off = 0;
      queue[s] = p;
      q_ready[s] = 1u;
    }
  }
}

// The same for a forest (batched sets; set q's nodes from 2 leaf_off[q] - q on,
// its root first), a thread per node, bound by its gathers of two children
// (12 us for 512 sets of 256 to 65,536 particles): slots of every internal node by
// global id, rows without predicted slots, the two pieces of every set with a
// pair, and the nodes per level of all sets.  A set with tied codes is
// flagged: the host then runs the generation walk.
__global__ void k_pw_forest_slots(const float* __restrict__ center,
                                  const float* __restrict__ radius,
                                  const float* __restrict__ max_extent,
                                  const int32_t* __restrict__ left32,
                                  const int32_t* __restrict__ right32,
                                  const int32_t* __restrict__ leafpos,
                                  const int32_t* __restrict__ level32, int32_t total,
                                  const int64_t* __restrict__ leaf_off, int64_t S,
                                  const uint32_t* __restrict__ seg_flags, int mac,
                                  float dehnen_scale, float4* __restrict__ sc,
                                  int32_t* __restrict__ sid, PwPiece* __restrict__ queue,
                                  unsigned int* __restrict__ q_ready, unsigned int q_cap,
                                  TwCtl* __restrict__ ctl, PwRow* __restrict__ rows,
                                  PwRow* __restrict__ near_rows, int64_t* __restrict__ levels,
                                  uint32_t* __restrict__ status) {
  __shared__ unsigned s_levels[kTwHist / 2];
  for (int k = threadIdx.x; k < kTwHist / 2; k += blockDim.x) s_levels[k] = 0;
  __syncthreads();
  auto extent = [&](int32_t v) {  // _build_mac_extents (_interactions_impl.py:993-1061)
    const float e = mac == kTwBH ? max_extent[v] : radius[v];
    return mac == kTwDehnen ? __fmul_rn(dehnen_scale, e) : e;
  };
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < total; k += gridDim.x * blockDim.x) {
    rows[k] = PwRow{0, 0, k};
    if (!(extent(k) > 0.0f)) raise_flag(status, kFlagBadInput);
    const int lv = level32[k];
    atomicAdd(&s_levels[lv < 0 ? 0 : lv < kTwHist / 2 ? lv : kTwHist / 2 - 1], 1u);
    const int32_t ch[2] = {left32[k], right32[k]};
    if (ch[0] < 0) {
      near_rows[k] = PwRow{0, 0, leafpos[k]};
      continue;
    }
    for (int side = 0; side < 2; ++side) {
      const int32_t c = ch[side];
      const bool in = (unsigned)c < (unsigned)total;
      if (!in) raise_flag(status, kFlagBadInput);  // ends there, as a leaf (see k_pw_slots)
      sc[2 * k + side] = in ? make_float4(center[3 * c], center[3 * c + 1], center[3 * c + 2],
                                          extent(c))
                            : make_float4(0.f, 0.f, 0.f, 0.f);
      sid[2 * k + side] = !in || left32[c] < 0 ? (int32_t)((uint32_t)(in ? c : k) | kPwLeaf) : c;
    }
  }
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < S;
       q += (int64_t)gridDim.x * blockDim.x) {
    if (leaf_off[q + 1] - leaf_off[q] < 2) continue;
    // no tree to walk, or one whose build gave up: nothing of it is queued
    if (const uint32_t f = seg_flags[q] & (kFlagMalformed | kFlagTimeout)) {
      raise_flag(status, f);
      ctl->stop = 1u;
      ctl->q_head = q_cap;  // no warp takes a piece of any set
      continue;
    }
    const uint32_t root = (uint32_t)(2 * leaf_off[q] - q);
    const unsigned at = atomicAdd(&ctl->q_tail, 2u);
    if (at + 2u > q_cap) {
      raise_flag(status, kFlagLogOverflow);
      ctl->stop = 1u;
      continue;
    }
    for (uint32_t side = 0; side < 2; ++side) {
      queue[at + side] = PwPiece{(2u * root + side) | kPwGen, kPwSibling, 0u, 0u, 0ull, 0ull};
      q_ready[at + side] = 1u;
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kTwHist / 2; k += blockDim.x)
    if (s_levels[k])
      atomicAdd(reinterpret_cast<unsigned long long*>(levels) + k, (unsigned long long)s_levels[k]);
}

// Warp-collective: n staged ids of one row to the row's predicted slot where
// they fit, else to a pool chunk recorded as (row, offset in the row).  The
// offset is the warp's own count, or for a shared target the row counter's.
__device__ __noinline__ void pw_flush_row(const PwArgs& a, PwWarpSmem& W, int near, int shared,
                                          int n, int lane) {
  if (n == 0) return;
  pw_copy_wait();
  __syncwarp();
  const PwRow& R = W.row[near];
  const uint32_t* stg = near ? W.stg_b : W.stg_a;
  int32_t* cnt_row = (near ? a.near_cnt : a.far_cnt) + R.row;
  int within = 0;
  if (lane == 0) {
    if (shared) {
      within = atomicAdd(cnt_row, n);
    } else {
      within = W.cnt[near];
      W.cnt[near] = within + n;
    }
  }
  within = __shfl_sync(0xffffffffu, within, 0);
  if ((long long)within + n <= (long long)R.rcap) {
    int32_t* raw = (near ? a.near_raw : a.far_raw) + R.pad + within;
    for (int k = lane; k < n; k += 32) raw[k] = (int32_t)(stg[k] & kPwId);
    return;
  }
  unsigned long long off = 0, ri = 0;
  TwBlk* pb = near ? &W.al.near_ : &W.al.far;
  TwBlk* rb = near ? &W.al.near_r : &W.al.far_r;
  const bool fits =
      tw_take(pb, (unsigned long long)n, a.blk_entries,
              near ? &a.ctl->near_cur : &a.ctl->far_cur, near ? a.near_cap : a.far_cap, lane,
              &off) &&
      tw_take(rb, 1ull, a.blk_records, near ? &a.ctl->near_rec_cur : &a.ctl->far_rec_cur,
              near ? a.near_rec_cap : a.far_rec_cap, lane, &ri);
  if (!fits) {
    if (lane == 0) raise_flag(a.status, kFlagLogOverflow);
    return;
  }
  int32_t* pool = near ? a.near_pool : a.far_pool;
  for (int k = lane; k < n; k += 32) pool[off + k] = (int32_t)(stg[k] & kPwId);
  if (lane == 0) {
    (near ? a.near_keys : a.far_keys)[ri] =
        ((unsigned long long)(uint32_t)R.row << 32) | (unsigned long long)(uint32_t)within;
    TwChunk c;
    c.off = (long long)off;
    c.cnt = n;
    c.t = R.row;
    (near ? a.near_recs : a.far_recs)[ri] = c;
    unsigned* fo = near ? a.first_ovf_near : a.first_ovf_far;
    if (fo) {
      if (shared) atomicMin(fo + R.row, (unsigned)within);
      else if ((unsigned)within < fo[R.row]) fo[R.row] = (unsigned)within;
    }
  }
}

// Warp-collective: n staged split-list entries.  One warp's target: appended
// to one array (the tail of the warp's own pool block; a list that outgrows
// the block moves to a new one of twice its length).  Shared target: a chunk
// linked to the node, joined when its last piece ends.
__device__ __noinline__ void pw_flush_split(const PwArgs& a, PwWarpSmem& W, int t, int shared,
                                            int n, int lane) {
  if (n == 0) return;
  if (!shared) {
    unsigned long long off = W.s_off;
    const int len = W.s_len;
    TwBlk& b = W.al.s;
    if (off + (unsigned long long)(len + n) > b.end) {
      unsigned long long g = 0;
      int ok = 1;
      const unsigned long long want = 2ull * (unsigned long long)(len + n);
      const unsigned long long sz = want > a.blk_entries ? want : a.blk_entries;
      if (lane == 0) {
        g = atomicAdd(&a.ctl->s_cur, sz);
        ok = g + sz <= a.s_cap;
        if (!ok) raise_flag(a.status, kFlagLogOverflow);
      }
      g = __shfl_sync(0xffffffffu, g, 0);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      __syncwarp();  // b was read by every lane
      if (!ok) {     // children see an empty list (the result is discarded)
        if (lane == 0) {
          b.cur = b.end = 0;
          W.s_off = 0;
          W.s_len = 0;
        }
        __syncwarp();
        return;
      }
      for (int k = lane; k < len; k += 32) a.s_pool[g + k] = __ldcg(&a.s_pool[off + k]);
      if (lane == 0) {
        b.end = g + sz;
        W.s_off = g;
      }
      off = g;
    }
    for (int k = lane; k < n; k += 32) a.s_pool[off + len + k] = W.stg_b[k];
    __syncwarp();
    if (lane == 0) {
      W.s_len = len + n;
      b.cur = off + (unsigned long long)(len + n);
    }
    __syncwarp();
    return;
  }
  unsigned long long off = 0, ri = 0;
  const bool fits =
      tw_take(&W.al.s, (unsigned long long)n, a.blk_entries, &a.ctl->s_cur, a.s_cap, lane, &off) &&
      tw_take(&W.al.s_r, 1ull, a.blk_records, &a.ctl->s_rec_cur, a.s_rec_cap, lane, &ri);
  if (!fits) {
    if (lane == 0) raise_flag(a.status, kFlagLogOverflow);
    return;
  }
  for (int k = lane; k < n; k += 32) a.s_pool[off + k] = W.stg_b[k];
  if (lane == 0) {
    TwSChunk c;
    c.off = (long long)off;
    c.cnt = n;
    c.key = 0;
    c.pad = 0;
    c.next = atomicExch(&a.s_head[t], (int)ri);
    a.s_recs[ri] = c;
    atomicAdd(&a.s_cnt[t], n);
    atomicAdd(&a.s_nch[t], 1);
  }
}

// Warp-collective, by the warp that ends a shared target's last piece: the
// target's split-list chunks as one array (W.s_off, W.s_len).
__device__ __noinline__ void pw_join_split(const PwArgs& a, PwWarpSmem& W, int t, int lane) {
  const int nch = ld_volatile_i32_(&a.s_nch[t]);
  const int total = ld_volatile_i32_(&a.s_cnt[t]);
  int r = ld_volatile_i32_(&a.s_head[t]);
  if (nch <= 1) {
    if (lane == 0) {
      W.s_len = nch == 0 ? 0 : total;
      W.s_off = nch == 0 ? 0ull : (unsigned long long)a.s_recs[r].off;
    }
    __syncwarp();
    return;
  }
  unsigned long long off = 0;
  if (lane == 0) {
    atomicMax(&a.ctl->max_cmp, (unsigned)nch);
    off = atomicAdd(&a.ctl->s_cur, (unsigned long long)total);
  }
  off = __shfl_sync(0xffffffffu, off, 0);
  int len = 0;
  if (off + (unsigned long long)total > a.s_cap) {
    if (lane == 0) raise_flag(a.status, kFlagLogOverflow);
  } else {
    for (int k = 0; k < nch && r >= 0; ++k) {
      const TwSChunk c = a.s_recs[r];
      for (int e = lane; e < c.cnt; e += 32) a.s_pool[off + len + e] = __ldcg(&a.s_pool[c.off + e]);
      len += c.cnt;
      r = c.next;
    }
  }
  if (lane == 0) {
    W.s_off = off;
    W.s_len = len;
  }
  __syncwarp();
}

// Warp-collective: the stack and the source candidates from `cur` on become
// continuation pieces for other warps.  A target that was run by one warp so
// far becomes shared first: its counts go to the row counters and its split
// list becomes the first chunk.  The row's place may still be on its way here: a
// leaf target can be handed off before anything was flushed (budget 1, a stack
// full after a few refining windows, hungry warps), so the copy is waited for.
__device__ __noinline__ void pw_hand_off(const PwArgs& a, PwWarpSmem& W, const PwPiece pc, int t,
                                         int t_leaf, int cur, int stk_n, int lane) {
  pw_copy_wait();  // (lane 0 issued the copy and reads the row)
  const int shared = (pc.flags & kPwShared) != 0;
  if (!shared) {
    const int s_len = t_leaf ? 0 : W.s_len;
    unsigned long long ri = 0;
    const bool fits = s_len == 0 || tw_take(&W.al.s_r, 1ull, a.blk_records, &a.ctl->s_rec_cur,
                                            a.s_rec_cap, lane, &ri);
    if (lane == 0) {
      a.far_cnt[t] = W.cnt[0];
      if (t_leaf) a.near_cnt[W.row[1].row] = W.cnt[1];
      a.s_head[t] = -1;
      if (s_len > 0 && fits) {
        TwSChunk c;
        c.off = (long long)W.s_off;
        c.cnt = s_len;
        c.key = 0;
        c.next = -1;
        c.pad = 0;
        a.s_recs[ri] = c;
        a.s_head[t] = (int)ri;
        a.s_cnt[t] = s_len;
        a.s_nch[t] = 1;
      }
      if (!fits) raise_flag(a.status, kFlagLogOverflow);
    }
  }
  unsigned long long off = 0;
  if (lane == 0 && stk_n > 0) off = atomicAdd(&a.ctl->spill_cur, (unsigned long long)stk_n);
  off = __shfl_sync(0xffffffffu, off, 0);
  int room = 1;
  if (off + (unsigned long long)stk_n > a.spill_cap) {
    if (lane == 0) raise_flag(a.status, kFlagLogOverflow);
    room = 0;
  }
  if (room)
    for (int j = lane; j < stk_n; j += 32) a.spill[off + j] = W.stk[j];
  const int np_sp = room ? (stk_n + kPwSpillGroup - 1) / kPwSpillGroup : 0;
  const int n_inh = (int)pc.n_inh;
  const int src_len = n_inh + (int)(pc.flags & kPwSibling);
  const int rem = n_inh > cur ? n_inh - cur : 0;
  const int sib = (pc.flags & kPwSibling) && cur < src_len;
  const int np_in = rem > 0 ? (rem + kPwInhGroup - 1) / kPwInhGroup : sib;
  const int np = np_sp + np_in;
  unsigned slot = 0;
  int n_ok = 0;
  if (lane == 0) {
    if (np > 0) {
      slot = atomicAdd(&a.ctl->q_tail, (unsigned)np);
      n_ok = slot >= a.q_cap ? 0 : (int)min((unsigned)np, a.q_cap - slot);
      if (n_ok < np) {
        raise_flag(a.status, kFlagLogOverflow);
        a.ctl->stop = 1u;  // dropped pieces: the walk is re-run with a longer queue
      }
    }
    // counted before any of them can be taken (and finished) by another warp
    atomicAdd(&a.pieces_left[t], n_ok + (shared ? 0 : 1));
    __threadfence();
  }
  slot = __shfl_sync(0xffffffffu, slot, 0);
  n_ok = __shfl_sync(0xffffffffu, n_ok, 0);
  __syncwarp();
  for (int k = lane; k < n_ok; k += 32) {
    PwPiece q;
    q.et = pc.et;
    q.flags = kPwShared;
    q.n_spill = q.n_inh = 0;
    q.spill_off = q.inh_off = 0;
    if (k < np_sp) {
      q.spill_off = off + (unsigned long long)k * kPwSpillGroup;
      q.n_spill = (uint32_t)min(kPwSpillGroup, stk_n - k * kPwSpillGroup);
    } else {
      const int j = k - np_sp;
      q.inh_off = pc.inh_off + (unsigned long long)(cur + j * kPwInhGroup);
      q.n_inh = (uint32_t)max(0, min(kPwInhGroup, rem - j * kPwInhGroup));
      if (sib && j == np_in - 1) q.flags |= kPwSibling;
    }
    a.queue[slot + k] = q;
    pw_store_release(&a.q_ready[slot + k], 1u);
  }
  __syncwarp();
}

// Both children's records: 32 bytes, one load.
__device__ __forceinline__ void pw_load_pair(const float4* p, float4& c0, float4& c1) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(c0.x), "=f"(c0.y), "=f"(c0.z), "=f"(c0.w), "=f"(c1.x), "=f"(c1.y), "=f"(c1.z),
        "=f"(c1.w)
      : "l"(p));
}

// The MAC of target (centre and extent T) and source record c, in the
// reference's fp32 operation order (_interactions_impl.py:338-395).
template <int kMac>
__device__ __forceinline__ bool pw_accept(const float4 T, const float4 c, const PwArgs& a) {
  const float dx = __fsub_rn(T.x, c.x);
  const float dy = __fsub_rn(T.y, c.y);
  const float dz = __fsub_rn(T.z, c.z);
  float d2 = __fmul_rn(dx, dx);
  d2 = __fadd_rn(d2, __fmul_rn(dy, dy));
  d2 = __fadd_rn(d2, __fmul_rn(dz, dz));
  float lhs;
  if (kMac == kTwEngblom)
    lhs = __fadd_rn(fmax_nan(T.w, c.w), __fmul_rn(a.theta, fmin_nan(T.w, c.w)));
  else
    lhs = __fadd_rn(T.w, c.w);
  return d2 > 0.0f && __fmul_rn(lhs, lhs) <= __fmul_rn(a.theta_sq, d2);
}

// Whether a source that is not far is kept (near, or split on the target's
// side).  Leaf target: a leaf source is near, an internal one splits.
// Internal target: it splits itself unless the source is larger (canonical
// orientation, :1444-1454: the lower id splits on a tie).
template <bool kLeaf>
__device__ __forceinline__ bool pw_keep(int t, float et, int s, float es) {
  const bool s_leaf = s < 0;  // kPwLeaf
  return kLeaf ? s_leaf : (s_leaf || (t < s ? et >= es : !(es >= et)));
}

// One piece of target t: its candidates evaluated 64 at a time -- two per
// lane: the children of 32 stack words, or, while the stack is short, the
// next 64 source entries -- until none are left or the rest was handed off.
// Returns whether the target is (now) shared.
template <int kMac, bool kLeaf>
__device__ __forceinline__ bool pw_run_piece(const PwArgs& a, PwSmem& sm, PwWarpSmem& W,
                                             const PwPiece pc, int t, const float4 Tc, int lane,
                                             unsigned lt) {
  const int n_inh = (int)pc.n_inh;
  const int src_len = n_inh + (int)(pc.flags & kPwSibling);
  const uint32_t* src = a.s_pool + pc.inh_off;
  bool shared = (pc.flags & kPwShared) != 0;
  int cur = 0, stk_n = (int)pc.n_spill, steps = 0, lanes = 0;
  int n_a = 0, n_b = 0, tot_a = 0, tot_b = 0;
  if (lane < stk_n) W.stk[lane] = __ldcg(&a.spill[pc.spill_off + lane]);
  __syncwarp();
  while (stk_n > 0 || cur < src_len) {
    uint32_t e0 = 0u, e1 = 0u;
    float4 c0, c1;
    int s0, s1;
    bool act0, act1;
    if (stk_n >= 32 || cur >= src_len) {
      const int m = stk_n < 32 ? stk_n : 32;
      stk_n -= m;
      act0 = act1 = lane < m;
      if (act0) e0 = W.stk[stk_n + lane];
      e1 = e0 + 1u;
      const uint32_t slot = e0 & kPwSlotMask;
      pw_load_pair(a.sc + slot, c0, c1);
      const int2 k = __ldg(reinterpret_cast<const int2*>(a.sid + slot));
      s0 = k.x;
      s1 = k.y;
      lanes += 2 * m;
    } else {
      const int q0 = cur + 2 * lane, q1 = q0 + 1;
      act0 = q0 < src_len;
      act1 = q1 < src_len;
      if (act0) e0 = q0 < n_inh ? __ldcg(src + q0) : (pc.et ^ 1u);
      if (act1) e1 = q1 < n_inh ? __ldcg(src + q1) : (pc.et ^ 1u);
      const uint32_t l0 = e0 & kPwSlotMask, l1 = e1 & kPwSlotMask;
      c0 = __ldg(a.sc + l0);
      c1 = __ldg(a.sc + l1);
      s0 = __ldg(a.sid + l0);
      s1 = __ldg(a.sid + l1);
      lanes += src_len - cur < 64 ? src_len - cur : 64;
      cur += 64;
    }
    ++steps;
    if (act0) atomicAdd(&sm.hist[e0 >> 24], 1u);
    if (act1) atomicAdd(&sm.hist[e1 >> 24], 1u);
    const bool a0 = act0 && pw_accept<kMac>(Tc, c0, a);
    const bool a1 = act1 && pw_accept<kMac>(Tc, c1, a);
    const bool b0 = act0 && !a0 && pw_keep<kLeaf>(t, Tc.w, s0, c0.w);
    const bool b1 = act1 && !a1 && pw_keep<kLeaf>(t, Tc.w, s1, c1.w);
    const bool r0 = act0 && !a0 && !b0, r1 = act1 && !a1 && !b1;
    // (the ballots also order this window's stack reads before the pushes)
    const unsigned mR0 = __ballot_sync(0xffffffffu, r0), mR1 = __ballot_sync(0xffffffffu, r1);
    const unsigned mA0 = __ballot_sync(0xffffffffu, a0), mA1 = __ballot_sync(0xffffffffu, a1);
    const unsigned mB0 = __ballot_sync(0xffffffffu, b0), mB1 = __ballot_sync(0xffffffffu, b1);
    __syncwarp();
    // siblings stay side by side (a lane's two candidates in order)
    const int iR = stk_n + __popc(mR0 & lt) + __popc(mR1 & lt);
    const int iA = n_a + __popc(mA0 & lt) + __popc(mA1 & lt);
    const int iB = n_b + __popc(mB0 & lt) + __popc(mB1 & lt);
    if (r0) W.stk[iR] = (e0 & ~kPwSlotMask) + kPwGen + 2u * (uint32_t)s0;
    if (r1) W.stk[iR + (r0 ? 1 : 0)] = (e1 & ~kPwSlotMask) + kPwGen + 2u * (uint32_t)s1;
    if (a0) W.stg_a[iA] = (uint32_t)s0;
    if (a1) W.stg_a[iA + (a0 ? 1 : 0)] = (uint32_t)s1;
    if (b0) W.stg_b[iB] = kLeaf ? (uint32_t)s0 : e0 + kPwGen;
    if (b1) W.stg_b[iB + (b0 ? 1 : 0)] = kLeaf ? (uint32_t)s1 : e1 + kPwGen;
    stk_n += __popc(mR0) + __popc(mR1);
    n_a += __popc(mA0) + __popc(mA1);
    n_b += __popc(mB0) + __popc(mB1);
    __syncwarp();
    if (n_a > kPwStg - 64) {
      pw_flush_row(a, W, 0, shared, n_a, lane);
      __syncwarp();
      tot_a += n_a;
      n_a = 0;
    }
    if (n_b > kPwStg - 64) {
      if (kLeaf) pw_flush_row(a, W, 1, shared, n_b, lane);
      else pw_flush_split(a, W, t, shared, n_b, lane);
      __syncwarp();
      tot_b += n_b;
      n_b = 0;
    }
    // Hand the rest off when the budget is spent, when the stack could not
    // take another window's pushes, or when many warps wait for work.
    bool give = steps >= a.budget || stk_n > kPwStk - 64;
    if ((steps & 31) == 0 && !give) {
      int hungry = 0;
      if (lane == 0)
        hungry = (int)(pw_load_relaxed(&a.ctl->q_head) - pw_load_relaxed(&a.ctl->q_tail)) >
                 a.hungry;
      give = __shfl_sync(0xffffffffu, hungry, 0) != 0;
    }
    if (give && (stk_n > 0 || cur < src_len)) {
      pw_hand_off(a, W, pc, t, kLeaf, cur, stk_n, lane);
      shared = true;
      break;
    }
  }
  pw_copy_wait();  // also where nothing is flushed: the row is read and reused after this
  tot_a += n_a;
  tot_b += n_b;
  pw_flush_row(a, W, 0, shared, n_a, lane);
  if (kLeaf) pw_flush_row(a, W, 1, shared, n_b, lane);
  else pw_flush_split(a, W, t, shared, n_b, lane);
  if (lane == 0) {
    W.st.acc += (unsigned long long)tot_a;
    if (kLeaf) W.st.near_ += (unsigned long long)tot_b;
    W.st.ref += (unsigned long long)(lanes - tot_a - (kLeaf ? tot_b : 0));
    W.st.steps += (unsigned long long)steps;
    W.st.lanes += (unsigned long long)lanes;
  }
  __syncwarp();
  return shared;
}

template <int kMac>
__global__ void __launch_bounds__(kPwThreads, kPwBlocksPerSM)
    k_pair_walk(const __grid_constant__ PwArgs a) {
  extern __shared__ __align__(16) unsigned char pw_smem_raw[];
  PwSmem& sm = *reinterpret_cast<PwSmem*>(pw_smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PwWarpSmem& W = sm.w[warp];
  for (int i = threadIdx.x; i < kTwHist; i += kPwThreads) sm.hist[i] = 0;
  if (threadIdx.x < 8) sm.sums[threadIdx.x] = 0ull;
  if (lane == 0) {
    W.al.far = W.al.near_ = W.al.s = W.al.far_r = W.al.near_r = W.al.s_r = TwBlk{0ull, 0ull};
    W.st = TwWarpStats{0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
    W.t_mark = clock64();
  }
  __syncthreads();
  const unsigned lt = lanemask_lt_();
  unsigned fin = 0;   // targets this warp finished and has not reported (lane 0)
  bool have = false;  // pc holds the next piece (a finished target's left child)
  int room = 1;       // whether its sibling was queued (lane 0)
  PwPiece pc;
  while (true) {
    if (!have) {
      // ---- the next queue slot, in ticket order; a bounded wait for its piece
      unsigned ticket = 0;
      int got = 0;
      if (lane == 0) {
        ticket = atomicAdd(&a.ctl->q_head, 1u);
        if (ticket < a.q_cap && pw_load_relaxed(&a.q_ready[ticket])) {
          got = 1;
        } else {
          if (fin) {
            if (atomicAdd(&a.ctl->finished, fin) + fin >= (unsigned)a.n_targets) a.ctl->stop = 1u;
            fin = 0;
          }
          unsigned sleep = 32;
          for (uint32_t idle = 0;; ++idle) {
            if (idle >= a.spin_limit) {
              raise_flag(a.status, kFlagTimeout);
              a.ctl->stop = 1u;
              break;
            }
            if (ticket < a.q_cap && pw_load_relaxed(&a.q_ready[ticket])) {
              got = 1;
              break;
            }
            if ((idle & 3u) == 3u && pw_load_relaxed(&a.ctl->stop)) break;
            __nanosleep(sleep);
            sleep = sleep < 512 ? sleep * 2 : 512;
          }
        }
        if (got) pw_load_acquire(&a.q_ready[ticket]);
      }
      got = __shfl_sync(0xffffffffu, got, 0);
      ticket = __shfl_sync(0xffffffffu, ticket, 0);
      __syncwarp();
      if (!got) break;
      const uint4* q = reinterpret_cast<const uint4*>(a.queue + ticket);
      const uint4 q0 = __ldcg(q), q1 = __ldcg(q + 1);
      pc.et = q0.x;
      pc.flags = q0.y;
      pc.n_spill = q0.z;
      pc.n_inh = q0.w;
      pc.spill_off = (unsigned long long)q1.x | ((unsigned long long)q1.y << 32);
      pc.inh_off = (unsigned long long)q1.z | ((unsigned long long)q1.w << 32);
    }
    have = false;
    const uint32_t slot = pc.et & kPwSlotMask;
    const float4 Tc = __ldg(a.sc + slot);
    const int t_id = __ldg(a.sid + slot);
    const bool t_leaf = t_id < 0;
    const int t = t_id & (int)kPwId;
    if (lane == 0) {
      const long long now = clock64();
      W.st.idle += (unsigned long long)(now - W.t_mark);
      W.t_mark = now;
      W.st.pieces += 1ull;
      W.cnt[0] = W.cnt[1] = 0;
      W.s_off = W.al.s.cur;
      W.s_len = 0;
      // the rows' places arrive while the first candidates are evaluated
      pw_copy16(&W.row[0], a.rows + t);
      if (t_leaf) pw_copy16(&W.row[1], a.near_rows + t);
    }
    __syncwarp();
    const bool shared = t_leaf ? pw_run_piece<kMac, true>(a, sm, W, pc, t, Tc, lane, lt)
                               : pw_run_piece<kMac, false>(a, sm, W, pc, t, Tc, lane, lt);
    // ---- the piece is done; the target too, unless other pieces are left
    int complete = 1;
    if (shared) {
      if (lane == 0) {
        __threadfence();
        complete = atomicSub(&a.pieces_left[t], 1) == 1;
        if (complete) __threadfence();
      }
      complete = __shfl_sync(0xffffffffu, complete, 0);
      __syncwarp();
      if (complete && !t_leaf) pw_join_split(a, W, t, lane);
    } else if (lane == 0) {
      a.far_cnt[t] = W.cnt[0];
      if (t_leaf) a.near_cnt[W.row[1].row] = W.cnt[1];
    }
    if (lane == 0) {
      fin += (unsigned)complete;
      const long long now = clock64();
      W.st.busy += (unsigned long long)(now - W.t_mark);
      W.t_mark = now;
    }
    // both children inherit the split list: the right one is queued, this warp
    // goes on with the left one.  Not after a push that found no room: the walk
    // is re-run with a longer queue anyway, and a chain of left children that no
    // queue entry pays for ends only if the tree does (the children that a C
    // caller gives may form a cycle).  The push before is the one looked at,
    // so that nothing waits for this one's round trip (walk of 16 M particles
    // 7.23 -> 7.25 ms, of 1 M 0.77 -> 0.78).
    const bool go = complete && !t_leaf && __shfl_sync(0xffffffffu, room, 0) != 0;
    room = 1;
    if (go) {
      pc.et = (2u * (uint32_t)t) | ((pc.et & ~kPwSlotMask) + kPwGen);
      pc.flags = kPwSibling;
      pc.n_spill = 0;
      pc.n_inh = (uint32_t)W.s_len;
      pc.spill_off = 0;
      pc.inh_off = W.s_off;
      __syncwarp();
      if (lane == 0) {
        const unsigned qs = atomicAdd(&a.ctl->q_tail, 1u);
        if (qs < a.q_cap) {
          PwPiece q = pc;
          q.et += 1u;
          a.queue[qs] = q;
          pw_store_release(&a.q_ready[qs], 1u);
        } else {
          room = 0;
          raise_flag(a.status, kFlagLogOverflow);
          a.ctl->stop = 1u;
        }
      }
      have = true;
    }
  }
  // ---- unused record slots of this warp's last blocks: empty chunks
  __syncwarp();
  const TwChunk none{0, 0, 0};
  for (unsigned long long k = W.al.far_r.cur + lane; k < W.al.far_r.end; k += 32) {
    a.far_keys[k] = 0ull;
    a.far_recs[k] = none;
  }
  for (unsigned long long k = W.al.near_r.cur + lane; k < W.al.near_r.end; k += 32) {
    a.near_keys[k] = 0ull;
    a.near_recs[k] = none;
  }
  // ---- statistics: one atomic per CTA and counter
  if (lane == 0) {
    W.st.idle += (unsigned long long)(clock64() - W.t_mark);
    const TwWarpStats& q = W.st;
    const unsigned long long v[8] = {q.acc, q.near_, q.ref, q.busy, q.idle, q.pieces, q.steps,
                                     q.lanes};
    for (int k = 0; k < 8; ++k)
      if (v[k]) atomicAdd(&sm.sums[k], v[k]);
  }
  __syncthreads();
  if (threadIdx.x < 8 && sm.sums[threadIdx.x]) {
    unsigned long long* out[8] = {&a.ctl->acc_sides,   &a.ctl->near_sides,  &a.ctl->ref_sides,
                                  &a.ctl->busy_cycles, &a.ctl->idle_cycles, &a.ctl->pieces,
                                  &a.ctl->steps,       &a.ctl->lanes};
    atomicAdd(out[threadIdx.x], sm.sums[threadIdx.x]);
  }
  for (int i = threadIdx.x; i < kTwHist; i += kPwThreads)
    if (sm.hist[i]) atomicAdd(&a.gen_hist[i], sm.hist[i]);
}

}  // namespace
}  // namespace ygx
