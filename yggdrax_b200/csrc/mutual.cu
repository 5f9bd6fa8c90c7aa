// Canonical mutual dual-tree walk: every unordered node pair once
// (dual_tree_walk_mutual, yggdrax/_interactions_impl.py:6357-6560).
//
// The reference walks a fixed-capacity wavefront breadth-first and appends
// accepted / near pairs to flat lists in wavefront order, children in the
// order of their parents, each parent's children in the refinement order of
// _count_refine_pairs_single (:174-221).  Those orders are part of its
// output, so each generation here is a stable compaction: every pair is
// evaluated (MAC, action, number of children), prefix sums give every child,
// far and near pair its slot, and the pairs are written there.  All
// generations run in one cooperative launch (genwalk.cuh); the counters
// follow the reference's overflow rules, and the host reads them once.
#include "genwalk.cuh"

namespace ygx {

namespace {

constexpr uint32_t kMutFarOver = 1u << 0;
constexpr uint32_t kMutNearOver = 1u << 1;
constexpr uint32_t kMutQueueOver = 1u << 2;
constexpr uint32_t kMutBadInput = 1u << 3;
constexpr int kMutMaxGens = 1 << 16;

struct MutualCtl {
  long long far_n;   // far pairs the flat list would hold (counted past its capacity)
  long long near_n;
  unsigned int flags;
  unsigned int gens;
  unsigned int arrived;   // grid barrier
  unsigned int timeout;
};

struct MutualArgs {
  const float4* rec;   // per node: centre, radius
  const int2* kids;    // per node: children, -1 on leaves
  int64_t total;
  float theta_sq;
  int2* wf[2];         // wavefronts of `cap` pairs
  uint8_t* kind;       // per pair of the current wavefront
  int64_t cap, far_cap, near_cap;
  int index_bits;
  void *far_a, *far_b, *near_a, *near_b;
  GenTotals* totals;
  MutualCtl* ctl;
  uint32_t spin_limit;
};

// What becomes of a pair (kind): its refinement case in the low bits -- 0
// none, 1 both children of a diagonal pair, 2 both sides of an off-diagonal
// pair, 3 the first node only, 4 the second node only -- or far / near.
constexpr uint8_t kMutFar = 8, kMutNear = 16;

__global__ void k_mut_prepare(const void* __restrict__ left, const void* __restrict__ right,
                              int index_bits, const float* __restrict__ centers,
                              const float* __restrict__ radii, int64_t total, int32_t root,
                              float4* __restrict__ rec, int2* __restrict__ kids,
                              int2* __restrict__ wf0, MutualCtl* __restrict__ ctl) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += (int64_t)gridDim.x * blockDim.x) {
    rec[k] = make_float4(centers[3 * k], centers[3 * k + 1], centers[3 * k + 2], radii[k]);
    kids[k] = make_int2((int32_t)load_idx(left, index_bits, k),
                        (int32_t)load_idx(right, index_bits, k));
    if (k == 0) {
      wf0[0] = make_int2(root, root);
      *ctl = MutualCtl{0, 0, 0u, 0u, 0u, 0u};
    }
  }
}

__device__ __forceinline__ uint8_t mut_evaluate(const MutualArgs& a, int2 p, bool* bad) {
  const int32_t sa = p.x, sb = p.y;
  if (!(sa >= 0 && sb >= 0 && sa < a.total && sb < a.total)) {
    *bad |= sa >= a.total || sb >= a.total;
    return 0;
  }
  const float4 A = a.rec[sa], B = a.rec[sb];
  const bool a_leaf = a.kids[sa].x < 0, b_leaf = a.kids[sb].x < 0, same = sa == sb;
  // delta = centers[b] - centers[a]; sum of squares in written order
  const float dx = __fsub_rn(B.x, A.x), dy = __fsub_rn(B.y, A.y), dz = __fsub_rn(B.z, A.z);
  const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
  const float rs = __fadd_rn(A.w, B.w);
  // theta * d > r_a + r_b, squared, strict; never for a self-pair
  if (!same && __fmul_rn(a.theta_sq, d2) > __fmul_rn(rs, rs)) return kMutFar;
  if (a_leaf && b_leaf) return same ? 0 : kMutNear;
  const bool split_a = !a_leaf && (same || b_leaf || A.w >= B.w);
  const bool split_b = !b_leaf && (same || a_leaf || B.w > A.w);
  return split_a && split_b ? (same ? 1 : 2) : split_a ? 3 : split_b ? 4 : 0;
}
__device__ __forceinline__ int mut_children(uint8_t kind) {
  return kind == 1 ? 3 : kind == 2 ? 4 : kind == 3 || kind == 4 ? 2 : 0;
}

template <typename T>
__device__ __forceinline__ void put_pair(void* a, void* b, long long slot, int2 p) {
  reinterpret_cast<T*>(a)[slot] = (T)p.x;
  reinterpret_cast<T*>(b)[slot] = (T)p.y;
}

__device__ __forceinline__ void mut_fill(void* list, int index_bits, long long from,
                                         long long cap) {
  for (long long k = from + (long long)blockIdx.x * blockDim.x + threadIdx.x; k < cap;
       k += (long long)gridDim.x * blockDim.x)
    store_idx(list, index_bits, k, -1);
}

// The whole walk.  A list overflows when any of a generation's pairs gets a
// slot at or past its capacity; the wavefront keeps its first `cap` children;
// the walk stops after the generation that overflowed (_flat_append and the
// push rules).  Every CTA follows the same counters.  500,000 Plummer
// particles, leaf 32, theta 0.6 (58 generations): 0.89 ms, and the call 1.0 ms
// against 3.6 ms with eight launches and a read-back per generation.
__global__ void __launch_bounds__(kGenThreads, 2) k_mut_walk(const MutualArgs a) {
  long long size = 1, far_n = 0, near_n = 0;
  unsigned flags = 0, gens = 0, target = 0;
  int cur = 0;
  bool ok = true;
  while (size > 0 && flags == 0 && gens < (unsigned)kMutMaxGens) {
    const int2* wf = a.wf[cur];
    int2* next = a.wf[cur ^ 1];
    const int64_t slice = gen_slice(size);
    const int64_t lo = blockIdx.x * slice, hi = lo + slice < size ? lo + slice : size;
    unsigned long long nc = 0, nf = 0, nn = 0;
    bool bad = false;
    for (int64_t i = lo + threadIdx.x; i < hi; i += kGenThreads) {
      const uint8_t kd = mut_evaluate(a, __ldcg(wf + i), &bad);
      a.kind[i] = kd;
      nc += mut_children(kd);
      nf += kd == kMutFar;
      nn += kd == kMutNear;
    }
    if (bad) atomicOr(&a.ctl->flags, kMutBadInput);
    gen_publish(nc, nf, nn, a.totals);
    if (!(ok = gen_barrier(&a.ctl->arrived, &target, a.spin_limit))) break;
    GenTotals pre, all;
    gen_prefix(a.totals, &pre, &all);
    flags = __ldcg(&a.ctl->flags);
    for (int64_t c0 = lo; c0 < hi; c0 += kGenThreads) {
      const int64_t i = c0 + threadIdx.x;
      const uint8_t kd = i < hi ? a.kind[i] : 0;
      // children (at most 4 x 512) | far << 12 | near << 22
      const unsigned v = (unsigned)mut_children(kd) | (kd == kMutFar ? 1u << 12 : 0u) |
                         (kd == kMutNear ? 1u << 22 : 0u);
      unsigned sum;
      const unsigned at = gen_block_scan(v, &sum);
      if (kd) {
        const int2 p = __ldcg(wf + i);
        if (kd == kMutFar) {
          const long long slot = far_n + (long long)pre.x + ((at >> 12) & 1023u);
          if (slot < a.far_cap) {
            if (a.index_bits == 32) put_pair<int32_t>(a.far_a, a.far_b, slot, p);
            else put_pair<int64_t>(a.far_a, a.far_b, slot, p);
          }
        } else if (kd == kMutNear) {
          const long long slot = near_n + (long long)pre.y + (at >> 22);
          if (slot < a.near_cap) {
            if (a.index_bits == 32) put_pair<int32_t>(a.near_a, a.near_b, slot, p);
            else put_pair<int64_t>(a.near_a, a.near_b, slot, p);
          }
        } else {
          const int2 A = a.kids[p.x], B = a.kids[p.y];
          const int64_t base = (int64_t)pre.child + (at & 4095u);
          // children in _count_refine_pairs_single order, canonical (min, max)
          auto put = [&](int k, int x, int y) {
            if (base + k < a.cap) next[base + k] = x < y ? make_int2(x, y) : make_int2(y, x);
          };
          if (kd == 1) {
            put(0, A.x, A.x);
            put(1, A.x, A.y);
            put(2, A.y, A.y);
          } else if (kd == 2) {
            put(0, A.x, B.x);
            put(1, A.x, B.y);
            put(2, A.y, B.x);
            put(3, A.y, B.y);
          } else if (kd == 3) {
            put(0, A.x, p.y);
            put(1, A.y, p.y);
          } else {
            put(0, p.x, B.x);
            put(1, p.x, B.y);
          }
        }
      }
      pre.child += sum & 4095u;
      pre.x += (sum >> 12) & 1023u;
      pre.y += sum >> 22;
    }
    const long long children = (long long)all.child, f = (long long)all.x, n = (long long)all.y;
    if (f > 0 && far_n + f > a.far_cap) flags |= kMutFarOver;
    if (n > 0 && near_n + n > a.near_cap) flags |= kMutNearOver;
    if (children > a.cap) flags |= kMutQueueOver;
    far_n += f;
    near_n += n;
    size = children < a.cap ? children : a.cap;
    cur ^= 1;
    ++gens;
    // the next generation reads what every CTA wrote, and writes where this
    // one read
    if (!(ok = gen_barrier(&a.ctl->arrived, &target, a.spin_limit))) break;
  }
  // -1 past the lists' ends
  mut_fill(a.far_a, a.index_bits, far_n, a.far_cap);
  mut_fill(a.far_b, a.index_bits, far_n, a.far_cap);
  mut_fill(a.near_a, a.index_bits, near_n, a.near_cap);
  mut_fill(a.near_b, a.index_bits, near_n, a.near_cap);
  if (threadIdx.x == 0) {
    if (!ok) a.ctl->timeout = 1u;
    if (blockIdx.x == 0) {
      a.ctl->far_n = far_n;
      a.ctl->near_n = near_n;
      atomicOr(&a.ctl->flags, flags);
      a.ctl->gens = size > 0 && flags == 0 ? (unsigned)kMutMaxGens + 1u : gens;
    }
  }
}

struct MutualScratch {
  MutualCtl* ctl;
  float4* rec;
  int2* kids;
  int2* wf[2];
  uint8_t* kind;
  GenTotals* totals;
};

MutualScratch carve_mutual(Arena& a, int64_t total, int64_t cap) {
  MutualScratch s;
  s.ctl = a.take<MutualCtl>(1);
  s.rec = a.take<float4>(total);
  s.kids = a.take<int2>(total);
  for (int k = 0; k < 2; ++k) s.wf[k] = a.take<int2>(cap);
  s.kind = a.take<uint8_t>(cap);
  s.totals = a.take<GenTotals>(kGenMaxBlocks);
  return s;
}

}  // namespace

}  // namespace ygx

extern "C" {

size_t ygx_mutual_walk_workspace_size(int64_t total, int64_t max_pair_queue) {
  ygx::Arena a{nullptr, 0, 0};
  ygx::carve_mutual(a, total > 0 ? total : 1, max_pair_queue > 0 ? max_pair_queue : 1);
  return a.used + 256;
}

int ygx_mutual_walk(const void* left_full, const void* right_full, int index_bits,
                    const float* centers, const float* radii, int64_t total, float theta,
                    int64_t root, int64_t max_pair_queue, int64_t far_cap, int64_t near_cap,
                    void* far_a, void* far_b, void* near_a, void* near_b, int64_t* counts_out,
                    uint32_t* flags_out, int* gens_out, void* ws, size_t ws_bytes,
                    cudaStream_t stream) {
  if (total < 1 || total > INT32_MAX || root < 0 || root >= total || max_pair_queue < 1 ||
      max_pair_queue > INT32_MAX || far_cap < 1 || near_cap < 1 ||
      (index_bits != 32 && index_bits != 64) || !left_full || !right_full || !centers ||
      !radii || !far_a || !far_b || !near_a || !near_b || !counts_out || !flags_out || !ws)
    return YGX_ERR_ARG;
  if (ws_bytes < ygx_mutual_walk_workspace_size(total, max_pair_queue)) return YGX_ERR_ARG;
  ygx::Arena a{(char*)ws, 0, ws_bytes};
  ygx::MutualScratch s = ygx::carve_mutual(a, total, max_pair_queue);
  const int64_t Q = max_pair_queue;
  // theta^2 in fp32 (jnp.asarray(theta, centers.dtype) ** 2)
  const float th = theta;
  const float theta_sq = th * th;
  ygx::k_mut_prepare<<<ygx::grid_for(total, 256), 256, 0, stream>>>(
      left_full, right_full, index_bits, centers, radii, total, (int32_t)root, s.rec, s.kids,
      s.wf[0], s.ctl);
  YGX_CHECK_LAUNCH();
  ygx::MutualArgs args{s.rec,   s.kids,     total,       theta_sq,   {s.wf[0], s.wf[1]},
                       s.kind,  Q,          far_cap,     near_cap,   index_bits,
                       far_a,   far_b,      near_a,      near_b,     s.totals,
                       s.ctl,   (uint32_t)ygx::g_tune.spin_limit};
  const int grid = ygx::gen_grid(ygx::k_mut_walk);
  void* params[] = {&args};
  if (grid < 1 || cudaLaunchCooperativeKernel((const void*)ygx::k_mut_walk, dim3((unsigned)grid),
                                              dim3(ygx::kGenThreads), params, 0,
                                              stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return YGX_ERR_CUDA;
  }
  YGX_CHECK_LAUNCH();
  ygx::MutualCtl h;
  if (cudaMemcpyAsync(&h, s.ctl, sizeof(h), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess)
    return YGX_ERR_CUDA;
  if (h.timeout) return YGX_ERR_TIMEOUT;
  const bool endless = h.gens > (unsigned)ygx::kMutMaxGens;
  const int rc = endless ? YGX_ERR_QUEUE_OVERFLOW : YGX_OK;
  const int gen = endless ? ygx::kMutMaxGens : (int)h.gens;
  counts_out[0] = h.far_n;
  counts_out[1] = h.near_n;
  flags_out[0] = h.flags;
  if (gens_out) gens_out[0] = gen;
  if (h.flags & ygx::kMutBadInput) return YGX_ERR_ARG;
  return rc;
}

}  // extern "C"
