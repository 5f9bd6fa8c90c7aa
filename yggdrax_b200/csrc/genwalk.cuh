// Breadth-first walks in one launch: the pieces shared by the mutual walk
// (mutual.cu) and the native octree walk (octwalk.cu).
//
// Their wavefronts are stable compactions: the children of a generation's
// pairs, and the pairs it accepts, keep the wavefront's order.  Every CTA of a
// cooperative launch owns one contiguous slice of the wavefront.  Per
// generation it evaluates its slice and publishes the slice's totals, and
// after a grid barrier it knows its slice's offsets (the sums of the slices
// before it) and writes children and pairs in place, a chunk of the block at a
// time; a second barrier ends the generation.  Two barriers replace the eight
// launches and the host's read of the counters that a generation took, which
// were what the walk spent its time on: most of its generations hold few
// pairs (the figures stand in mutual.cu and octwalk.cu).
#pragma once
#include "common.cuh"

namespace ygx {
namespace {

constexpr int kGenThreads = 512;
constexpr int kGenWarps = kGenThreads / 32;
constexpr int kGenMaxBlocks = kNumSMs * 2;  // at most kGenThreads: one thread per slice total

// Totals of one slice: children, and the two kinds of emitted pairs.
struct GenTotals {
  unsigned long long child, x, y;
};

// Barrier over the launch's CTAs (all resident).  `arrived` counts arrivals
// since the launch, `target` is this barrier's.  A wait longer than `limit`
// polls gives up: false, in every thread of the CTA.
__device__ __forceinline__ bool gen_barrier(unsigned* arrived, unsigned* target, uint32_t limit) {
  __shared__ int s_ok;
  __syncthreads();
  *target += gridDim.x;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrived, 1u);
    int ok = 1;
    unsigned v;
    for (uint32_t k = 0;; ++k) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
      if ((int)(v - *target) >= 0) break;
      if (k >= limit) {
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  __syncthreads();
  return ok;
}

// The slice of CTA b in a wavefront of n pairs: whole chunks of the block.
__device__ __forceinline__ int64_t gen_slice(int64_t n) {
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  return (per + kGenThreads - 1) / kGenThreads * kGenThreads;
}

// Block-wide sum of a per-thread triple, published as the slice's totals.
__device__ __forceinline__ void gen_publish(unsigned long long child, unsigned long long x,
                                            unsigned long long y, GenTotals* out) {
  __shared__ GenTotals s[kGenWarps];
  for (int o = 16; o > 0; o >>= 1) {
    child += __shfl_xor_sync(0xffffffffu, child, o);
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
  }
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = GenTotals{child, x, y};
  __syncthreads();
  if (threadIdx.x == 0) {
    GenTotals t{0, 0, 0};
    for (int w = 0; w < kGenWarps; ++w) {
      t.child += s[w].child;
      t.x += s[w].x;
      t.y += s[w].y;
    }
    out[blockIdx.x] = t;
  }
}

// Sums of the slices before this CTA's (pre) and of all slices (all).
__device__ __forceinline__ void gen_prefix(const GenTotals* totals, GenTotals* pre,
                                           GenTotals* all) {
  __shared__ GenTotals s_pre[kGenWarps], s_all[kGenWarps];
  GenTotals t{0, 0, 0};
  if (threadIdx.x < gridDim.x) {
    const unsigned long long* p = &totals[threadIdx.x].child;
    t.child = __ldcg(p);
    t.x = __ldcg(p + 1);
    t.y = __ldcg(p + 2);
  }
  const bool before = threadIdx.x < blockIdx.x;
  GenTotals b = before ? t : GenTotals{0, 0, 0};
  for (int o = 16; o > 0; o >>= 1) {
    t.child += __shfl_xor_sync(0xffffffffu, t.child, o);
    t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
    t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
    b.child += __shfl_xor_sync(0xffffffffu, b.child, o);
    b.x += __shfl_xor_sync(0xffffffffu, b.x, o);
    b.y += __shfl_xor_sync(0xffffffffu, b.y, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_all[threadIdx.x >> 5] = t;
    s_pre[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  GenTotals a{0, 0, 0}, c{0, 0, 0};
  for (int w = 0; w < kGenWarps; ++w) {
    a.child += s_all[w].child;
    a.x += s_all[w].x;
    a.y += s_all[w].y;
    c.child += s_pre[w].child;
    c.x += s_pre[w].x;
    c.y += s_pre[w].y;
  }
  *all = a;
  *pre = c;
  __syncthreads();
}

// Block-wide exclusive scan of packed counters; *total gets their sum.
template <typename U>
__device__ __forceinline__ U gen_block_scan(U v, U* total) {
  __shared__ U s_w[kGenWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  U incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const U w = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += w;
  }
  if (lane == 31) s_w[warp] = incl;
  __syncthreads();
  U before = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < kGenWarps; ++w) {
    const U x = s_w[w];
    if (w < warp) before += x;
    sum += x;
  }
  __syncthreads();
  *total = sum;
  return before + incl - v;
}

// CTAs of a cooperative launch of `kernel` on the current device (0: none).
template <typename Kernel>
inline int gen_grid(Kernel kernel) {
  int dev = 0, per_sm = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kGenThreads, 0) !=
          cudaSuccess)
    return 0;
  const int g = per_sm * sms;
  return g < kGenMaxBlocks ? g : kGenMaxBlocks;
}

}  // namespace
}  // namespace ygx
