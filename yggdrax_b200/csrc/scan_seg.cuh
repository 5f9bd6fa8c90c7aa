// Several exclusive scans in one go, each writing its results where they are
// used: a functor F says, for scan s, its length n(s), its i-th value
// get(s, i), what becomes of prefix p before item i (put(s, i, p, v)) and of
// the total (end(s, total)).
//
// Lists and slots are planned from a handful of counters per tree, so what a
// scan costs is its launches.  Four scans with their gathers and tables took
// 19; here they take three, and one when every scan has at most kSegDirect
// tiles -- each CTA then sums the tiles before its own itself instead of
// waiting for anybody.  With the walk's five host reads made one, a step of
// 4,000 particles went from 1,070 to 912 us, of 1,000,003 from 2,313 to 2,197.
#pragma once
#include "scan.cuh"

namespace ygx {
namespace {

constexpr int kSegDirect = 16;  // tiles: 65,536 values, re-read at most 15 times from L2

__device__ __forceinline__ int64_t seg_block_sum(int64_t v, int64_t* s_warp) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
  __syncthreads();
  int64_t t = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_warp[w];
  __syncthreads();
  return t;
}

// tmp: per scan, (tiles of the longest scan) sums.
template <typename F>
__global__ void __launch_bounds__(kScanThreads)
    k_seg_sums(const F f, int64_t stride, int64_t* __restrict__ tmp) {
  __shared__ int64_t s_warp[kScanThreads / 32];
  const int s = blockIdx.y;
  const int64_t n = f.n(s), base = (int64_t)blockIdx.x * kScanTile;
  int64_t acc = 0;
  for (int k = threadIdx.x; k < kScanTile; k += kScanThreads)
    if (base + k < n) acc += f.get(s, base + k);
  acc = seg_block_sum(acc, s_warp);
  if (threadIdx.x == 0) tmp[s * stride + blockIdx.x] = acc;
}

__global__ void __launch_bounds__(1024)
    k_seg_mid(int64_t* __restrict__ tmp, int64_t stride) {
  __shared__ int64_t s_w[32];
  int64_t* t = tmp + blockIdx.x * stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t carry = 0;
  for (int64_t b = 0; b < stride; b += 1024) {
    const int64_t i = b + threadIdx.x;
    const int64_t v = i < stride ? t[i] : 0;
    int64_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t w = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += w;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    int64_t before = carry, sum = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += s_w[w];
      sum += s_w[w];
    }
    if (i < stride) t[i] = before + incl - v;
    carry += sum;
    __syncthreads();
  }
}

template <typename F>
__global__ void __launch_bounds__(kScanThreads)
    k_seg_write(const F f, int64_t stride, const int64_t* __restrict__ tmp) {
  __shared__ int64_t s_warp[kScanThreads / 32];
  const int s = blockIdx.y;
  const int64_t n = f.n(s), base = (int64_t)blockIdx.x * kScanTile;
  if (base >= n && !(n == 0 && blockIdx.x == 0)) return;
  int64_t before;
  if (tmp) {
    before = tmp[s * stride + blockIdx.x];
  } else {
    int64_t acc = 0;
    for (int64_t i = threadIdx.x; i < base; i += kScanThreads) acc += f.get(s, i);
    before = seg_block_sum(acc, s_warp);
  }
  // rounds of one item per thread: coalesced reads and writes
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
    const int64_t v = i < n ? f.get(s, i) : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t w = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += w;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int64_t p = before, sum = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
      const int64_t x = s_warp[w];
      if (w < warp) p += x;
      sum += x;
    }
    __syncthreads();
    p += incl - v;
    if (i < n) f.put(s, i, p, v);
    if (i == n - 1 || (n == 0 && i == 0)) f.end(s, p + v);
    before += sum;
    if (base + (int64_t)(k + 1) * kScanThreads >= n) break;
  }
}

// Runs `scans` (at most 65535) scans of at most n_max values each; tmp:
// seg_scan_elems(n_max, scans) int64s.
inline size_t seg_scan_elems(int64_t n_max, int scans) {
  const int64_t t = scan_tiles(n_max > 0 ? n_max : 1);
  return (size_t)(t * scans);
}
template <typename F>
int seg_scan(const F& f, int64_t n_max, int scans, int64_t* tmp, cudaStream_t st) {
  const int64_t tiles = scan_tiles(n_max > 0 ? n_max : 1);
  const dim3 grid((unsigned)tiles, (unsigned)scans);
  if (tiles > kSegDirect) {
    k_seg_sums<F><<<grid, kScanThreads, 0, st>>>(f, tiles, tmp);
    YGX_CHECK_LAUNCH();
    k_seg_mid<<<scans, 1024, 0, st>>>(tmp, tiles);
    YGX_CHECK_LAUNCH();
  }
  k_seg_write<F><<<grid, kScanThreads, 0, st>>>(f, tiles, tiles > kSegDirect ? tmp : nullptr);
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

}  // namespace
}  // namespace ygx
