// Per-node mass and multipole moments (yggdrax/tree_moments.py:686-877).
//
// The reference forms, for every particle, the mass-weighted monomials
// m x^a y^b z^c of all multi-indices up to the order (packed layout: level by
// level, multi_index_tuples order), takes their prefix sums over the
// Morton-sorted particles, differences them at each node's particle range,
// and shifts the raw sums to the node's expansion centre with the binomial
// stencil; the tensors (second ... fourth moments and their trace-free
// quadrupole / octupole / hexadecapole) follow per node.  Here:
//   k_tile_moments, k_col_tile_scan, k_prefix_moments: fp32 inclusive prefix
//                 per column (reduce, scan the tile sums, rescan), so the
//                 column sums are O(N) work,
//   k_node_moments 16 nodes per CTA: range differences, centre of mass, the
//                 shift to the expansion centre and the STF tensors.
// Arithmetic follows the reference's written fp32 order (cumprod powers,
// left-to-right monomial products, sequential sums over the stencil); the
// prefix sums are a parallel scan, so values agree with the reference to fp32
// rounding of the prefix sums, not bit for bit.
#include "common.cuh"

namespace ygx {

namespace {

constexpr int kMaxOrder = 4;
constexpr int kMaxCoef = 35;  // total_coefficients(4)
constexpr int kScanTileF = 2048;
constexpr int kScanThreads = 256;
constexpr int kScanPer = kScanTileF / kScanThreads;

// multi_index_tuples(level) for level 0..4, concatenated (multipole_utils.py);
// a lower order uses a prefix.
struct Exps {
  int a[kMaxCoef], b[kMaxCoef], c[kMaxCoef];
};
__host__ __device__ constexpr Exps make_exps() {
  Exps k{};
  int n = 0;
  for (int lv = 0; lv <= kMaxOrder; ++lv)
    for (int i = 0; i <= lv; ++i)
      for (int j = 0; j <= lv - i; ++j) {
        k.a[n] = i;
        k.b[n] = j;
        k.c[n] = lv - i - j;
        ++n;
      }
  return k;
}

// cumprod([1, v, v, v, v])[p]
__device__ __forceinline__ void powers(float v, float p[kMaxOrder + 1]) {
  p[0] = 1.0f;
#pragma unroll
  for (int k = 1; k <= kMaxOrder; ++k) p[k] = __fmul_rn(p[k - 1], v);
}
template <int P>
__device__ __forceinline__ float power(float v) {
  float r = 1.0f;
#pragma unroll
  for (int k = 0; k < P; ++k) r = __fmul_rn(r, v);
  return r;
}

// The prefix sums read the particles once per pass and keep no monomial in
// memory: a CTA takes 2048 particles and forms all columns from their
// positions in registers (first the tile sums, then, with the tiles' offsets,
// the prefixes).  With the monomials written as columns and read twice, 262,143
// particles at order 4 took 78 us in three kernels; these two take 31.
// The order of every sum is fixed: per thread, butterfly, then warp by warp.
template <int kCols>
__global__ void __launch_bounds__(kScanThreads)
    k_tile_moments(const float* __restrict__ pos, const float* __restrict__ mass, int64_t n,
                   int64_t tiles, float* __restrict__ tile_sums) {
  constexpr Exps E = make_exps();
  __shared__ float s_w[kCols][kScanThreads / 32];
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    float acc[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) acc[c] = 0.0f;
    for (int k = threadIdx.x; k < kScanTileF; k += kScanThreads) {
      const int64_t i = t * kScanTileF + k;
      if (i >= n) break;
      float px[kMaxOrder + 1], py[kMaxOrder + 1], pz[kMaxOrder + 1];
      powers(pos[3 * i], px);
      powers(pos[3 * i + 1], py);
      powers(pos[3 * i + 2], pz);
      const float m = mass[i];
#pragma unroll
      for (int c = 0; c < kCols; ++c)
        acc[c] = __fadd_rn(
            acc[c], __fmul_rn(m, __fmul_rn(__fmul_rn(px[E.a[c]], py[E.b[c]]), pz[E.c[c]])));
    }
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
      float v = acc[c];
      for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
      if ((threadIdx.x & 31) == 0) s_w[c][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < kCols) {
      float v = 0.0f;
      for (int w = 0; w < kScanThreads / 32; ++w) v = __fadd_rn(v, s_w[threadIdx.x][w]);
      tile_sums[(int64_t)threadIdx.x * tiles + t] = v;
    }
    __syncthreads();
  }
}

// Exclusive prefix of each column's tile sums (one CTA per column, serial
// over the tiles in chunks of the block).
__global__ void k_col_tile_scan(float* __restrict__ tile_sums, int64_t tiles) {
  const int c = blockIdx.x;
  float* ts = tile_sums + (int64_t)c * tiles;
  __shared__ float s[1024];
  float carry = 0.0f;
  for (int64_t b0 = 0; b0 < tiles; b0 += blockDim.x) {
    const int64_t k = b0 + threadIdx.x;
    const float v = k < tiles ? ts[k] : 0.0f;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < (int)blockDim.x; off <<= 1) {
      const float add = (int)threadIdx.x >= off ? s[threadIdx.x - off] : 0.0f;
      __syncthreads();
      s[threadIdx.x] = __fadd_rn(s[threadIdx.x], add);
      __syncthreads();
    }
    const float incl = s[threadIdx.x];
    if (k < tiles) ts[k] = __fadd_rn(carry, __fsub_rn(incl, v));  // exclusive
    __syncthreads();
    carry = __fadd_rn(carry, s[blockDim.x - 1]);
    __syncthreads();
  }
}

// prefix[c * stride + i] = inclusive prefix of column c at particle i (stride
// a multiple of 4, so a thread writes its 8 particles as two float4).
template <int kCols>
struct RescanSmem {
  float xyz[3 * kScanTileF], m[kScanTileF];
  float s[2][kCols][kScanThreads];
};
template <int kCols, int C>
__device__ __forceinline__ void rescan_column(const RescanSmem<kCols>& sm, int buf, int64_t tile,
                                              int64_t tiles, int64_t n, int64_t stride,
                                              const float* __restrict__ tile_off,
                                              float* __restrict__ prefix) {
  constexpr Exps E = make_exps();
  const int t0 = threadIdx.x * kScanPer;
  const float before =
      __fadd_rn(tile_off[(int64_t)C * tiles + tile],
                threadIdx.x > 0 ? sm.s[buf][C][threadIdx.x - 1] : 0.0f);
  float run = 0.0f, v[kScanPer];
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const float* p = sm.xyz + 3 * (t0 + k);
    const float mono =
        __fmul_rn(__fmul_rn(power<E.a[C]>(p[0]), power<E.b[C]>(p[1])), power<E.c[C]>(p[2]));
    run = __fadd_rn(run, __fmul_rn(sm.m[t0 + k], mono));
    v[k] = __fadd_rn(before, run);
  }
  const int64_t i = tile * kScanTileF + t0;
  float* out = prefix + (int64_t)C * stride + i;
#pragma unroll
  for (int h = 0; h < kScanPer; h += 4)
    if (i + h < stride)  // padding past n stays within the column
      *reinterpret_cast<float4*>(out + h) = make_float4(v[h], v[h + 1], v[h + 2], v[h + 3]);
  if constexpr (C + 1 < kCols)
    rescan_column<kCols, C + 1>(sm, buf, tile, tiles, n, stride, tile_off, prefix);
}
template <int kCols>
__global__ void __launch_bounds__(kScanThreads)
    k_prefix_moments(const float* __restrict__ pos, const float* __restrict__ mass, int64_t n,
                     int64_t tiles, int64_t stride, const float* __restrict__ tile_off,
                     float* __restrict__ prefix) {
  constexpr Exps E = make_exps();
  extern __shared__ __align__(16) unsigned char rescan_raw[];
  RescanSmem<kCols>& sm = *reinterpret_cast<RescanSmem<kCols>*>(rescan_raw);
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t base = t * kScanTileF;
    const int cnt = n - base < kScanTileF ? (int)(n - base) : kScanTileF;
    // a particle past the end has mass 0 at the origin
    for (int k = threadIdx.x; k < 3 * kScanTileF; k += kScanThreads)
      sm.xyz[k] = k < 3 * cnt ? pos[3 * base + k] : 0.0f;
    for (int k = threadIdx.x; k < kScanTileF; k += kScanThreads)
      sm.m[k] = k < cnt ? mass[base + k] : 0.0f;
    __syncthreads();
    {
      float run[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) run[c] = 0.0f;
      for (int k = 0; k < kScanPer; ++k) {
        const int i = threadIdx.x * kScanPer + k;
        float px[kMaxOrder + 1], py[kMaxOrder + 1], pz[kMaxOrder + 1];
        powers(sm.xyz[3 * i], px);
        powers(sm.xyz[3 * i + 1], py);
        powers(sm.xyz[3 * i + 2], pz);
        const float m = sm.m[i];
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          run[c] = __fadd_rn(
              run[c], __fmul_rn(m, __fmul_rn(__fmul_rn(px[E.a[c]], py[E.b[c]]), pz[E.c[c]])));
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) sm.s[0][c][threadIdx.x] = run[c];
    }
    __syncthreads();
    // inclusive scan of the threads' sums, all columns between two barriers
    int buf = 0;
    for (int off = 1; off < kScanThreads; off <<= 1) {
      const bool add = (int)threadIdx.x >= off;
#pragma unroll 5
      for (int c = 0; c < kCols; ++c)
        sm.s[buf ^ 1][c][threadIdx.x] = __fadd_rn(
            sm.s[buf][c][threadIdx.x], add ? sm.s[buf][c][threadIdx.x - off] : 0.0f);
      buf ^= 1;
      __syncthreads();
    }
    rescan_column<kCols, 0>(sm, buf, t, tiles, n, stride, tile_off, prefix);
    __syncthreads();
  }
}

template <int kCols>
int prefix_moments(const float* pos, const float* mass, int64_t n, int64_t tiles, int64_t stride,
                   float* tsum, float* prefix, cudaStream_t stream) {
  k_tile_moments<kCols><<<grid_for(tiles, 1), kScanThreads, 0, stream>>>(pos, mass, n, tiles, tsum);
  YGX_CHECK_LAUNCH();
  k_col_tile_scan<<<kCols, 1024, 0, stream>>>(tsum, tiles);
  YGX_CHECK_LAUNCH();
  static std::atomic<uint64_t> attr{0};
  const int smem = (int)sizeof(RescanSmem<kCols>);
  if (ensure_smem_limit(k_prefix_moments<kCols>, smem, attr) != cudaSuccess) return YGX_ERR_CUDA;
  k_prefix_moments<kCols><<<grid_for(tiles, 1), kScanThreads, smem, stream>>>(
      pos, mass, n, tiles, stride, tsum, prefix);
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

// Fixed tables of the packed layout (orders 0..4; a lower order is a prefix):
// the packed index of every tensor element, and per coefficient alpha the
// terms beta <= alpha of the shift stencil, beta ascending:
// beta | gamma_x << 6 | gamma_y << 9 | gamma_z << 12 | binomial << 16.
constexpr int kMaxTerms = 256;
struct Tables {
  unsigned char i2[9], i3[27], i4[81];
  unsigned short start[kMaxCoef + 1];
  unsigned int term[kMaxTerms];
};
constexpr int ccomb(int n, int k) {
  int r = 1;
  for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
  return r;
}
constexpr Tables make_tables() {
  Tables t{};
  int A[kMaxCoef] = {}, B[kMaxCoef] = {}, D[kMaxCoef] = {};
  int n = 0;
  for (int lv = 0; lv <= kMaxOrder; ++lv)
    for (int i = 0; i <= lv; ++i)
      for (int j = 0; j <= lv - i; ++j) {
        A[n] = i;
        B[n] = j;
        D[n] = lv - i - j;
        ++n;
      }
  for (int rank = 2; rank <= 4; ++rank) {
    const int size = rank == 2 ? 9 : rank == 3 ? 27 : 81;
    for (int at = 0; at < size; ++at) {
      int cnt[3] = {0, 0, 0}, r = at;
      for (int k = 0; k < rank; ++k) {
        ++cnt[r % 3];
        r /= 3;
      }
      int found = 0;
      for (int c = 0; c < kMaxCoef; ++c)
        if (A[c] == cnt[0] && B[c] == cnt[1] && D[c] == cnt[2]) found = c;
      (rank == 2 ? t.i2[at] : rank == 3 ? t.i3[at] : t.i4[at]) = (unsigned char)found;
    }
  }
  int m = 0;
  for (int i = 0; i < kMaxCoef; ++i) {
    t.start[i] = (unsigned short)m;
    for (int j = 0; j < kMaxCoef; ++j)
      if (A[i] >= A[j] && B[i] >= B[j] && D[i] >= D[j])
        t.term[m++] = (unsigned)(j | (A[i] - A[j]) << 6 | (B[i] - B[j]) << 9 |
                                 (D[i] - D[j]) << 12 |
                                 ccomb(A[i], A[j]) * ccomb(B[i], B[j]) * ccomb(D[i], D[j]) << 16);
  }
  t.start[kMaxCoef] = (unsigned short)m;
  return t;
}
__device__ const Tables kTables = make_tables();

// Raw range sums, mass / centre of mass, the binomial shift to the expansion
// centre (centre of mass, or `centers` when given), and the tensors.  Outputs
// (per node): mass, com (3), center (3), packed (C), dipole (3), second (9),
// quad (9), third (27), oct (27), fourth (81), hexa (81).
//
// A node has up to 300 outputs from 70 prefix values, so the work is spread
// over (node, coefficient) and (node, output) pairs: a CTA takes kMomNodes
// nodes, keeps their sums and coefficients in shared memory, and writes every
// output array as one contiguous run.  One thread per node (its 35 sums in
// local memory, the full 35 x 35 stencil read from memory, outputs 324 bytes
// apart in a warp) was latency bound: 321 us for the 16,383 nodes of a
// 262,143-particle tree against 27 us here.
constexpr int kMomNodes = 16;
constexpr int kMomThreads = 256;
constexpr int kMomPad = kMaxCoef + 1;

template <typename F>
__device__ __forceinline__ void mom_outputs(int cnt, int size, F f) {
  for (int x = threadIdx.x; x < cnt * size; x += kMomThreads) f(x, x / size, x % size);
}

__global__ void __launch_bounds__(kMomThreads)
    k_node_moments(const float* __restrict__ prefix, int64_t stride, const void* ranges,
                   int index_bits, int64_t nodes, int order, int C, int Ccols,
                   const float* __restrict__ centers, float* __restrict__ o_mass,
                   float* __restrict__ o_com, float* __restrict__ o_center,
                   float* __restrict__ o_packed, float* __restrict__ o_dipole,
                   float* __restrict__ o_second, float* __restrict__ o_quad,
                   float* __restrict__ o_third, float* __restrict__ o_oct,
                   float* __restrict__ o_fourth, float* __restrict__ o_hexa) {
  __shared__ Tables tb;
  __shared__ float raw[kMomNodes][kMomPad], pk[kMomNodes][kMomPad];
  __shared__ float pw[kMomNodes][3][kMaxOrder + 1];
  __shared__ float trace[kMomNodes], r2rk[kMomNodes][3], r2[kMomNodes][9], r4[kMomNodes];
  __shared__ int odd[kMomNodes];   // a sum is infinite or NaN
  __shared__ int64_t rng[kMomNodes][2];
  for (int k = threadIdx.x; k < (int)(sizeof(Tables) / 4); k += kMomThreads)
    reinterpret_cast<unsigned*>(&tb)[k] = reinterpret_cast<const unsigned*>(&kTables)[k];
  for (int64_t q0 = (int64_t)blockIdx.x * kMomNodes; q0 < nodes;
       q0 += (int64_t)gridDim.x * kMomNodes) {
    const int cnt = nodes - q0 < kMomNodes ? (int)(nodes - q0) : kMomNodes;
    __syncthreads();  // the previous tile's outputs are written (and tb is there)
    if (threadIdx.x < 2 * kMomNodes && (int)(threadIdx.x >> 1) < cnt)
      rng[threadIdx.x >> 1][threadIdx.x & 1] =
          load_idx(ranges, index_bits, 2 * q0 + threadIdx.x) - 1 + (threadIdx.x & 1);
    if (threadIdx.x < kMomNodes) odd[threadIdx.x] = 0;
    __syncthreads();
    for (int x = threadIdx.x; x < cnt * Ccols; x += kMomThreads) {
      const int v = x % cnt, c = x / cnt;
      const float* col = prefix + (int64_t)c * stride;
      // inclusive prefixes at the last particle and before the first one
      const float hi = rng[v][1] >= 0 ? col[rng[v][1]] : 0.0f;
      const float lo = rng[v][0] >= 0 ? col[rng[v][0]] : 0.0f;
      const float r = __fsub_rn(hi, lo);
      raw[v][c] = r;
      if (!(fabsf(r) <= 3.402823466e38f)) odd[v] = 1;
    }
    __syncthreads();
    // compute_tree_mass_moments: mass, centre of mass (0 for massless nodes);
    // the weighted-position columns are the level-1 combos (1,0,0), (0,1,0),
    // (0,0,1) = packed indices 3, 2, 1
    for (int x = threadIdx.x; x < cnt * 3; x += kMomThreads) {
      const int v = x / 3, ax = x % 3;
      const float m = raw[v][0];
      const float cm =
          (Ccols < 4 || m == 0.0f) ? 0.0f : __fdiv_rn(raw[v][3 - ax], m == 0.0f ? 1.0f : m);
      if (o_com) o_com[3 * q0 + x] = cm;
      if (ax == 0) o_mass[q0 + v] = m;
      if (o_packed) {
        const float ct = centers ? centers[3 * q0 + x] : cm;
        o_center[3 * q0 + x] = ct;
        powers(-ct, pw[v][ax]);
      }
    }
    if (!o_packed) continue;
    __syncthreads();
    // the shift: sum over beta ascending of (centre factor * binomial) *
    // raw[beta].  Terms outside the stencil are 0 * raw: left out, except
    // where a sum is infinite or NaN and they count.
    for (int x = threadIdx.x; x < cnt * C; x += kMomThreads) {
      const int v = x / C, i = x % C;
      const int t1 = tb.start[i + 1];
      int t = tb.start[i];
      float acc = 0.0f;
      if (!odd[v]) {
        for (; t < t1; ++t) {
          const unsigned w = tb.term[t];
          const float cf = __fmul_rn(__fmul_rn(pw[v][0][(w >> 6) & 7u], pw[v][1][(w >> 9) & 7u]),
                                     pw[v][2][(w >> 12) & 7u]);
          acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(cf, (float)(w >> 16)), raw[v][w & 63u]));
        }
      } else {
        for (int j = 0; j < C; ++j) {
          float tr = 0.0f;
          if (t < t1 && (int)(tb.term[t] & 63u) == j) {
            const unsigned w = tb.term[t++];
            tr = __fmul_rn(__fmul_rn(__fmul_rn(pw[v][0][(w >> 6) & 7u], pw[v][1][(w >> 9) & 7u]),
                                     pw[v][2][(w >> 12) & 7u]),
                           (float)(w >> 16));
          }
          acc = __fadd_rn(acc, __fmul_rn(tr, raw[v][j]));
        }
      }
      pk[v][i] = acc;
      o_packed[q0 * C + x] = acc;
    }
    __syncthreads();
    // contractions of the trace-free tensors (_moments_from_raw_packed, :312-395)
    auto sec = [&](int v, int at) { return order >= 2 ? pk[v][tb.i2[at]] : 0.0f; };
    auto thr = [&](int v, int at) { return order >= 3 ? pk[v][tb.i3[at]] : 0.0f; };
    auto fou = [&](int v, int at) { return order >= 4 ? pk[v][tb.i4[at]] : 0.0f; };
    mom_outputs(cnt, 9, [&](int, int v, int kl) {
      r2[v][kl] = __fadd_rn(__fadd_rn(fou(v, kl), fou(v, 36 + kl)), fou(v, 72 + kl));
      if (kl < 3)
        r2rk[v][kl] = __fadd_rn(__fadd_rn(thr(v, kl), thr(v, 12 + kl)), thr(v, 24 + kl));
      if (kl == 3) trace[v] = __fadd_rn(__fadd_rn(sec(v, 0), sec(v, 4)), sec(v, 8));
      if (kl == 4)
        r4[v] = __fadd_rn(
            __fadd_rn(__fadd_rn(fou(v, 0), fou(v, 40)), fou(v, 80)),
            __fmul_rn(2.0f, __fadd_rn(__fadd_rn(fou(v, 4), fou(v, 8)), fou(v, 44))));
    });
    __syncthreads();
    auto massless = [&](int v) { return pk[v][0] == 0.0f; };
    mom_outputs(cnt, 3, [&](int x, int v, int ax) {
      o_dipole[3 * q0 + x] = massless(v) || order < 1 ? 0.0f : pk[v][3 - ax];
    });
    // quadrupole = 3 S - tr(S) I
    mom_outputs(cnt, 9, [&](int x, int v, int at) {
      const float sv = sec(v, at);
      const float w = __fsub_rn(__fmul_rn(3.0f, sv), at % 4 == 0 ? trace[v] : 0.0f);
      o_second[9 * q0 + x] = massless(v) ? 0.0f : sv;
      o_quad[9 * q0 + x] = massless(v) ? 0.0f : w;
    });
    // octupole (:233-256)
    mom_outputs(cnt, 27, [&](int x, int v, int at) {
      const int i = at / 9, j = at / 3 % 3, k = at % 3;
      const float tv = thr(v, at);
      float w = 0.0f;
      if (order >= 3) {
        w = __fmul_rn(5.0f, tv);
        if (i == j) w = __fsub_rn(w, r2rk[v][k]);
        if (i == k) w = __fsub_rn(w, r2rk[v][j]);
        if (j == k) w = __fsub_rn(w, r2rk[v][i]);
      }
      o_third[27 * q0 + x] = massless(v) ? 0.0f : tv;
      o_oct[27 * q0 + x] = massless(v) ? 0.0f : w;
    });
    // hexadecapole (:258-298)
    mom_outputs(cnt, 81, [&](int x, int v, int at) {
      const int i = at / 27, j = at / 9 % 3, k = at / 3 % 3, l = at % 3;
      const float fv = fou(v, at);
      float w = 0.0f;
      if (order >= 4) {
        w = __fmul_rn(35.0f, fv);
        float term = 0.0f;
        if (i == j) term = __fadd_rn(term, r2[v][3 * k + l]);
        if (i == k) term = __fadd_rn(term, r2[v][3 * j + l]);
        if (i == l) term = __fadd_rn(term, r2[v][3 * j + k]);
        if (j == k) term = __fadd_rn(term, r2[v][3 * i + l]);
        if (j == l) term = __fadd_rn(term, r2[v][3 * i + k]);
        if (k == l) term = __fadd_rn(term, r2[v][3 * i + j]);
        w = __fsub_rn(w, __fmul_rn(5.0f, term));
        const int df = (i == j && k == l) + (i == k && j == l) + (i == l && j == k);
        if (df) w = __fadd_rn(w, __fmul_rn(r4[v], (float)df));
      }
      o_fourth[81 * q0 + x] = massless(v) ? 0.0f : fv;
      o_hexa[81 * q0 + x] = massless(v) ? 0.0f : w;
    });
  }
}

}  // namespace

}  // namespace ygx

extern "C" {

size_t ygx_moments_workspace_size(int64_t n, int max_order) {
  if (max_order < 0 || max_order > ygx::kMaxOrder || n < 1) return 0;
  const int oc = max_order < 1 ? 1 : max_order;  // the centre of mass needs order 1
  const int C = (oc + 1) * (oc + 2) * (oc + 3) / 6;
  const int64_t tiles = (n + ygx::kScanTileF - 1) / ygx::kScanTileF;
  ygx::Arena a{nullptr, 0, 0};
  a.take<float>((size_t)C * ((n + 3) / 4 * 4));
  a.take<float>((size_t)C * tiles);
  return a.used + 256;
}

// Mass moments (compute_tree_mass_moments, tree_moments.py:686-744) when
// o_packed is null; otherwise also the multipole moments about `centers`
// (null: the centres of mass) through max_order (compute_tree_multipole_moments,
// :747-877).  ranges: the topology's node_ranges (nodes x 2, inclusive) in the
// index dtype.  Does not synchronize.
int ygx_tree_moments(const float* positions_sorted, const float* masses_sorted, int64_t n,
                     const void* node_ranges, int index_bits, int64_t nodes, int max_order,
                     const float* centers, float* o_mass, float* o_com, float* o_center,
                     float* o_packed, float* o_dipole, float* o_second, float* o_quad,
                     float* o_third, float* o_oct, float* o_fourth, float* o_hexa, void* ws,
                     size_t ws_bytes, cudaStream_t stream) {
  if (n < 1 || nodes < 1 || max_order < 0 || max_order > ygx::kMaxOrder || !positions_sorted ||
      !masses_sorted || !node_ranges || !o_mass || (index_bits != 32 && index_bits != 64))
    return YGX_ERR_ARG;
  if (o_packed && (!o_center || !o_dipole || !o_second || !o_quad || !o_third || !o_oct ||
                   !o_fourth || !o_hexa))
    return YGX_ERR_ARG;
  if (ws_bytes < ygx_moments_workspace_size(n, max_order)) return YGX_ERR_ARG;
  // columns through order max(max_order, 1): the centre of mass needs the
  // weighted positions; the packed output holds C coefficients
  const int order = o_packed ? max_order : 0;
  const int oc = max_order < 1 ? 1 : max_order;
  const int Ccols = (oc + 1) * (oc + 2) * (oc + 3) / 6;
  const int C = (order + 1) * (order + 2) * (order + 3) / 6;
  const int64_t tiles = (n + ygx::kScanTileF - 1) / ygx::kScanTileF;
  ygx::Arena a{(char*)ws, 0, ws_bytes};
  const int64_t stride = (n + 3) / 4 * 4;
  float* prefix = a.take<float>((size_t)Ccols * stride);
  float* tsum = a.take<float>((size_t)Ccols * tiles);
  int rc;
  switch (Ccols) {
    case 4:
      rc = ygx::prefix_moments<4>(positions_sorted, masses_sorted, n, tiles, stride, tsum, prefix,
                                  stream);
      break;
    case 10:
      rc = ygx::prefix_moments<10>(positions_sorted, masses_sorted, n, tiles, stride, tsum, prefix,
                                  stream);
      break;
    case 20:
      rc = ygx::prefix_moments<20>(positions_sorted, masses_sorted, n, tiles, stride, tsum, prefix,
                                  stream);
      break;
    default:
      rc = ygx::prefix_moments<35>(positions_sorted, masses_sorted, n, tiles, stride, tsum, prefix,
                                   stream);
      break;
  }
  if (rc) return rc;
  ygx::k_node_moments<<<ygx::grid_for(nodes, ygx::kMomNodes), ygx::kMomThreads, 0, stream>>>(
      prefix, stride, node_ranges, index_bits, nodes, order, C, Ccols, centers, o_mass, o_com,
      o_center, o_packed, o_dipole, o_second, o_quad, o_third, o_oct, o_fourth, o_hexa);
  YGX_CHECK_LAUNCH();
  return YGX_OK;
}

}  // extern "C"
