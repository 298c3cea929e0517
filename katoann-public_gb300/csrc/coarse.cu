// Exact SQ16 distance tiles (the reference's sq16_l2 / sq16_high_l2) and the
// coarse top-nprobe selection.
//
// A 16-bit code is h * 256 + l, so q.x = 65536 (qh.xh) + 256 (qh.xl + ql.xh)
// + ql.xl (include/katoann/kernels.h:163-170). Each of the three byte sums is
// accumulated in an exact 32-bit integer with packed 4-byte dot products
// (each sum is at most 2 * 4096 * 255^2 < 2^32), combined in 64 bits, and the
// squared L2 qn + xn - 2 q.x is mapped to the reference's float value by
// dist_value() (src/kernels.cpp:203-210).
#include "kcommon.cuh"

namespace kato {

namespace {

constexpr int kTile = 64;     // queries x database rows per CTA
constexpr int kKw = 16;       // 32-bit words (64 bytes) of each row per k-step
constexpr int kSw = kKw + 1;  // padded words per staged row

template <bool kFull>
__global__ void __launch_bounds__(256) sq16_tile_kernel(
    const uint8_t *qhi, const uint8_t *qlo, const uint8_t *__restrict__ xhi,
    const uint8_t *__restrict__ xlo, const int64_t *qn, const int64_t *__restrict__ xn,
    DistScale scale, uint32_t m, uint32_t n, uint32_t dims, uint32_t qstride, uint32_t xstride,
    float *out) {
  after_previous();
  __shared__ uint32_t sqh[kTile * kSw], sxh[kTile * kSw];
  __shared__ uint32_t sql[kFull ? kTile * kSw : 1], sxl[kFull ? kTile * kSw : 1];
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const uint32_t m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
  uint32_t hh[4][4], mx[4][4], ll[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) hh[a][b] = mx[a][b] = ll[a][b] = 0;

  // Staging: 64 rows x 64 bytes per array = 256 16-byte loads, one per thread.
  const int lr = t >> 2, lw = (t & 3) * 4;
  for (uint32_t k0 = 0; k0 < dims; k0 += kKw * 4) {
    {
      const uint32_t qi = m0 + lr, xi = n0 + lr;
      uint4 vqh = make_uint4(0, 0, 0, 0), vql = vqh, vxh = vqh, vxl = vqh;
      if (qi < m) {
        vqh = *reinterpret_cast<const uint4 *>(qhi + static_cast<size_t>(qi) * qstride + k0 + lw * 4);
        if (kFull) vql = *reinterpret_cast<const uint4 *>(qlo + static_cast<size_t>(qi) * qstride + k0 + lw * 4);
      }
      if (xi < n) {
        vxh = *reinterpret_cast<const uint4 *>(xhi + static_cast<size_t>(xi) * xstride + k0 + lw * 4);
        if (kFull) vxl = *reinterpret_cast<const uint4 *>(xlo + static_cast<size_t>(xi) * xstride + k0 + lw * 4);
      }
      uint32_t *dq = sqh + lr * kSw + lw, *dx = sxh + lr * kSw + lw;
      dq[0] = vqh.x; dq[1] = vqh.y; dq[2] = vqh.z; dq[3] = vqh.w;
      dx[0] = vxh.x; dx[1] = vxh.y; dx[2] = vxh.z; dx[3] = vxh.w;
      if (kFull) {
        uint32_t *eq = sql + lr * kSw + lw, *ex = sxl + lr * kSw + lw;
        eq[0] = vql.x; eq[1] = vql.y; eq[2] = vql.z; eq[3] = vql.w;
        ex[0] = vxl.x; ex[1] = vxl.y; ex[2] = vxl.z; ex[3] = vxl.w;
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int w = 0; w < kKw; ++w) {
      uint32_t a_h[4], a_l[4], b_h[4], b_l[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        a_h[a] = sqh[(ty + 16 * a) * kSw + w];
        if (kFull) a_l[a] = sql[(ty + 16 * a) * kSw + w];
      }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        b_h[b] = sxh[(tx + 16 * b) * kSw + w];
        if (kFull) b_l[b] = sxl[(tx + 16 * b) * kSw + w];
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          hh[a][b] = dp4(a_h[a], b_h[b], hh[a][b]);
          if (kFull) {
            mx[a][b] = dp4(a_h[a], b_l[b], mx[a][b]);
            mx[a][b] = dp4(a_l[a], b_h[b], mx[a][b]);
            ll[a][b] = dp4(a_l[a], b_l[b], ll[a][b]);
          }
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const uint32_t qi = m0 + ty + 16 * a;
    if (qi >= m) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const uint32_t xi = n0 + tx + 16 * b;
      if (xi >= n) continue;
      const int64_t dot = kFull ? static_cast<int64_t>((static_cast<uint64_t>(hh[a][b]) << 16) +
                                                       (static_cast<uint64_t>(mx[a][b]) << 8) +
                                                       ll[a][b])
                                : static_cast<int64_t>(hh[a][b]);
      out[static_cast<size_t>(qi) * n + xi] = dist_value(qn[qi] + xn[xi] - 2 * dot, scale);
    }
  }
}

// Smallest `p` of a row of `n` float distances (all >= 0, so their bit
// patterns order like the values) by (distance, list id), ascending.
// One CTA per query: radix selection of the p-th distance over 8-bit digits,
// then, among lists tied at that distance, of the smallest ids; the p chosen
// are then sorted (bitonic, in shared memory) when p <= kSortMax.
constexpr int kSelThreads = 256;
constexpr int kSortMax = 4096;

__device__ __forceinline__ uint32_t block_scan_bins(uint32_t *hist, uint32_t rank, uint32_t *sh_sel,
                                                    uint32_t *sh_below) {
  // Serial over 256 bins by warp 0 with a warp prefix sum.
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    uint32_t carry = 0;
    for (int base = 0; base < 256; base += 32) {
      const uint32_t v = hist[base + lane];
      uint32_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t excl = carry + incl - v;
      // the bin holding the rank-th element (0-based)
      const bool hit = excl <= rank && rank < excl + v;
      const uint32_t mask = __ballot_sync(0xffffffffu, hit);
      if (mask) {
        const int src = __ffs(mask) - 1;
        const uint32_t e = __shfl_sync(0xffffffffu, excl, src);
        if (lane == 0) {
          *sh_sel = base + src;
          *sh_below = e;
        }
        break;
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncthreads();
  return *sh_sel;
}

// Smallest p keys of a row by (key, index) in up to six passes over the row
// (8-bit radix digits of the p-th key, then of the tied indices, then the
// gather). sel holds np2(p) 64-bit words, hist 256 counters, scal 4 words.
__device__ void select_passes(const uint32_t *keys, uint32_t n, uint32_t p, uint32_t *outp,
                              uint32_t *cnt, unsigned long long *tie_count, unsigned long long *sel,
                              uint32_t *hist, uint32_t *scal) {
  const uint32_t tid = threadIdx.x;
  // 1) the p-th smallest key (rank p-1), and how many keys are below it.
  uint32_t prefix = 0, rank = p - 1, below = 0;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (uint32_t i = tid; i < 256; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const uint32_t hmask = shift == 24 ? 0u : (0xFFFFFFFFu << (shift + 8));
    for (uint32_t i = tid; i < n; i += blockDim.x) {
      const uint32_t k = keys[i];
      if ((k & hmask) == prefix) atomicAdd(&hist[(k >> shift) & 0xFFu], 1u);
    }
    __syncthreads();
    const uint32_t bin = block_scan_bins(hist, rank, scal, scal + 1);
    rank -= scal[1];
    below += scal[1];
    prefix |= bin << shift;
    __syncthreads();
  }
  const uint32_t T = prefix;        // the p-th smallest key
  const uint32_t need = rank + 1;   // ids to take among keys == T
  // 2) among keys == T, the need-th smallest list id (only when ties exceed need).
  if (tid == 0) scal[3] = 0;
  __syncthreads();
  for (uint32_t i = tid; i < n; i += blockDim.x)
    if (keys[i] == T) atomicAdd(&scal[3], 1u);
  __syncthreads();
  const uint32_t neq = scal[3];
  uint32_t idmax = 0xFFFFFFFFu;
  if (neq > need) {
    if (tid == 0 && tie_count) atomicAdd(tie_count, 1ull);
    uint32_t ip = 0, ir = need - 1;
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (uint32_t i = tid; i < 256; i += blockDim.x) hist[i] = 0;
      __syncthreads();
      const uint32_t hmask = shift == 24 ? 0u : (0xFFFFFFFFu << (shift + 8));
      for (uint32_t i = tid; i < n; i += blockDim.x)
        if (keys[i] == T && (i & hmask) == ip) atomicAdd(&hist[(i >> shift) & 0xFFu], 1u);
      __syncthreads();
      const uint32_t bin = block_scan_bins(hist, ir, scal, scal + 1);
      ir -= scal[1];
      ip |= bin << shift;
      __syncthreads();
    }
    idmax = ip;
  }
  // 3) gather the p selected.
  if (tid == 0) scal[2] = 0;
  __syncthreads();
  const bool sorted = p <= kSortMax;
  for (uint32_t i = tid; i < n; i += blockDim.x) {
    const uint32_t k = keys[i];
    if (k < T || (k == T && i <= idmax)) {
      const uint32_t pos = atomicAdd(&scal[2], 1u);
      if (cnt) atomicAdd(&cnt[i], 1u);
      if (sorted) sel[pos] = (static_cast<unsigned long long>(k) << 32) | i;
      else outp[pos] = i;
    }
  }
  __syncthreads();
  if (!sorted) return;
  // 4) bitonic sort of the p selected, padded to a power of two.
  uint32_t np2 = 1;
  while (np2 < p) np2 <<= 1;
  for (uint32_t i = p + tid; i < np2; i += blockDim.x) sel[i] = ~0ull;
  __syncthreads();
  for (uint32_t size = 2; size <= np2; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = tid; i < np2; i += blockDim.x) {
        const uint32_t j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const unsigned long long a = sel[i], b = sel[j];
          if ((a > b) == up) {
            sel[i] = b;
            sel[j] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = tid; i < p; i += blockDim.x) outp[i] = static_cast<uint32_t>(sel[i] & 0xFFFFFFFFu);
}

// Rows are written `stride` apart. With `cnt`, each selected list's counter
// there is incremented (the inversion's counts). With `only`, rows whose only[q] is at
// most only_above are skipped (a second, deeper selection for the queries
// that need it).
__global__ void __launch_bounds__(kSelThreads) select_topp_kernel(
    const float *dists, uint32_t n, uint32_t p, uint32_t stride, uint32_t *probed, uint32_t *cnt,
    unsigned long long *tie_count, const uint32_t *only, uint32_t only_above) {
  after_previous();
  extern __shared__ unsigned long long sel[];  // up to kSortMax (key << 32 | id)
  __shared__ uint32_t hist[256], scal[4];
  const uint32_t q = blockIdx.x;
  if (only && only[q] <= only_above) return;
  select_passes(reinterpret_cast<const uint32_t *>(dists) + static_cast<size_t>(q) * n, n, p,
                probed + static_cast<size_t>(q) * stride, cnt, tie_count, sel, hist, scal);
}

// In-shared-memory bitonic sort of n 64-bit keys, ascending.
__device__ void sort_keys(unsigned long long *key, uint32_t n) {
  uint32_t np2 = 1;
  while (np2 < n) np2 <<= 1;
  for (uint32_t i = n + threadIdx.x; i < np2; i += blockDim.x) key[i] = ~0ull;
  __syncthreads();
  for (uint32_t size = 2; size <= np2; size <<= 1)
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x) {
        const uint32_t j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const unsigned long long a = key[i], b = key[j];
          if ((a > b) == up) {
            key[i] = b;
            key[j] = a;
          }
        }
      }
      __syncthreads();
    }
}

// Smallest p of a row of n non-negative float distances by (distance, list),
// ascending, for p <= kSortMax, in one pass over the row: it stays in registers
// (V 16-byte loads per thread; V = 0: longer rows are read again).
//
//   1. The p-th smallest of the minima of disjoint groups of keys bounds the p-th
//      smallest key from above, and closely: p of G minima leave about
//      -G ln(1 - p / G) keys at or below it (84 for p = 72, G = 512). A group
//      is what a thread holds (level 0), four neighbours (1) or one key (2).
//   2. A histogram over the range of the minima finds the p-th to 1/1024 of
//      that range, from above.
//   3. Every key up to it is gathered. A few are ranked by counting the smaller
//      ones of each; more by a histogram of their own range, whose prefix sums
//      leave a handful of keys to compare in each bin. (Counting c keys reads
//      shared memory c^2 / 32 times: 460 keys of 5,000 took 184 us for 2000 rows, 39
//      with the bins.)
//
// More than `cap` gathered keys (many equal distances) fall back to
// select_passes, crowded bins to a bitonic sort. The rows' DRAM reads and, between
// them, the chain of barriers bound it: 4096 rows of 16,384 lists, p = 72, take
// 78 us (HBM needs 41 for their 268 MB) where a histogram of all keys, a second
// pass and the sort of its boundary bin took 127; 4,096 lists 25 us for 52.
constexpr uint32_t kSelBins = 1024;

__device__ __forceinline__ uint32_t min4(uint4 x) { return min(min(x.x, x.y), min(x.z, x.w)); }

template <uint32_t NT, uint32_t V>
__global__ void __launch_bounds__(NT) select_topp_near_kernel(
    const float *dists, uint32_t n, uint32_t p, uint32_t stride, uint32_t level, uint32_t cap,
    uint32_t *probed, uint32_t *cnt, unsigned long long *tie_count, const uint32_t *only,
    uint32_t only_above) {
  after_previous();
  extern __shared__ unsigned long long cand[];  // cap keys (key << 32 | list)
  uint16_t *order = reinterpret_cast<uint16_t *>(cand + cap);
  __shared__ uint32_t hist[kSelBins], wlo[NT / 32], whi[NT / 32], wsum[NT / 32], scal[4];
  constexpr uint32_t kNone = 0xFFFFFFFFu;  // no key: above every distance
  constexpr uint32_t kPer = kSelBins / NT;
  const uint32_t q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (only && only[q] <= only_above) return;
  const uint32_t *keys = reinterpret_cast<const uint32_t *>(dists) + static_cast<size_t>(q) * n;
  uint32_t *outp = probed + static_cast<size_t>(q) * stride;
  const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15) == 0;
  // keys 4 i .. 4 i + 3
  auto load = [&](uint32_t i) -> uint4 {
    const uint32_t i4 = 4 * i;
    if (vec && i4 + 4 <= n) return reinterpret_cast<const uint4 *>(keys)[i];
    return make_uint4(i4 < n ? keys[i4] : kNone, i4 + 1 < n ? keys[i4 + 1] : kNone,
                      i4 + 2 < n ? keys[i4 + 2] : kNone, i4 + 3 < n ? keys[i4 + 3] : kNone);
  };
  uint4 held[V ? V : 1];
  if constexpr (V > 0) {
#pragma unroll
    for (uint32_t v = 0; v < V; ++v) held[v] = load(v * NT + tid);
  }
  for (uint32_t i = tid; i < kSelBins; i += NT) hist[i] = 0;
  if (tid < 4) scal[tid] = 0;
  // f(four keys, the first one's index) over the thread's keys
  auto each = [&](auto f) {
    if constexpr (V > 0) {
#pragma unroll
      for (uint32_t v = 0; v < V; ++v) f(held[v], 4 * (v * NT + tid));
    } else {
      for (uint32_t i = tid; i < (n + 3) / 4; i += NT) f(load(i), 4 * i);
    }
  };
  // 1) the range of the minima
  uint32_t tmin = kNone, hi = 0;
  auto top = [&](uint32_t k) { hi = k == kNone ? hi : max(hi, k); };
  each([&](uint4 x, uint32_t) {
    const uint32_t m = min4(x);
    tmin = min(tmin, m);
    if (level == 1) top(m);
    if (level == 2) top(x.x), top(x.y), top(x.z), top(x.w);
  });
  if (level == 0) top(tmin);
  const uint32_t wl = __reduce_min_sync(0xffffffffu, tmin), wh = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) wlo[warp] = wl, whi[warp] = wh;
  __syncthreads();
  const uint32_t lo = __reduce_min_sync(0xffffffffu, wlo[lane % (NT / 32)]);
  const uint32_t range = __reduce_max_sync(0xffffffffu, whi[lane % (NT / 32)]) - lo;
  const uint32_t shift = range < kSelBins ? 0 : 32 - __clz(range) - 10;
  // 2) the bin of rank p - 1: each thread owns kPer consecutive bins
  auto tally = [&](uint32_t k) {
    if (k != kNone) atomicAdd(&hist[(k - lo) >> shift], 1u);
  };
  if (level == 0) {
    tally(tmin);
  } else {
    each([&](uint4 x, uint32_t) {
      if (level == 1) tally(min4(x));
      else tally(x.x), tally(x.y), tally(x.z), tally(x.w);
    });
  }
  __syncthreads();
  // the keys in bins below the thread's own, and in them
  uint32_t sum;
  auto scan_bins = [&]() -> uint32_t {
    sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) sum += hist[tid * kPer + j];
    uint32_t incl = sum;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t below = incl - sum;
#pragma unroll
    for (uint32_t w = 0; w < NT / 32; ++w) below += w < warp ? wsum[w] : 0;
    return below;
  };
  uint32_t below = scan_bins();
  if (p - 1 >= below && p - 1 < below + sum) {
    uint32_t j = 0;
    for (; j < kPer - 1; ++j) {
      below += hist[tid * kPer + j];
      if (p - 1 < below) break;
    }
    scal[0] = min(lo + min(((tid * kPer + j + 1) << shift) - 1, ~lo), kNone - 1);
  }
  __syncthreads();
  // 3) the keys up to it
  const uint32_t T = scal[0];
  for (uint32_t i = tid; i < kSelBins; i += NT) hist[i] = 0;
  each([&](uint4 x, uint32_t i) {
    if (min4(x) > T) return;
    const uint32_t k[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      if (k[j] > T) continue;
      const uint32_t at = atomicAdd(&scal[1], 1u);
      if (at < cap) cand[at] = (static_cast<unsigned long long>(k[j]) << 32) | (i + j);
    }
  });
  __syncthreads();
  const uint32_t c = scal[1];
  if (c > cap) {
    select_passes(keys, n, p, outp, cnt, tie_count, cand, hist, scal);
    return;
  }
  // 4) the first p of them in order
  auto put = [&](uint32_t at, uint32_t list) {
    outp[at] = list;
    if (cnt) atomicAdd(&cnt[list], 1u);
  };
  auto ranked = [&](uint32_t at, unsigned long long k) {
    if (at < p) put(at, static_cast<uint32_t>(k));
    if (at + 1 == p) scal[2] = static_cast<uint32_t>(k >> 32);
    if (at == p) scal[3] = static_cast<uint32_t>(k >> 32);
  };
  if (c <= NT / 4) {
    // 2^lg threads count the keys below each
    uint32_t lg = 0;
    while (lg < 5 && (c << (lg + 1)) <= NT) ++lg;
    const uint32_t g = tid >> lg;
    const unsigned long long mine = cand[min(g, c - 1)];
    uint32_t less = 0;
    for (uint32_t j = tid & ((1u << lg) - 1); j < c; j += 1u << lg) less += cand[j] < mine;
    for (uint32_t o = 1; o < 1u << lg; o <<= 1) less += __shfl_xor_sync(0xffffffffu, less, o);
    if (g < c && (tid & ((1u << lg) - 1)) == 0) ranked(less, mine);
    __syncthreads();
    if (tid == 0 && tie_count && c > p && scal[2] == scal[3]) atomicAdd(tie_count, 1ull);
    return;
  }
  const uint32_t near = T - lo, shift2 = near < kSelBins ? 0 : 32 - __clz(near) - 10;
  auto bin_of = [&](unsigned long long k) { return (static_cast<uint32_t>(k >> 32) - lo) >> shift2; };
  for (uint32_t i = tid; i < c; i += NT) atomicAdd(&hist[bin_of(cand[i])], 1u);
  __syncthreads();
  below = scan_bins();
  bool crowded = false;
#pragma unroll
  for (uint32_t j = 0; j < kPer; ++j) {
    const uint32_t h = hist[tid * kPer + j];
    crowded |= h > 32;
    hist[tid * kPer + j] = below;
    below += h;
  }
  if (!__syncthreads_or(crowded)) {
    for (uint32_t i = tid; i < c; i += NT) order[atomicAdd(&hist[bin_of(cand[i])], 1u)] = static_cast<uint16_t>(i);
    __syncthreads();
    // bin b is now order[hist[b - 1]] .. order[hist[b] - 1]
    for (uint32_t i = tid; i < c; i += NT) {
      const unsigned long long mine = cand[i];
      const uint32_t b = bin_of(mine), end = hist[b];
      uint32_t less = b ? hist[b - 1] : 0;
      if (less > p) continue;
      for (uint32_t j = less; j < end; ++j) less += cand[order[j]] < mine;
      ranked(less, mine);
    }
    __syncthreads();
    if (tid == 0 && tie_count && c > p && scal[2] == scal[3]) atomicAdd(tie_count, 1ull);
  } else {
    sort_keys(cand, c);
    for (uint32_t i = tid; i < p; i += NT) put(i, static_cast<uint32_t>(cand[i]));
    if (tid == 0 && tie_count && c > p && (cand[p] >> 32) == (cand[p - 1] >> 32)) atomicAdd(tie_count, 1ull);
  }
}

__global__ void dist_values_kernel(const int64_t *l2, uint32_t n, DistScale s, float *out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = dist_value(l2[i], s);
}

}  // namespace

int sq16_tiles(const uint8_t *qhi, const uint8_t *qlo, const uint8_t *xhi, const uint8_t *xlo,
               const int64_t *qn, const int64_t *xn, double step_sq, uint32_t m, uint32_t n,
               uint32_t dims, uint32_t qstride, uint32_t xstride, float *out, bool full,
               cudaStream_t st) {
  if (m == 0 || n == 0) return KATO_OK;
  if (dims % 64 || dims == 0) return invalid("dims must be a positive multiple of 64");
  if (qstride % 16 || xstride % 16) return invalid("row strides must be multiples of 16 bytes");
  const DistScale s = make_dist_scale(step_sq);
  dim3 grid(div_up(n, kTile), div_up(m, kTile));
  if (grid.y > 65535) return invalid("too many query rows for one call");
  if (full) launch(sq16_tile_kernel<true>, grid, 256, 0, st, qhi, qlo, xhi, xlo, qn, xn, s, m, n, dims, qstride, xstride, out);
  else launch(sq16_tile_kernel<false>, grid, 256, 0, st, qhi, qlo, xhi, xlo, qn, xn, s, m, n, dims, qstride, xstride, out);
  KATO_LAUNCHED("sq16_tile_kernel");
  return KATO_OK;
}

int select_topp_ex(const float *dists, uint32_t nq, uint32_t n, uint32_t p, uint32_t stride,
                   uint32_t *probed, uint32_t *cnt, unsigned long long *tie_count,
                   const uint32_t *only, uint32_t only_above, cudaStream_t st) {
  if (nq == 0) return KATO_OK;
  if (p == 0 || p > n || stride < p) return invalid("need 1 <= nprobe <= nlist");
  if (p <= kSortMax) {
    uint32_t cap = 1024;
    while (cap < p) cap <<= 1;
    cap *= 2;
    // A row in one thread block's registers where it fits: the smallest block
    // that takes at most 8 loads a thread, as smaller blocks overlap one row's
    // loads with another's ranking (4096 rows of 4,096 lists: 25 us with 256
    // threads, 36 with 512; 2000 rows of 5,000, p = 384: 39 and 49). 16,384
    // lists: 512 threads 78 us, 256 with 16 loads 96, 1024 with four 127, reading
    // the row again 90; 2000 rows of 5,000 read again 41.
    auto go = [&](auto kern, uint32_t threads) -> int {
      if (const int rc = smem_limit(reinterpret_cast<const void *>(kern), 2 * kSortMax * 10,
                                    "select_topp_near_kernel shared memory"))
        return rc;
      // the largest groups that still leave few keys below the bound: p of 3 p
      // minima leave 1.2 p, p of 3 p / 2 leave 1.7 p
      const uint32_t level = std::min(threads, div_up(n, 4)) >= 3 * p ? 0 : div_up(n, 4) >= 3 * p / 2 ? 1 : 2;
      launch(kern, nq, threads, cap * 10, st, dists, n, p, stride, level, cap, probed,
                                                                  cnt, tie_count, only, only_above);
      KATO_LAUNCHED("select_topp_near_kernel");
      return KATO_OK;
    };
    if (n <= 1024) return go(select_topp_near_kernel<128, 2>, 128);
    if (n <= 4096) return go(select_topp_near_kernel<256, 4>, 256);
    if (n <= 8192) return go(select_topp_near_kernel<256, 8>, 256);
    if (n <= 16384) return go(select_topp_near_kernel<512, 8>, 512);
    return go(select_topp_near_kernel<512, 0>, 512);
  }
  launch(select_topp_kernel, nq, kSelThreads, 0, st, dists, n, p, stride, probed, cnt, tie_count,
                                                  only, only_above);
  KATO_LAUNCHED("select_topp_kernel");
  return KATO_OK;
}

int select_topp(const float *dists, uint32_t nq, uint32_t n, uint32_t p, uint32_t *probed,
                unsigned long long *tie_count, cudaStream_t st) {
  return select_topp_ex(dists, nq, n, p, p, probed, nullptr, tie_count, nullptr, 0, st);
}

int dist_values(const int64_t *l2, uint32_t n, double step_sq, float *out, cudaStream_t st) {
  if (n == 0) return KATO_OK;
  dist_values_kernel<<<div_up(n, 256), 256, 0, st>>>(l2, n, make_dist_scale(step_sq), out);
  KATO_LAUNCHED("dist_values_kernel");
  return KATO_OK;
}

}  // namespace kato
