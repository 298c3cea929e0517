// Dot products of one query with many rows' high bytes on the CUDA cores, and
// radix selection over computed keys, by one CTA: the seed bounds and the
// overflow rescan of the ranking pass.
#pragma once

#include "kcommon.cuh"
#include "scan.cuh"

namespace kato {

// The squared L2 over the first h high bytes of a row and a query whose bytes
// are in shared memory as words; dp4a over 16 bytes per step.
__device__ __forceinline__ uint32_t row_dot(const uint8_t *row, const uint32_t *qw, uint32_t h) {
  const uint4 *rv = reinterpret_cast<const uint4 *>(row);
  uint32_t dot = 0;
  uint32_t u = 0;
  for (; u + 4 <= h / 16; u += 4) {  // four loads in flight
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __ldg(rv + u + j);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t *w = qw + 4 * (u + j);
      dot = dp4(v[j].x, w[0], dp4(v[j].y, w[1], dp4(v[j].z, w[2], dp4(v[j].w, w[3], dot))));
    }
  }
  for (; u < h / 16; ++u) {
    const uint4 v = __ldg(rv + u);
    const uint32_t *w = qw + 4 * u;
    dot = dp4(v.x, w[0], dp4(v.y, w[1], dp4(v.z, w[2], dp4(v.w, w[3], dot))));
  }
  return dot;
}

// Dot products of a query (its h bytes as words in shared memory) with rows
// row(0) .. row(n - 1) of a byte plane, lanes split along each row: a group of
// G = 4, 8, 16 or 32 lanes (32 from h = 512 on, whose last step some sit out
// where h / 16 is no multiple of it) reads a row as one coalesced run of 16-byte
// loads and sums over the group by shuffles. A warp takes 32 rows at a time
// (G steps, all loads of the batch in flight together) and hands row
// base + l of the batch to one lane, so f(i, dot) runs on all 32 lanes at
// once. All threads of the CTA take part.
//
// pre(i) - a per-row value the callback needs (e.g. the row's norm) - is
// loaded at the start of the batch by the lane that later calls
// f(i, dot, pre(i)), so that it arrives with the rows instead of after them.

template <uint32_t G, typename F, typename Pre, typename RowAt>
__device__ __forceinline__ void rows_split(const uint8_t *__restrict__ x, uint32_t dc, uint32_t h,
                                           const uint32_t *qw, RowAt row, uint32_t n, Pre pre,
                                           F f) {
  constexpr uint32_t RPW = 32 / G;  // rows per step
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t sub = lane / G, gl = lane % G, units = h / 16;
  for (uint32_t base = warp * 32; base < n; base += nw * 32) {
    uint32_t mine = 0;
    const uint32_t my_row = base + gl * RPW + sub;
    const int64_t pv = my_row < n ? pre(my_row) : 0;
    if (G <= 16 && units == G) {
      // every load of the batch first, then the sums
      uint4 v[G <= 16 ? G : 1];
      const uint32_t *w = qw + 4 * gl;
#pragma unroll
      for (uint32_t it = 0; it < (G <= 16 ? G : 1); ++it) {
        const uint32_t i = base + it * RPW + sub;
        v[it] = i < n ? __ldg(reinterpret_cast<const uint4 *>(x + static_cast<size_t>(row(i)) * dc) + gl)
                      : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (uint32_t it = 0; it < (G <= 16 ? G : 1); ++it) {
        uint32_t dot = dp4(v[it].x, w[0], dp4(v[it].y, w[1], dp4(v[it].z, w[2], dp4(v[it].w, w[3], 0))));
#pragma unroll
        for (uint32_t o = G / 2; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (gl == it) mine = dot;
      }
    } else {
#pragma unroll 4
      for (uint32_t it = 0; it < G; ++it) {
        const uint32_t i = base + it * RPW + sub;
        uint32_t dot = 0;
        if (i < n) {
          const uint4 *rv = reinterpret_cast<const uint4 *>(x + static_cast<size_t>(row(i)) * dc);
          for (uint32_t c = 0; c < (units + G - 1) / G; ++c) {
            const uint32_t u = gl + c * G;
            if (u >= units) break;
            const uint4 vv = __ldg(rv + u);
            const uint32_t *w = qw + 4 * u;
            dot = dp4(vv.x, w[0], dp4(vv.y, w[1], dp4(vv.z, w[2], dp4(vv.w, w[3], dot))));
          }
        }
#pragma unroll
        for (uint32_t o = G / 2; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (gl == it) mine = dot;
      }
    }
    if (my_row < n) f(my_row, mine, pv);
  }
}

// rows_split with the group size for h.
template <typename F, typename Pre, typename RowAt>
__device__ __forceinline__ void for_rows_at(const uint8_t *__restrict__ x, uint32_t dc, uint32_t h,
                                            const uint32_t *qw, RowAt row, uint32_t n, F f, Pre pre) {
  const uint32_t g = min(32u, h / 16);
  if (g == 16) rows_split<16>(x, dc, h, qw, row, n, pre, f);
  else if (g == 32) rows_split<32>(x, dc, h, qw, row, n, pre, f);
  else if (g == 8) rows_split<8>(x, dc, h, qw, row, n, pre, f);
  else rows_split<4>(x, dc, h, qw, row, n, pre, f);
}

// The same over the contiguous rows r0 .. r0 + n - 1.
template <typename F, typename Pre>
__device__ __forceinline__ void for_rows_split(const uint8_t *__restrict__ x, uint32_t dc, uint32_t h,
                                               const uint32_t *qw, uint32_t r0, uint32_t n, F f,
                                               Pre pre) {
  for_rows_at(x, dc, h, qw, [r0](uint32_t i) { return r0 + i; }, n, f, pre);
}

// The rank-th smallest 64-bit key produced by key(i), i < n, by 8-bit radix
// digits; all threads of the CTA call it and get the key.
template <typename KeyAt>
__device__ unsigned long long block_select64(uint32_t n, uint32_t rank, KeyAt key, uint32_t *hist,
                                             uint32_t *sel) {
  __shared__ uint32_t wsum[8];
  unsigned long long prefix = 0;
  for (int shift = 56; shift >= 0; shift -= 8) {
    for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const unsigned long long hm = shift == 56 ? 0ull : (~0ull << (shift + 8));
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned long long k = key(i);
      if ((k & hm) == prefix) atomicAdd(&hist[(k >> shift) & 0xFFu], 1u);
    }
    __syncthreads();
    block_pick_digit(hist, rank, sel, wsum);
    rank -= sel[1];
    prefix |= static_cast<unsigned long long>(sel[0]) << shift;
    __syncthreads();
  }
  return prefix;
}

struct RowKey {
  const uint8_t *xhi;
  const int64_t *xnorm;
  const uint32_t *ids;
  uint32_t dc, h;
  DistScale scale;
  __device__ unsigned long long operator()(uint32_t row, const uint32_t *qw, int64_t qn) const {
    const uint32_t dot = row_dot(xhi + static_cast<size_t>(row) * dc, qw, h);
    const int64_t l2 = qn + xnorm[row] - 2 * static_cast<int64_t>(dot);
    return (static_cast<unsigned long long>(__float_as_uint(dist_value(l2, scale))) << 32) | ids[row];
  }
};

__device__ __forceinline__ void load_query_words(const uint8_t *qhi, uint32_t q, uint32_t dc,
                                                 uint32_t h, uint32_t *qw) {
  for (uint32_t i = threadIdx.x; i < h / 4; i += blockDim.x)
    qw[i] = reinterpret_cast<const uint32_t *>(qhi + static_cast<size_t>(q) * dc)[i];
}

}  // namespace kato
