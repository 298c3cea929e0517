// Exclusive prefix sums of four sequences at once by one CTA of 1024 threads
// (the list-sized scans of the search: nlist is at most a few 10^5), and a
// radix-selection step.
#pragma once

#include <cstdint>

namespace kato {

__device__ __forceinline__ uint4 add4(uint4 a, uint4 b) {
  return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ uint4 warp_scan4(uint4 x, uint32_t lane) {  // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint4 y = make_uint4(__shfl_up_sync(0xffffffffu, x.x, o), __shfl_up_sync(0xffffffffu, x.y, o),
                               __shfl_up_sync(0xffffffffu, x.z, o), __shfl_up_sync(0xffffffffu, x.w, o));
    if (lane >= static_cast<uint32_t>(o)) x = add4(x, y);
  }
  return x;
}

// val(i) gives the values at i < n; out(i, sums) receives the exclusive prefix
// sums there. Tiles of 4096: each thread takes 4 consecutive values (coalesced
// across the CTA), warps scan with shuffles. Returns the totals; all threads
// of the CTA must call it.
template <typename Val, typename Out>
__device__ uint4 block_scan4(uint32_t n, Val val, Out out) {
  __shared__ uint4 wsum[32];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint4 carry = make_uint4(0, 0, 0, 0);
  for (uint32_t base = 0; base < n; base += 4096) {
    const uint32_t i0 = base + t * 4;
    uint4 v[4], ts = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = i0 + k < n ? val(i0 + k) : make_uint4(0, 0, 0, 0);
      ts = add4(ts, v[k]);
    }
    const uint4 x = warp_scan4(ts, lane);
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    // every warp scans the warp totals: no second barrier round
    const uint4 w = warp_scan4(wsum[lane], lane);
    const int before = warp ? static_cast<int>(warp) - 1 : 0;
    uint4 e = make_uint4(__shfl_sync(0xffffffffu, w.x, before), __shfl_sync(0xffffffffu, w.y, before),
                         __shfl_sync(0xffffffffu, w.z, before), __shfl_sync(0xffffffffu, w.w, before));
    const uint4 tile = make_uint4(__shfl_sync(0xffffffffu, w.x, 31), __shfl_sync(0xffffffffu, w.y, 31),
                                  __shfl_sync(0xffffffffu, w.z, 31), __shfl_sync(0xffffffffu, w.w, 31));
    if (warp == 0) e = make_uint4(0, 0, 0, 0);
    e = add4(carry, add4(e, make_uint4(x.x - ts.x, x.y - ts.y, x.z - ts.z, x.w - ts.w)));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k < n) out(i0 + k, e);
      e = add4(e, v[k]);
    }
    carry = add4(carry, tile);
    __syncthreads();  // wsum is written again
  }
  return carry;
}

// Radix-selection step by a whole CTA (blockDim.x >= 256, whole warps): the
// bin of a 256-bin histogram that holds the rank-th smallest value (rank <
// the histogram's total), into sel[0], and the count below that bin, into
// sel[1]. Thread t owns bin t; warp scans and the 8 warp totals (wsum) give
// each bin's exclusive prefix, and the one bin whose range holds the rank
// writes. Contains barriers: every thread of the CTA calls it.
__device__ __forceinline__ void block_pick_digit(const uint32_t *hist, uint32_t rank, uint32_t *sel,
                                                 uint32_t *wsum) {
  const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint32_t h = t < 256 ? hist[t] : 0u;
  uint32_t incl = h;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (t < 256 && lane == 31) wsum[w] = incl;
  __syncthreads();
  if (t < 256) {
    uint32_t base = 0;
    for (uint32_t i = 0; i < w; ++i) base += wsum[i];
    const uint32_t excl = base + incl - h;
    if (rank >= excl && rank < excl + h) {
      sel[0] = t;
      sel[1] = excl;
    }
  }
  __syncthreads();
}

}  // namespace kato
