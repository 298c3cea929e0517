// Inversion of the probe lists and the ranking pass's work items.
//
// The reference inverts the probe lists into a hash map (invert,
// src/index.cpp:403-412) and scans each probed list once for all the queries
// that probe it (:998-1044). Here the inversion is a CSR of list -> (query,
// rank): counts (left by the coarse selection itself, unless budgets cut the
// probes), one scan of everything that follows from them, and one kernel that
// scatters the entries and writes the work items. These steps move little; a
// small search pays for their launches, so there are two instead of seven.
#include <algorithm>

#include "invert.cuh"
#include "scan.cuh"

namespace kato {

namespace {

// A (query, rank) pair i = query * p + rank is probed when the query's
// budget (if any) exceeds the rank: its p nearest lists are in order, so a
// budget of b probes exactly the lists a fixed nprobe of b would.
__device__ __forceinline__ bool probed_pair(uint32_t i, uint32_t p,
                                            const uint32_t *qprobes) {
  return !qprobes || i % p < qprobes[i / p];
}

__global__ void count_kernel(const uint32_t *probed, uint32_t total, uint32_t p,
                             const uint32_t *qprobes, uint32_t *cnt) {
  after_previous();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total && probed_pair(i, p, qprobes)) atomicAdd(&cnt[probed[i]], 1u);
}

// The cost of a slab of an item of ne queries: by default in steps of about
// 20 instructions (180 for the rows and 40 per group of 8 queries), or
// 64 + beta * width (16, 32 or N queries).
__device__ __forceinline__ uint32_t slab_cost(uint32_t ne, uint32_t N, uint32_t beta) {
  if (beta == 0) return 9 + 2 * ((ne + 7) / 8);
  return 64 + beta * (ne <= 16 ? 16u : (ne <= 32 && N > 32 ? 32u : N));
}

// Per list, the exclusive sums of its queries (off, cur), items (ceil(queries /
// N); on the tensor-core pass none for an empty list), slabs and cost (base),
// with the totals after them.
__global__ void __launch_bounds__(1024) invert_scan_kernel(const InvertArgs A) {
  after_previous();
  const uint32_t L = A.L, N = A.N;
  uint32_t *ci = A.base, *cs = ci + L + 1, *cc = cs + L + 1;
  const uint4 tot = block_scan4(
      L,
      [&](uint32_t c) {
        const uint32_t v = A.cnt[c];
        if (!A.items) return make_uint4(v, (v + N - 1) / N, 0, 0);
        const uint32_t n = A.list_off[c + 1] - A.list_off[c];
        const uint32_t slabs = (n + kTcSlab - 1) / kTcSlab, full = v / N, rem = v % N;
        const uint32_t cost = full * slab_cost(N, N, A.beta) + (rem ? slab_cost(rem, N, A.beta) : 0);
        const uint32_t items = n ? full + (rem != 0) : 0;
        return make_uint4(v, items, items * slabs, slabs * cost);
      },
      [&](uint32_t c, uint4 s) {
        A.off[c] = A.cur[c] = s.x;
        ci[c] = s.y;
        cs[c] = s.z;
        cc[c] = s.w;
      });
  if (threadIdx.x == 0) {
    A.off[L] = tot.x;
    ci[L] = tot.y;
    cs[L] = tot.z;
    cc[L] = tot.w;
    if (A.items) A.tile_off[tot.y] = tot.z;
  }
}

// Thread i: scatters probe slot i, writes the items of list i and finds where
// share i starts.
__global__ void invert_expand_kernel(const InvertArgs A) {
  after_previous();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, L = A.L, N = A.N;
  const uint32_t *ci = A.base, *cs = ci + L + 1;
  if (i < A.B * A.p && probed_pair(i, A.p, A.qprobes))
    A.entries[atomicAdd(&A.cur[A.probed[i]], 1u)] = i;
  if (!A.items) {
    if (i < L)
      for (uint32_t j = ci[i]; j < ci[i + 1]; ++j) A.work[j] = Work{i, (j - ci[i]) * N};
    return;
  }
  if (i <= A.ctas) {
    const uint32_t *unit = A.by_cost ? cs + L + 1 : cs;  // a list's first unit
    uint2 at = make_uint2(cs[L], ci[L]);  // the end: all slabs, all items
    if (i < A.ctas && unit[L]) {
      // share i starts at unit total * i / ctas: the list that holds it, then
      // the item (every one before a list's last is full) and the slab
      const uint32_t u = static_cast<uint32_t>(static_cast<uint64_t>(unit[L]) * i / A.ctas);
      uint32_t lo = 0, hi = L;  // unit[lo] <= u < unit[hi]
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (unit[mid] <= u) lo = mid;
        else hi = mid;
      }
      const uint32_t n = A.cnt[lo], slabs = (A.list_off[lo + 1] - A.list_off[lo] + kTcSlab - 1) / kTcSlab;
      const uint32_t full = slabs * (A.by_cost ? slab_cost(N, N, A.beta) : 1), in = u - unit[lo];
      const uint32_t j = min(in / full, (n - 1) / N);
      const uint32_t per = A.by_cost ? slab_cost(min(N, n - j * N), N, A.beta) : 1;
      at = make_uint2(cs[lo] + j * slabs + (in - j * full) / per, ci[lo] + j);
    }
    A.share[i] = at;
  }
  if (blockIdx.x * blockDim.x >= L) return;  // whole CTAs: the statistics take whole warps
  uint32_t hist[6] = {0, 0, 0, 0, 0, 0}, lists = 0, probed_rows = 0;
  if (i < L) {
    const uint32_t i0 = ci[i], n_items = ci[i + 1] - i0;
    const uint32_t row0 = A.list_off[i], rows = A.list_off[i + 1] - row0;
    const uint32_t slabs = (rows + kTcSlab - 1) / kTcSlab, tiles = (rows + kTcRows - 1) / kTcRows;
    if (n_items) lists = 1, probed_rows = rows;
    for (uint32_t j = 0; j < n_items; ++j) {
      const uint32_t ne = min(N, A.cnt[i] - j * N);
      A.items[i0 + j] = TcItem{A.off[i] + j * N, ne, row0, rows};
      A.tile_off[i0 + j] = cs[i] + j * slabs;
      hist[ne <= 2 ? 0 : ne <= 4 ? 1 : ne <= 8 ? 2 : ne <= 16 ? 3 : ne <= 32 ? 4 : 5] += tiles;
    }
  }
  // one add per warp and counter
  auto add = [&](unsigned long long *to, uint32_t v) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(to, static_cast<unsigned long long>(v));
    return v;
  };
  uint32_t all = 0;
#pragma unroll
  for (int b = 0; b < 6; ++b) all += add(A.tile_hist + b, hist[b]);
  add(A.tile_hist + 6, lists);
  add(A.tile_hist + 7, probed_rows);
  if ((threadIdx.x & 31) == 0 && all) atomicAdd(A.tiles, static_cast<unsigned long long>(all));
}

}  // namespace

int invert(const InvertArgs &A, bool counted, uint32_t *launches, cudaStream_t st) {
  const uint32_t total = A.B * A.p;
  if (!counted) {
    launch(count_kernel, div_up(total, 256), 256, 0, st, A.probed, total, A.p, A.qprobes, A.cnt);
    ++*launches;
  }
  launch(invert_scan_kernel, 1, 1024, 0, st, A);
  launch(invert_expand_kernel, div_up(std::max(std::max(total, A.L), A.ctas + 1), 256), 256, 0, st, A);
  *launches += 2;
  KATO_LAUNCHED("inversion kernels");
  return KATO_OK;
}

}  // namespace kato
