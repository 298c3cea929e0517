// From each query's probed lists to the ranking pass's work (invert.cu).
#pragma once

#include <cstdint>

#include "kcommon.cuh"
#include "rank_tc.cuh"

namespace kato {

// A work item of the CUDA-core ranking pass: a list and the first of up to N
// of its probe entries.
struct Work {
  uint32_t list, first;
};

struct InvertArgs {
  const uint32_t *probed;   // B x p lists, nearest first
  const uint32_t *qprobes;  // per-query budgets, or null
  uint32_t B, p, L, N;      // N: queries per item
  const uint32_t *list_off;
  uint32_t *cnt;            // L: queries per list (0 before the pass)
  uint32_t *off;            // L + 1: first probe entry of each list
  uint32_t *cur;            // L: scatter cursors
  uint32_t *base;           // 3 x (L + 1): first item, first slab, first cost unit of each list
  uint32_t *entries;        // the probe slots (query * p + rank), grouped by list
  Work *work;               // CUDA-core pass: its items (count in base[L])
  // tensor-core pass (items non-null): items, their first slabs (one more: the
  // total), the shares of ctas CTAs (one more) of equal slabs or, by_cost, of
  // equal cost: what a slab's instructions do with beta 0, or 64 + beta w for
  // an item of width w (16, 32 or N)
  TcItem *items;
  uint32_t *tile_off;
  uint2 *share;
  uint32_t ctas, beta;
  bool by_cost;
  // 6 counters of 128-row tiles by item width, then the distinct probed lists
  // and their rows; all tiles
  unsigned long long *tile_hist, *tiles;
};

// Inverts the probes (counted: cnt already holds the counts, from the
// selection) and lays out the work; adds its launches.
int invert(const InvertArgs &A, bool counted, uint32_t *launches, cudaStream_t st);

}  // namespace kato
