// The end of a search (finish.cu): per query, the best candidates of the
// ranking pass, their exact distances and the top-k.
#pragma once

#include <cstdint>

#include "kcommon.cuh"

namespace kato {

struct FinishArgs {
  uint2 *slots;             // per query: per_query candidates (distance bits, row)
  uint32_t per_query, per_probe;
  const uint32_t *qcount;   // candidates per query (bit 31: some were dropped), or null: fixed slots
  const uint32_t *qprobes;  // per-query budgets, or null
  const uint8_t *qhi, *qlo;
  const int64_t *qnorm;     // over all dimensions, 16-bit codes
  const uint8_t *xhi, *xlo;
  const int64_t *xnorm;
  const uint32_t *ids;
  uint32_t npts, dc, S, k;
  DistScale scale;
  uint32_t *out_ids;
  float *out_dists;
  unsigned long long *ties;     // queries tied at the survivor boundary
  unsigned long long *rescans;  // [0] queries rescanned, [1] most candidates of one
  // the rescan of a query with more than per_query candidates (with qcount)
  const int64_t *rank_xnorm, *rank_qnorm;
  const uint32_t *probed, *list_off;
  uint32_t h, nprobe;
  // where a query can probe more rows than its buffer holds: per query, whether
  // it was rescanned by the whole grid before, and the key it was rescanned for;
  // those queries and their number (0 before the pass)
  uint32_t *over, *over_list, *over_n;
  unsigned long long *over_key;
};

// The first rescan of queries with more candidates than their buffers hold (with
// `over`; writes qcount), by the whole grid.
int rescan_overflows(const FinishArgs &A, uint32_t *qcount, uint32_t nq, cudaStream_t st);
// Survivors, refinement and top-k of nq queries (ranked modes).
int finish(const FinishArgs &A, uint32_t nq, cudaStream_t st);
// Top-k of slots of exact distances (full ranking): per query per_query
// entries, of which qcount are used or, without it, per_probe for each of its
// probes.
int merge_topk(const uint2 *slots, uint32_t per_query, uint32_t per_probe, const uint32_t *qcount,
               const uint32_t *qprobes, const uint32_t *ids, uint32_t nq, uint32_t k, uint32_t *out_ids, float *out_dists,
               unsigned long long *ties, cudaStream_t st);

}  // namespace kato
