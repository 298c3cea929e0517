// Declarations shared by the tensor-core ranking pass (rank_tc.cu) and the
// search orchestration (search.cu).
#pragma once

#include <cuda_fp16.h>

#include <atomic>

#include <cstdint>

#include "kcommon.cuh"

namespace kato {

// One work item: a list's rows [row0, +nrows) and up to N of the queries that
// probe it (probe entries [e0, +ne)); its slabs are the rows, 64 each.
struct TcItem {
  uint32_t e0, ne, row0, nrows;
};

struct RankTcArgs {
  const __half *qr16;        // B query rows of the ranking bytes in fp16, zero-padded to chunks
  const int2 *qcn;           // per query: sums of its squared values over f and over h dimensions
  const uint32_t *entries;   // probe slots (query * nprobe + rank) grouped by list
  const TcItem *items;
  const uint32_t *tile_off;  // per item: first global slab; [nitems] = total slabs
  const uint2 *share;        // per CTA and one more: its first slab and that slab's item
  const int32_t *bound;      // per query: rows with a larger l2 cannot be selected
  uint32_t *qcount;          // per query: bit 31 is set when a record was dropped
  uint4 *rec;                // per CTA: rec_cap records (query, xn - 2 dot, row, partial)
  uint32_t *rec_n;           // per CTA: records written
  uint32_t rec_cap;
  uint32_t *timeouts;        // CTAs whose bounded pipeline wait ran out
  unsigned long long *prof;  // optional: cycle counters of the warp roles
  // f: dimensions of a filtered item (h: no item is filtered)
  uint32_t dc, h, f, nprobe;
  long long wait;            // cycles a pipeline wait may take before the CTA gives up
};

// Launch shape: N queries per item, Bs query buffers, Rs ring stages per
// scoring warp of `inner` bytes per row, f filter dimensions.
struct TcShape {
  uint32_t N, Bs, Rs, inner, f, smem;
  uint32_t centred;  // values enter as (byte - 128), not as the byte
};

// The ranking pass's copy of a batch's queries (rows null: none): their first
// h high bytes as fp16, centred or not, zero-padded to `width`, and the sums of
// the squared values over f and h.
struct RankRows {
  __half *rows;
  int2 *norms;
  uint32_t f, h, width, centred;
};

// A batch's coded queries (rows of dc) and what is derived from them
// (query_planes): byte planes, norms, and with hi16 the centred fp16 planes and
// terms of the coarse product. `zeros` words at `zero` are cleared on the way.
struct QueryPlanes {
  uint8_t *hi, *lo;
  int64_t *norm, *hinorm, *headnorm;
  uint32_t dc, head;
  __half *hi16, *lo16;
  int64_t *term;
  uint32_t *zero, zeros;
};
int query_planes(const float *x, uint32_t nrows, uint32_t d, float lo, double inv_step,
                 const QueryPlanes &P, const RankRows &rr, cudaStream_t st);

// Shared-memory carve-up of the ranking CTA.
struct TcSmem {
  uint32_t raw, b, qids, qbv, desc, bars, err, rcount, total;
};

__host__ __device__ inline uint32_t tc_take(uint32_t &o, uint32_t bytes, uint32_t align) {
  o = (o + align - 1) / align * align;
  const uint32_t at = o;
  o += bytes;
  return at;
}

constexpr uint32_t kDropped = 0x80000000u;  // qcount flag: a record did not fit
constexpr uint32_t kTcRows = 128;     // rows per tile of the statistics
// Dimensions of a filtered item: one chunk of 128 bytes per row.
constexpr uint32_t kTcFilterDims = 128;
constexpr uint32_t kTcBoxRows = 32;   // rows per TMA box: two mma row tiles
constexpr uint32_t kTcSlab = 64;      // rows per slab
constexpr uint32_t kTcScoreWarps = 8;
constexpr uint32_t kTcMaxStages = 4;  // ring stages per scoring warp, at most
constexpr uint32_t kTcMaxBufs = 4;    // query buffers, at most
constexpr uint32_t kTcDesc = 32;      // bytes per item description

// fp16 values of a query's row in RankTcArgs::qr16.
__host__ __device__ inline uint32_t tc_qrow(uint32_t h, const TcShape &s) {
  return (h + s.inner - 1) / s.inner * s.inner;
}

__host__ __device__ inline TcSmem tc_smem_layout(uint32_t h, const TcShape &s) {
  TcSmem L{};
  uint32_t o = 0;
  const uint32_t brow = tc_qrow(h, s) * 2;
  L.raw = tc_take(o, kTcScoreWarps * s.Rs * kTcSlab * s.inner, 1024);
  L.b = tc_take(o, s.Bs * s.N * brow, 128);
  L.qids = tc_take(o, s.Bs * s.N * 4, 16);
  L.qbv = tc_take(o, s.Bs * s.N * 4, 16);
  L.desc = tc_take(o, kTcMaxBufs * kTcDesc, 16);
  L.bars = tc_take(o, (kTcScoreWarps * kTcMaxStages + 3 * kTcMaxBufs) * 8, 8);
  L.err = tc_take(o, 4, 4);
  L.rcount = tc_take(o, 4 * 4, 4);
  L.total = (o + 127) / 128 * 128;
  return L;
}

// Rows a seed bound looks at unless set otherwise, for a query that probes few
// rows; one that probes many (65,536 by its nearest lists) looks at twice as many
// and scores 3 S instead of 2 S. A looser bound costs the ranking pass little where
// the candidates stay few, so there the seed's own time decides: 1,024 rows and
// 2 S take 88 us for 4096 queries at 1M x 1024 (S = 32), 2,048 and 3 S 127, for 2%
// fewer candidates. In long lists of tight clusters (10M, S = 64, 72 lists) they
// leave 2.4 times the candidates: 2.35 ms a search against 2.18.
inline uint32_t default_seed_rows(uint32_t S) { return std::max(1024u, 8 * std::min(S, 1u << 20)); }
// The shape for h ranking dimensions over rows of dc bytes, or false when h
// does not suit the pass (the caller then uses the CUDA-core pass).
bool rank_tc_plan(uint32_t h, uint32_t dc, bool rotated, TcShape *s);
// One CTA per SM walks an equal share of all tiles.
int rank_tc(const RankTcArgs &A, const uint8_t *xhi, uint32_t npts, const TcShape &s,
            cudaStream_t st);
// Per query, an upper bound on its final S-th ranking l2 over h <= 2048
// dimensions, from the first `rows` rows (at most 4096) of its probed lists in
// probe order: as an l2 that no row it could keep exceeds, or as the bits of
// the distance value of the ranking l2 or of the exact one (h = dc).
enum class SeedBound { kRanking, kRankingKey, kExactKey };
int rank_seed(const uint8_t *xhi, const int64_t *xnorm, const uint8_t *qhi, const int64_t *qnorm,
              const uint32_t *probed, const uint32_t *qprobes, const uint32_t *list_off, uint32_t B,
              uint32_t p, uint32_t dc, uint32_t h, uint32_t S, uint32_t rows, SeedBound kind,
              DistScale scale, int32_t *bound, cudaStream_t st);
// Process-wide knobs of the pass (0 = default): the largest item width and
// the cost weight of the CTA split.
extern std::atomic<uint32_t> g_tc_width, g_tc_beta;
// The pass's bounded pipeline waits give up after this many cycles (0: the
// default of 4e9, about 2 s); a CTA that gives up is counted in stats[3].
extern std::atomic<unsigned long long> g_tc_wait;
// Candidate records of the pass, completed over dimensions [f, h) where they
// are partial, into per-query buffers of cap entries (distance bits, row);
// qcount counts the candidates of each query and *found all of them.
int rank_tc_bucket(const uint4 *rec, const uint32_t *rec_n, uint32_t rec_cap, uint32_t ctas,
                   const uint8_t *xhi, const uint8_t *qhi, const int2 *qcn, const int32_t *bound,
                   uint32_t dc, uint32_t f, uint32_t h, uint32_t *qcount, uint2 *qbuf, uint32_t cap,
                   DistScale scale, unsigned long long *found, cudaStream_t st);
// CTAs of rank_tc (one per SM).
uint32_t rank_tc_ctas();

}  // namespace kato
