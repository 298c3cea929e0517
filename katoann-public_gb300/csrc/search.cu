// The batched search pipeline, from a batch's queries to its results.
//
// Reference: Index::search_sq16_ranked_ (src/index.cpp:909-1128) and
// Index::search_sq16_full_ (:1131-1219), which scan each probed list once for
// all the queries that probe it (:998-1044). Here the prefix and high-byte
// rankings run on the tensor cores (rank_tc.cu); rank_kernel below, for the
// full ranking and shapes that pass does not take, scores on the CUDA cores:
// each CTA takes one list and up to kQG of its queries, stages the list's rows
// in shared memory tile by tile and keeps, per query, the best S candidates by
// (distance, id) in shared memory. Selection by (distance, id)
// is the reference's Selection::kLocal result (:101-135 then :1063-1069) and
// its kThreshold result wherever that has no tie on the survivor boundary.
#include <algorithm>
#include <atomic>
#include <vector>

#include <cuda_fp16.h>

#include "finish.cuh"
#include "invert.cuh"
#include "kcommon.cuh"
#include "probe.cuh"
#include "rank_tc.cuh"

namespace kato {

thread_local uint32_t g_launches = 0;  // kernel launches of the last search pass
// Entries per query of the tensor-core ranking pass's candidate buffer.
std::atomic<uint32_t> g_candidate_cap{32768};
// Rows a query's seed bound looks at (0: default_seed_rows).
std::atomic<uint32_t> g_seed_rows{0};

namespace {

constexpr int kQG = 16;            // queries per ranking work item
constexpr int kRT = 32;            // list rows per ranking tile: two per thread
constexpr uint32_t kChunk = 512;   // bytes of a row staged at once
// Rows of a list per CTA: lists are skewed, and with a CTA for a whole list the
// longest one was the kernel's time (200,000 rows in 512 lists: 0.27 ms).
constexpr uint32_t kSplitRows = 256;
constexpr uint32_t kMaxParts = 65535;  // CTAs of a list: the grid's second dimension
// Candidate places (8 bytes) up to which the lists are split: 128 MiB. Exact
// ranking at 2M x 128, 512 lists, with 32 MiB, 128 MiB and 2 GiB: 256 queries of
// 24 lists with k = 100 1.52, 1.04, 1.04 ms, 1024 of them 5.0, 2.7, 2.6 ms; 4096 of
// 64 lists with k = 10 17.2, 16.5, 18.2 ms.
constexpr uint64_t kSplitEntries = 1ull << 24;
constexpr uint32_t kSelMax = 256;  // largest per-slot S kept in shared memory
constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr int kThreads = 256;
constexpr uint32_t kSortMax = 4096;

// ------------------------------------------------------------- ranking pass
struct RankArgs {
  const uint8_t *xhi, *xlo;
  const int64_t *xnorm;  // per row norm matching the mode
  const uint32_t *ids, *list_off;
  const uint8_t *qhi, *qlo;
  const int64_t *qnorm;  // per query norm matching the mode
  const Work *work;
  const uint32_t *woff_total;
  const uint32_t *off, *entries;
  uint32_t dc, dims, nprobe, S, SC;
  const uint32_t *bound;  // per query: no candidate with a larger key is needed (null: none)
  // selecting: per query, `cap` entries of (key, row), of which qcount are
  // used; otherwise SC of each probe slot (query * nprobe + rank), in row order
  uint2 *slots;
  uint32_t *qcount, cap, split;  // split: rows per CTA
  DistScale scale;
};

__host__ __device__ inline size_t rank_smem_bytes(int planes, bool select, uint32_t dims,
                                                  uint32_t S) {
  const uint32_t qw = dims / 4 + 1, kch = dims < kChunk ? dims : kChunk, rw = kch / 4 + 1;
  size_t b = static_cast<size_t>(planes) * kQG * qw * 4 + static_cast<size_t>(planes) * kRT * rw * 4;
  b += kRT * 4 + 3 * kQG * 4;           // sids, ccount, bcount, query ids
  b = (b + 15) / 16 * 16;
  b += kQG * 12;                        // query norms and bounds
  if (select) b += static_cast<size_t>(kQG) * S * 12 + static_cast<size_t>(kQG) * kRT * 12;
  return b;
}

// kFull: four products over dc (Ranking::kFull); otherwise high bytes over
// `dims` (kHighBytes: dims = dc; kPrefix: dims = head dims).
// kSelect: keep the best S per (query, list) in shared memory (S <= kSelMax);
// otherwise write every candidate to its slot (slot capacity >= list size).
template <bool kFull, bool kSelect>
__global__ void __launch_bounds__(kThreads) rank_kernel(RankArgs A) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t w = blockIdx.x;
  if (w >= *A.woff_total) return;
  const Work wk = A.work[w];
  const uint32_t c = wk.list;
  const uint32_t e0 = A.off[c] + wk.first;
  const uint32_t ne = min(static_cast<uint32_t>(kQG), A.off[c + 1] - e0);
  const uint32_t r0 = A.list_off[c], all_rows = A.list_off[c + 1] - r0;
  const uint32_t first = blockIdx.y * A.split, nrows = min(all_rows, first + A.split);
  if (first >= all_rows && (kSelect || blockIdx.y)) return;
  const uint32_t dims = A.dims, qw = dims / 4 + 1;
  const uint32_t kch = min(dims, kChunk), rw = kch / 4 + 1;
  constexpr int kPlanes = kFull ? 2 : 1;
  const uint32_t S = A.S;

  uint32_t *sq = reinterpret_cast<uint32_t *>(smem);   // [planes][kQG][qw]
  uint32_t *sr = sq + kPlanes * kQG * qw;              // [planes][kRT][rw]
  uint32_t *sids = sr + kPlanes * kRT * rw;            // [kRT]
  uint32_t *ccount = sids + kRT;                       // [kQG]
  uint32_t *bcount = ccount + kQG;                     // [kQG]
  uint32_t *sslot = bcount + kQG;                      // [kQG]
  size_t off = (reinterpret_cast<unsigned char *>(sslot + kQG) - smem + 15) / 16 * 16;
  int64_t *sqn = reinterpret_cast<int64_t *>(smem + off);                      // [kQG]
  uint32_t *sbound = reinterpret_cast<uint32_t *>(sqn + kQG);                  // [kQG]
  unsigned long long *bkid = reinterpret_cast<unsigned long long *>(sbound + kQG);  // [kQG][S]
  unsigned long long *ckid = bkid + (kSelect ? kQG * S : 0);                   // [kQG][kRT]
  uint32_t *brow = reinterpret_cast<uint32_t *>(ckid + (kSelect ? kQG * kRT : 0));  // [kQG][S]
  uint32_t *crow = brow + (kSelect ? kQG * S : 0);                             // [kQG][kRT]

  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int j = t & 15, rr = t >> 4;
  if (t < kQG) {
    ccount[t] = 0;
    bcount[t] = 0;
    sslot[t] = t < static_cast<int>(ne) ? A.entries[e0 + t] : 0;
  }
  __syncthreads();
  if (t < static_cast<int>(ne)) {
    const uint32_t q = sslot[t] / A.nprobe;
    sqn[t] = A.qnorm[q];
    sbound[t] = A.bound ? A.bound[q] : kEmpty;
  }
  // Stage the queries' bytes (16-byte loads; dims is a multiple of 64).
  const uint32_t v16 = dims / 16;
  for (uint32_t idx = t; idx < ne * v16 * kPlanes; idx += kThreads) {
    const uint32_t pl = idx / (ne * v16), rem = idx % (ne * v16);
    const uint32_t jj = rem / v16, v = rem % v16;
    const uint32_t q = sslot[jj] / A.nprobe;
    const uint8_t *src = (pl == 0 ? A.qhi : A.qlo) + static_cast<size_t>(q) * A.dc + v * 16;
    const uint4 x = *reinterpret_cast<const uint4 *>(src);
    uint32_t *dst = sq + (pl * kQG + jj) * qw + v * 4;
    dst[0] = x.x; dst[1] = x.y; dst[2] = x.z; dst[3] = x.w;
  }
  // Slots of rows past the list end are padding (store-all mode writes every row).
  if (!kSelect && blockIdx.y == 0) {
    for (uint32_t idx = t; idx < ne * (A.SC - min(all_rows, A.SC)); idx += kThreads) {
      const uint32_t jj = idx / (A.SC - all_rows), pos = all_rows + idx % (A.SC - all_rows);
      A.slots[static_cast<size_t>(sslot[jj]) * A.SC + pos] = make_uint2(kEmpty, 0);
    }
  }
  __syncthreads();

  for (uint32_t rt = first; rt < nrows; rt += kRT) {
    const uint32_t nr = min(static_cast<uint32_t>(kRT), nrows - rt);
    uint32_t hh[2] = {0, 0}, mx[2] = {0, 0}, ll[2] = {0, 0};  // rows rr and rr + 16
    for (uint32_t k0 = 0; k0 < dims; k0 += kch) {
      const uint32_t kc = min(kch, dims - k0), c16 = kc / 16;
      __syncthreads();
      for (uint32_t idx = t; idx < nr * c16 * kPlanes; idx += kThreads) {
        const uint32_t pl = idx / (nr * c16), rem = idx % (nr * c16);
        const uint32_t i = rem / c16, v = rem % c16;
        const uint8_t *src =
            (pl == 0 ? A.xhi : A.xlo) + static_cast<size_t>(r0 + rt + i) * A.dc + k0 + v * 16;
        const uint4 x = *reinterpret_cast<const uint4 *>(src);
        uint32_t *dst = sr + (pl * kRT + i) * rw + v * 4;
        dst[0] = x.x; dst[1] = x.y; dst[2] = x.z; dst[3] = x.w;
      }
      if (k0 == 0 && t < static_cast<int>(nr)) sids[t] = A.ids[r0 + rt + t];
      __syncthreads();
      if (j < static_cast<int>(ne) && rr < static_cast<int>(nr)) {
        const uint32_t *qa = sq + j * qw + k0 / 4;
        const uint32_t *xa = sr + rr * rw, *xa2 = xa + 16 * rw;  // (rows past nr: stale, unused)
        const uint32_t nw = kc / 4;
        if (kFull) {
          const uint32_t *qb = sq + (kQG + j) * qw + k0 / 4;
          const uint32_t *xb = sr + (kRT + rr) * rw, *xb2 = xb + 16 * rw;
#pragma unroll 8
          for (uint32_t u = 0; u < nw; ++u) {
            const uint32_t ah = qa[u], al = qb[u];
            const uint32_t bh = xa[u], bl = xb[u], ch = xa2[u], cl = xb2[u];
            hh[0] = dp4(ah, bh, hh[0]);
            mx[0] = dp4(ah, bl, mx[0]);
            mx[0] = dp4(al, bh, mx[0]);
            ll[0] = dp4(al, bl, ll[0]);
            hh[1] = dp4(ah, ch, hh[1]);
            mx[1] = dp4(ah, cl, mx[1]);
            mx[1] = dp4(al, ch, mx[1]);
            ll[1] = dp4(al, cl, ll[1]);
          }
        } else {
#pragma unroll 8
          for (uint32_t u = 0; u < nw; ++u) {
            hh[0] = dp4(qa[u], xa[u], hh[0]);
            hh[1] = dp4(qa[u], xa2[u], hh[1]);
          }
        }
      }
    }
    // The candidates of rows rr and rr + 16 with query j. The seed bound leaves
    // few lists any: merging every tile's candidates took a fifth of the kernel
    bool found = false;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = rr + 16 * i;
      if (j >= static_cast<int>(ne) || r >= static_cast<int>(nr)) continue;
      const uint32_t row = r0 + rt + r;
      const int64_t dot = kFull ? static_cast<int64_t>((static_cast<uint64_t>(hh[i]) << 16) +
                                                       (static_cast<uint64_t>(mx[i]) << 8) + ll[i])
                                : static_cast<int64_t>(hh[i]);
      const uint32_t key = __float_as_uint(dist_value(sqn[j] + A.xnorm[row] - 2 * dot, A.scale));
      if (kSelect) {
        const unsigned long long kid = (static_cast<unsigned long long>(key) << 32) | sids[r];
        const unsigned long long thr = bcount[j] == S ? bkid[j * S + S - 1] : ~0ull;
        if (kid < thr && key <= sbound[j]) {
          found = true;
          const uint32_t pos = atomicAdd(&ccount[j], 1u);
          ckid[j * kRT + pos] = kid;
          crow[j * kRT + pos] = row;
        }
      } else {
        A.slots[static_cast<size_t>(sslot[j]) * A.SC + rt + r] = make_uint2(key, row);
      }
    }
    if (kSelect && __syncthreads_or(found)) {
      // Merge each query's new candidates (at most kRT, unsorted) into its
      // sorted best list: one warp per query.
      for (int jj = warp; jj < static_cast<int>(ne); jj += kThreads / 32) {
        const uint32_t nc = ccount[jj];
        if (nc == 0) continue;
        const uint32_t nb = bcount[jj];
        unsigned long long *B = bkid + jj * S;
        uint32_t *Br = brow + jj * S;
        const unsigned long long ck = lane < static_cast<int>(nc) ? ckid[jj * kRT + lane] : ~0ull;
        const uint32_t cr = lane < static_cast<int>(nc) ? crow[jj * kRT + lane] : 0;
        // rank of this candidate among the candidates (ties by lane)
        uint32_t crank = 0;
        for (uint32_t i = 0; i < nc; ++i) {
          const unsigned long long o = __shfl_sync(0xffffffffu, ck, i);
          crank += (o < ck) || (o == ck && static_cast<int>(i) < lane);
        }
        // number of best entries <= candidate (upper bound)
        uint32_t lo = 0, hi = nb;
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (B[mid] <= ck) lo = mid + 1;
          else hi = mid;
        }
        const uint32_t cpos = lo + crank;
        // new index of each old entry
        constexpr int kPer = kSelMax / 32;
        unsigned long long okid[kPer];
        uint32_t orow[kPer], onew[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          const uint32_t b = lane + 32 * u;
          okid[u] = b < nb ? B[b] : ~0ull;
          orow[u] = b < nb ? Br[b] : 0;
          onew[u] = b < nb ? b : 0xFFFFFFFFu;
        }
        for (uint32_t i = 0; i < nc; ++i) {
          const unsigned long long o = __shfl_sync(0xffffffffu, ck, i);
#pragma unroll
          for (int u = 0; u < kPer; ++u) onew[u] += (onew[u] != 0xFFFFFFFFu && o < okid[u]);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kPer; ++u)
          if (onew[u] < S) {
            B[onew[u]] = okid[u];
            Br[onew[u]] = orow[u];
          }
        if (lane < static_cast<int>(nc) && cpos < S) {
          B[cpos] = ck;
          Br[cpos] = cr;
        }
        __syncwarp();
        if (lane == 0) {
          bcount[jj] = min(S, nb + nc);
          ccount[jj] = 0;
        }
      }
      __syncthreads();
    }
  }
  if (kSelect) {
    // append what was kept to the queries' candidates
    __syncthreads();
    if (t < static_cast<int>(ne)) ccount[t] = bcount[t] ? atomicAdd(&A.qcount[sslot[t] / A.nprobe], bcount[t]) : 0;
    __syncthreads();
    for (uint32_t idx = t; idx < ne * S; idx += kThreads) {
      const uint32_t jj = idx / S, i = idx % S;
      if (i < bcount[jj])
        A.slots[static_cast<size_t>(sslot[jj] / A.nprobe) * A.cap + ccount[jj] + i] =
            make_uint2(static_cast<uint32_t>(bkid[jj * S + i] >> 32), brow[jj * S + i]);
    }
  }
}

}  // namespace

// ------------------------------------------------------------ orchestration
int rotate_rows(const float *in, uint32_t nrows, uint32_t d, const float *rot, float *out,
                cudaStream_t st);
int sq16_tiles(const uint8_t *qhi, const uint8_t *qlo, const uint8_t *xhi, const uint8_t *xlo,
               const int64_t *qn, const int64_t *xn, double step_sq, uint32_t m, uint32_t n,
               uint32_t dims, uint32_t qstride, uint32_t xstride, float *out, bool full,
               cudaStream_t st);
bool coarse_tc_ok(uint32_t dc);
int coarse_tc(const __half *ch, const __half *cl, const int64_t *cterm, uint32_t n, const __half *qh,
              const __half *ql, const int64_t *qterm, uint32_t m, uint32_t dc, double step_sq,
              float *out, uint32_t *timeouts, unsigned long long *prof, cudaStream_t st);
size_t rotate_scratch_bytes(uint32_t nrows, uint32_t d);
int rotate_rows_kmajor(const float *in, uint32_t nrows, uint32_t d, const float *rot,
                       const float *rot_kmajor, void *scratch, float *out, uint32_t *timeouts,
                       uint32_t *launches, cudaStream_t st);
int select_topp_ex(const float *dists, uint32_t nq, uint32_t n, uint32_t p, uint32_t stride,
                   uint32_t *probed, uint32_t *cnt, unsigned long long *tie_count,
                   const uint32_t *only, uint32_t only_above, cudaStream_t st);

// Per pass: the KATO_PHASES + 1 phase boundaries, then a start and an end
// event around each timed kernel (KATO_TIMED_KERNELS: the query rotation,
// coarse_tc_kernel, rank_tc_kernel).
constexpr uint32_t kTimerStride = KATO_PHASES + 1 + 2 * KATO_TIMED_KERNELS;

struct PhaseTimer {
  std::vector<cudaEvent_t> ev;  // kTimerStride per pass
  std::vector<uint8_t> kdone;   // per pass: the kernels whose two events were recorded
  uint32_t max_passes = 0, used = 0;
  float kms[KATO_TIMED_KERNELS] = {};      // of the passes the last read summed
  uint32_t kn[KATO_TIMED_KERNELS] = {};
};

static void mark(PhaseTimer *t, uint32_t phase, cudaStream_t st) {
  if (!t || t->used >= t->max_passes) return;
  cudaEventRecord(t->ev[t->used * kTimerStride + phase], st);
}

static void kmark(PhaseTimer *t, uint32_t kernel, bool end, cudaStream_t st) {
  if (!t || t->used >= t->max_passes) return;
  cudaEventRecord(t->ev[t->used * kTimerStride + KATO_PHASES + 1 + 2 * kernel + end], st);
  if (end) t->kdone[t->used] |= static_cast<uint8_t>(1u << kernel);
}

struct Plan {
  uint32_t B, k, p, S, SC, dims;
  int ranking;
  bool select;
  bool tc;                          // tensor-core ranking pass
  bool coarse_tc;                   // tensor-core coarse product
  TcShape tcs;
  uint32_t tcitems, cap, seed_rows, ctas, rec_cap, beta;
  uint32_t split, per_query;        // CUDA-core pass: rows per CTA, candidate entries per query
  bool cost;                        // the ranking CTAs split the slabs' cost, not their count
  size_t off_fq, off_qhi, off_qlo, off_qn, off_qhn, off_qh0, off_cd, off_probed, off_cnt, off_off,
      off_base, off_cur, off_work, off_ent, off_slots, off_stats,
      off_tcitems, off_tileoff, off_over, off_qcount, off_bound,
      off_rec, off_recn, off_qh16, off_ql16, off_qterm, off_rot,
      off_qprobes, off_z, off_qcn, off_qr16, off_share, total;
};

static size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// With `coarse_only` the plan ends with the selected lists (the feature pass):
// it has no candidates.
int make_plan(const katoann_gpu_index *ix, uint32_t B, uint32_t k, uint32_t p, int ranking,
              uint32_t survivors, Plan *P, bool coarse_only = false) {
  if (k == 0 || p == 0 || p > ix->nlist) return invalid("need k >= 1 and 1 <= nprobe <= nlist");
  if (ranking == KATO_RANK_PREFIX && ix->head_dims == 0)
    return invalid("prefix ranking needs the rotation file (.dimc)");
  if (ranking < 0 || ranking > 2) return invalid("unknown ranking");
  Plan &pl = *P;
  pl.B = B;
  pl.k = k;
  pl.p = p;
  pl.ranking = ranking;
  pl.S = ranking == KATO_RANK_FULL ? k : std::max(survivors, k);
  if (pl.S > kSortMax) return invalid("survivors (or k) above 4096 are not supported on the GPU");
  const uint32_t ml = std::max(ix->max_list, 1u);
  pl.SC = std::min(pl.S, ml);
  pl.select = pl.SC <= kSelMax;
  if (!pl.select) pl.SC = ml;
  pl.dims = ranking == KATO_RANK_PREFIX ? ix->head_dims : ix->dc;
  const uint32_t L = ix->nlist;
  const size_t bp = static_cast<size_t>(B) * p;
  const size_t wmax = std::min<size_t>(L, bp) + bp / kQG + 1;
  // tensor-core ranking: every query's candidates within its seed bound go
  // to a buffer of `cap` entries (an overflowing query is rescanned exactly)
  pl.cap = g_candidate_cap.load();
  pl.tc = ranking != KATO_RANK_FULL && pl.S <= pl.cap && rank_tc_plan(pl.dims, ix->dc, ix->rotated != 0, &pl.tcs);
  // rows per CTA of the CUDA-core pass: each of a list's parts keeps up to SC
  // candidates per query. Within kSplitEntries places for them the parts are as
  // short as they should be, beyond it so many as fit, and one per list at least.
  // The places set aside are those of the shortest parts up to that bound (not
  // those of the parts taken, which are fewer where a larger batch leaves fewer),
  // so that a workspace also serves any smaller batch, k and nprobe.
  const uint32_t least = std::max(kSplitRows, div_up(div_up(ml, kMaxParts), kRT) * kRT);
  const uint32_t most = pl.select ? div_up(ml, least) : 1;
  auto kept = [&](uint32_t parts) {  // of a query: never more than the lists' rows
    return p * std::min<uint64_t>(ml, static_cast<uint64_t>(pl.SC) * parts);
  };
  pl.split = least;
  if (pl.select && !pl.tc && B * kept(most) > kSplitEntries) {
    const uint64_t parts = std::max<uint64_t>(1, kSplitEntries / (static_cast<uint64_t>(B) * p * pl.SC));
    pl.split = std::max(least, div_up(div_up(ml, static_cast<uint32_t>(parts)), kRT) * kRT);
  }
  const uint64_t per_query = kept(pl.select ? div_up(ml, pl.split) : 1);
  if (!pl.tc && per_query >= (1ull << 32)) return invalid("too many candidates per query");
  pl.per_query = static_cast<uint32_t>(per_query);
  if (pl.tc) {
    pl.select = true;
    pl.SC = pl.S;
    const uint32_t sr = g_seed_rows.load();
    pl.seed_rows = sr ? std::max(sr, pl.S) : default_seed_rows(pl.S);
    pl.tcitems = static_cast<uint32_t>(bp / pl.tcs.N + std::min<size_t>(L, bp) + 1);
    // candidate records per CTA: room for 32 S per query of the batch, spread
    // over the CTAs (a CTA that runs out flags the queries it drops)
    pl.ctas = rank_tc_ctas();
    pl.rec_cap = static_cast<uint32_t>(
        std::max<size_t>(8192, static_cast<size_t>(B) * pl.S * 32 / pl.ctas));
    // the cost split, unless its 32-bit cost units could overflow
    pl.beta = g_tc_beta.load();
    const uint64_t worst = static_cast<uint64_t>(pl.tcitems) * div_up(ix->max_list, kTcSlab) *
                           (pl.beta ? 64 + static_cast<uint64_t>(pl.beta) * pl.tcs.N : 32);
    pl.cost = worst < (1ull << 31);
  } else {
    pl.ctas = 1;
    pl.rec_cap = 0;
  }
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += align256(bytes);
    return at;
  };
  pl.off_stats = take(48 * sizeof(unsigned long long));
  pl.off_fq = take(static_cast<size_t>(B) * ix->dim * 4);
  pl.off_qhi = take(static_cast<size_t>(B) * ix->dc);
  pl.off_qlo = take(static_cast<size_t>(B) * ix->dc);
  pl.off_qn = take(static_cast<size_t>(B) * 8);
  pl.off_qhn = take(static_cast<size_t>(B) * 8);
  pl.off_qh0 = take(static_cast<size_t>(B) * 8);
  pl.off_cd = take(static_cast<size_t>(B) * L * 4);
  pl.off_probed = take(bp * 4);
  pl.off_cnt = take(static_cast<size_t>(L) * 4);  // cleared together with over and qcount after it
  pl.off_over = take(4);
  pl.off_qcount = take(static_cast<size_t>(B) * 4);
  pl.off_off = take((static_cast<size_t>(L) + 1) * 4);
  pl.off_base = take(3 * (static_cast<size_t>(L) + 1) * 4);
  pl.off_cur = take(static_cast<size_t>(L) * 4);
  pl.off_work = take(wmax * sizeof(Work));
  pl.off_ent = take(bp * 4);
  const uint64_t entries = coarse_only ? 0
                           : pl.tc     ? static_cast<uint64_t>(B) * pl.cap
                                       : std::max(B * kept(1), std::min(B * kept(most), kSplitEntries));
  pl.off_slots = take(entries * sizeof(uint2));
  pl.off_share = take((static_cast<size_t>(pl.ctas) + 1) * sizeof(uint2));
  pl.off_tcitems = take(pl.tc ? (static_cast<size_t>(pl.tcitems) + 1) * sizeof(TcItem) : 16);
  pl.off_tileoff = take(pl.tc ? (static_cast<size_t>(pl.tcitems) + 1) * 4 : 16);
  pl.off_bound = take(static_cast<size_t>(B) * 4);
  pl.off_rec = take(pl.tc ? static_cast<size_t>(pl.ctas) * pl.rec_cap * 16 : 16);
  pl.off_recn = take(static_cast<size_t>(pl.ctas) * 4);
  pl.coarse_tc = ix->d_chi16 && ix->d_clo16 && ix->d_cterm && coarse_tc_ok(ix->dc);
  const bool planes = pl.coarse_tc || pl.tc;  // the queries' centred fp16 planes
  pl.off_qh16 = take(planes ? static_cast<size_t>(B) * ix->dc * 2 : 16);
  pl.off_ql16 = take(planes ? static_cast<size_t>(B) * ix->dc * 2 : 16);
  pl.off_qr16 = take(pl.tc ? static_cast<size_t>(B) * tc_qrow(pl.dims, pl.tcs) * 2 : 16);
  pl.off_qcn = take(planes ? static_cast<size_t>(B) * sizeof(int2) : 16);
  pl.off_qterm = take(static_cast<size_t>(B) * 8);
  pl.off_rot = take(ix->rotated ? rotate_scratch_bytes(B, ix->dim) : 16);
  pl.off_qprobes = take(static_cast<size_t>(B) * 4);
  pl.off_z = take(static_cast<size_t>(B) * KATO_PROBE_FEATURES * 4);
  pl.total = o;
  return KATO_OK;
}

// Rotation, quantization, coarse product and top-p1 selection of nq queries
// (phases 0-2): leaves the query planes, the coarse distances (cd) and each
// query's p1 nearest lists in order (probed, rows pl.p apart) in the
// workspace.
int coarse_pass(const katoann_gpu_index *ix, const Plan &pl, const float *queries, uint32_t nq,
                unsigned char *ws, uint32_t p1, uint32_t *cnt, cudaStream_t st, PhaseTimer *tm) {
  int rc;
  const uint32_t L = ix->nlist, p = pl.p, dc = ix->dc;
  float *fq = reinterpret_cast<float *>(ws + pl.off_fq);
  uint8_t *qhi = ws + pl.off_qhi, *qlo = ws + pl.off_qlo;
  int64_t *qn = reinterpret_cast<int64_t *>(ws + pl.off_qn);
  int64_t *qhn = reinterpret_cast<int64_t *>(ws + pl.off_qhn);
  int64_t *qh0 = reinterpret_cast<int64_t *>(ws + pl.off_qh0);
  float *cd = reinterpret_cast<float *>(ws + pl.off_cd);
  uint32_t *probed = reinterpret_cast<uint32_t *>(ws + pl.off_probed);
  unsigned long long *stats = reinterpret_cast<unsigned long long *>(ws + pl.off_stats);

  mark(tm, 0, st);
  // 1. rotation and quantization of the queries (src/index.cpp:895-899, :917-943)
  const float *src = queries;
  if (ix->rotated) {
    kmark(tm, 0, false, st);
    if ((rc = rotate_rows_kmajor(queries, nq, ix->dim, ix->d_rotation, ix->d_rotation_t,
                                 ws + pl.off_rot, fq, reinterpret_cast<uint32_t *>(stats + 3),
                                 &g_launches, st)))
      return rc;
    kmark(tm, 0, true, st);
    src = fq;
  }
  // the queries' planes, for the exact distances and both tensor-core passes;
  // the counts of the inversion and of the candidates start at 0
  __half *qh16 = reinterpret_cast<__half *>(ws + pl.off_qh16);
  __half *ql16 = reinterpret_cast<__half *>(ws + pl.off_ql16);
  int64_t *qterm = reinterpret_cast<int64_t *>(ws + pl.off_qterm);
  QueryPlanes P{qhi, qlo, qn, qhn, qh0, dc, ix->head_dims, nullptr, nullptr, nullptr,
                reinterpret_cast<uint32_t *>(ws + pl.off_cnt),
                static_cast<uint32_t>((pl.off_qcount - pl.off_cnt) / 4 + pl.B)};
  RankRows rr{};
  if (pl.coarse_tc || pl.tc) P.hi16 = qh16, P.lo16 = ql16, P.term = qterm;
  if (pl.tc)
    rr = RankRows{reinterpret_cast<__half *>(ws + pl.off_qr16),
                  reinterpret_cast<int2 *>(ws + pl.off_qcn), pl.tcs.f, pl.dims,
                  tc_qrow(pl.dims, pl.tcs), pl.tcs.centred};
  if ((rc = query_planes(src, nq, ix->dim, ix->lo, ix->inv_step, P, rr, st))) return rc;
  g_launches += 1 + 2;  // planes, coarse, select
  mark(tm, 1, st);
  // 2. coarse product and top-nprobe (:846-877)
  if (pl.coarse_tc) {
    kmark(tm, 1, false, st);
    if ((rc = coarse_tc(reinterpret_cast<const __half *>(ix->d_chi16),
                        reinterpret_cast<const __half *>(ix->d_clo16), ix->d_cterm, L, qh16, ql16,
                        qterm, nq, dc, ix->step_sq, cd, reinterpret_cast<uint32_t *>(stats + 3),
                        stats + 32, st)))
      return rc;
    kmark(tm, 1, true, st);
  } else if ((rc = sq16_tiles(qhi, qlo, ix->d_chi, ix->d_clo, qn, ix->d_cnorm, ix->step_sq, nq, L,
                              dc, dc, dc, cd, true, st))) {
    return rc;
  }
  mark(tm, 2, st);
  if ((rc = select_topp_ex(cd, nq, L, p1, p, probed, cnt, stats + 0, nullptr, 0, st))) return rc;
  mark(tm, 3, st);
  return KATO_OK;
}

int search_pass(const katoann_gpu_index *ix, const Plan &pl, const float *queries, uint32_t nq,
                unsigned char *ws, uint32_t *out_ids, float *out_dists, const Budget &bud,
                cudaStream_t st, PhaseTimer *tm) {
  int rc;
  const uint32_t L = ix->nlist, p = pl.p, dc = ix->dc;
  uint8_t *qhi = ws + pl.off_qhi, *qlo = ws + pl.off_qlo;
  int64_t *qn = reinterpret_cast<int64_t *>(ws + pl.off_qn);
  int64_t *qhn = reinterpret_cast<int64_t *>(ws + pl.off_qhn);
  int64_t *qh0 = reinterpret_cast<int64_t *>(ws + pl.off_qh0);
  float *cd = reinterpret_cast<float *>(ws + pl.off_cd);
  uint32_t *probed = reinterpret_cast<uint32_t *>(ws + pl.off_probed);
  uint32_t *cnt = reinterpret_cast<uint32_t *>(ws + pl.off_cnt);
  uint32_t *off = reinterpret_cast<uint32_t *>(ws + pl.off_off);
  uint32_t *base = reinterpret_cast<uint32_t *>(ws + pl.off_base);
  uint32_t *cur = reinterpret_cast<uint32_t *>(ws + pl.off_cur);
  Work *work = reinterpret_cast<Work *>(ws + pl.off_work);
  uint32_t *ent = reinterpret_cast<uint32_t *>(ws + pl.off_ent);
  uint2 *slots = reinterpret_cast<uint2 *>(ws + pl.off_slots);
  unsigned long long *stats = reinterpret_cast<unsigned long long *>(ws + pl.off_stats);

  // with a model, the selection first goes as deep as its features and then,
  // for the queries whose budget is deeper, to the cap
  const bool model = bud.model && !bud.nprobe_in;
  const uint32_t p1 = model ? std::min(p, bud.model->depth) : p;
  // without budgets the selection counts the inversion's lists on the way
  const bool counted = !bud.active();
  if ((rc = coarse_pass(ix, pl, queries, nq, ws, p1, counted ? cnt : nullptr, st, tm))) return rc;
  // 2'. per-query budgets: given, or from the model over the coarse distances
  uint32_t *qprobes = nullptr;
  if (bud.active()) {
    qprobes = reinterpret_cast<uint32_t *>(ws + pl.off_qprobes);
    if (bud.nprobe_in) {
      if ((rc = clamp_budget(bud.nprobe_in, nq, bud.cap, qprobes, st))) return rc;
      ++g_launches;
    } else {
      float *z = reinterpret_cast<float *>(ws + pl.off_z);
      if ((rc = probe_features(cd, L, probed, p, bud.model->d_rank, nq, z, st))) return rc;
      if ((rc = probe_budget(*bud.model, z, nq, bud.cap, nullptr, qprobes, st))) return rc;
      g_launches += 2;
      if (p1 < p) {
        if ((rc = select_topp_ex(cd, nq, L, p, p, probed, nullptr, nullptr, qprobes, p1, st))) return rc;
        ++g_launches;
      }
    }
    if (bud.nprobe_out)
      KATO_CUDA(cudaMemcpyAsync(bud.nprobe_out, qprobes, static_cast<size_t>(nq) * 4,
                                cudaMemcpyDeviceToDevice, st));
  } else if (bud.nprobe_out) {
    if ((rc = clamp_budget(nullptr, nq, p, bud.nprobe_out, st))) return rc;  // all p
    ++g_launches;
  }
  mark(tm, 4, st);
  // 3. inversion (:403-412)
  InvertArgs I{};
  I.probed = probed;
  I.qprobes = qprobes;
  I.B = nq;
  I.p = p;
  I.L = L;
  I.N = pl.tc ? pl.tcs.N : kQG;
  I.list_off = ix->d_list_off;
  I.cnt = cnt;
  I.off = off;
  I.cur = cur;
  I.base = base;
  I.entries = ent;
  I.work = work;
  if (pl.tc) {
    I.items = reinterpret_cast<TcItem *>(ws + pl.off_tcitems);
    I.tile_off = reinterpret_cast<uint32_t *>(ws + pl.off_tileoff);
    I.share = reinterpret_cast<uint2 *>(ws + pl.off_share);
    I.ctas = pl.ctas;
    I.beta = pl.beta;
    I.by_cost = pl.cost;
    I.tile_hist = stats + 40;
    I.tiles = stats + 4;
  }
  if ((rc = invert(I, counted, &g_launches, st))) return rc;
  mark(tm, 5, st);
  // (the CUDA-core pass that keeps every candidate has them in fixed slots)
  uint32_t *qcount = pl.select ? reinterpret_cast<uint32_t *>(ws + pl.off_qcount) : nullptr;
  const bool full = pl.ranking == KATO_RANK_FULL;
  const bool prefix_mode = pl.ranking == KATO_RANK_PREFIX;
  int32_t *bound = reinterpret_cast<int32_t *>(ws + pl.off_bound);
  const DistScale scale = make_dist_scale(ix->step_sq);
  const bool seeded = pl.select && !pl.tc && pl.dims <= 2048;
  if (seeded) {
    // seed bounds of the CUDA-core pass, over the same high bytes
    if ((rc = rank_seed(ix->d_hi, prefix_mode ? ix->d_headnorm : ix->d_hinorm, qhi,
                        prefix_mode ? qh0 : qhn, probed, qprobes, ix->d_list_off, nq, p, dc, pl.dims,
                        pl.S, default_seed_rows(pl.S),
                        full ? SeedBound::kExactKey : SeedBound::kRankingKey, scale, bound, st)))
      return rc;
    ++g_launches;
  }
  if (!pl.tc) mark(tm, 6, st);
  if (pl.tc) {
    // 4'. ranking pass on the tensor cores: seed bounds, work items, the
    // scan, and the exact rescan of any query whose buffer overflowed
    uint4 *rec = reinterpret_cast<uint4 *>(ws + pl.off_rec);
    uint32_t *rec_n = reinterpret_cast<uint32_t *>(ws + pl.off_recn);
    const int64_t *xnorm = prefix_mode ? ix->d_headnorm : ix->d_hinorm;
    const int64_t *qnorm = prefix_mode ? qh0 : qhn;
    if ((rc = rank_seed(ix->d_hi, xnorm, qhi, qnorm, probed, qprobes, ix->d_list_off, nq, p, dc,
                        pl.dims, pl.S, pl.seed_rows, SeedBound::kRanking, scale, bound, st)))
      return rc;
    mark(tm, 6, st);
    RankTcArgs T{};
    T.qr16 = reinterpret_cast<const __half *>(ws + pl.off_qr16);
    T.qcn = reinterpret_cast<const int2 *>(ws + pl.off_qcn);
    T.entries = ent;
    T.items = I.items;
    T.tile_off = I.tile_off;
    T.share = I.share;
    T.bound = bound;
    T.qcount = qcount;
    T.rec = rec;
    T.rec_n = rec_n;
    T.rec_cap = pl.rec_cap;
    T.timeouts = reinterpret_cast<uint32_t *>(stats + 3);
    T.prof = stats + 16;
    T.dc = dc;
    T.h = pl.dims;
    T.f = pl.tcs.f;
    T.nprobe = p;
    T.wait = g_tc_wait.load() ? static_cast<long long>(g_tc_wait.load()) : 4000000000ll;
    kmark(tm, 2, false, st);
    if ((rc = rank_tc(T, ix->d_hi, ix->npts, pl.tcs, st))) return rc;
    kmark(tm, 2, true, st);
    if ((rc = rank_tc_bucket(rec, rec_n, pl.rec_cap, pl.ctas, ix->d_hi, qhi, T.qcn, bound, dc,
                             pl.tcs.f, pl.dims, qcount, slots, pl.cap, scale, stats + 5, st)))
      return rc;
    g_launches += 3;  // seed, scan, bucket
  }
  // 4. ranking pass (:998-1044 / :1167-1204)
  RankArgs A{};
  A.xhi = ix->d_hi;
  A.xlo = ix->d_lo;
  A.xnorm = full ? ix->d_norm : (pl.ranking == KATO_RANK_PREFIX ? ix->d_headnorm : ix->d_hinorm);
  A.ids = ix->d_ids;
  A.list_off = ix->d_list_off;
  A.qhi = qhi;
  A.qlo = qlo;
  A.qnorm = full ? qn : (pl.ranking == KATO_RANK_PREFIX ? qh0 : qhn);
  A.work = work;
  A.woff_total = base + L;
  A.off = off;
  A.entries = ent;
  A.dc = dc;
  A.dims = pl.dims;
  A.nprobe = p;
  A.S = pl.SC;  // a slot never holds more than min(S, largest list) candidates
  A.SC = pl.SC;
  A.bound = seeded ? reinterpret_cast<const uint32_t *>(bound) : nullptr;
  A.slots = slots;
  A.qcount = reinterpret_cast<uint32_t *>(ws + pl.off_qcount);
  A.cap = pl.per_query;
  A.split = pl.split;
  A.scale = scale;
  const size_t bp = static_cast<size_t>(nq) * p;
  const dim3 grid(static_cast<uint32_t>(std::min<size_t>(L, bp) + bp / kQG + 1),
                  std::max(1u, div_up(ix->max_list, pl.split)));
  const size_t smem = rank_smem_bytes(full ? 2 : 1, pl.select, pl.dims, pl.SC);
  if (!pl.tc && smem > 227 * 1024) return invalid("ranking tile does not fit in shared memory");
  auto launch = [&](auto kern) -> int {
    if (const int rc2 = smem_limit(reinterpret_cast<const void *>(kern), static_cast<int>(smem),
                                   "rank_kernel shared memory"))
      return rc2;
    kato::launch(kern, grid, kThreads, smem, st, A);
    KATO_LAUNCHED("rank_kernel");
    return KATO_OK;
  };
  if (!pl.tc) {
    if (full) rc = pl.select ? launch(rank_kernel<true, true>) : launch(rank_kernel<true, false>);
    else rc = pl.select ? launch(rank_kernel<false, true>) : launch(rank_kernel<false, false>);
    if (rc) return rc;
    ++g_launches;
  }
  mark(tm, 7, st);
  // 5. the best of the slot lists: of the exact distances the top-k (:1205-1218),
  // of the ranking distances the survivors, their exact distances and the
  // top-k (:1058-1125)
  if (full) {
    rc = merge_topk(slots, pl.per_query, pl.SC, qcount, qprobes, ix->d_ids, nq, pl.k, out_ids, out_dists,
                    stats + 1, st);
  } else {
    FinishArgs F{};
    F.slots = slots;
    F.per_query = pl.tc ? pl.cap : pl.per_query;
    F.per_probe = pl.SC;
    F.qcount = qcount;
    F.qprobes = qprobes;
    F.qhi = qhi;
    F.qlo = qlo;
    F.qnorm = qn;
    F.xhi = ix->d_hi;
    F.xlo = ix->d_lo;
    F.xnorm = ix->d_norm;
    F.ids = ix->d_ids;
    F.npts = ix->npts;
    F.dc = dc;
    F.S = pl.S;
    F.k = pl.k;
    F.scale = scale;
    F.out_ids = out_ids;
    F.out_dists = out_dists;
    F.ties = stats + 1;
    F.rescans = stats + 6;
    if (pl.tc) {
      F.rank_xnorm = prefix_mode ? ix->d_headnorm : ix->d_hinorm;
      F.rank_qnorm = prefix_mode ? qh0 : qhn;
      F.probed = probed;
      F.list_off = ix->d_list_off;
      F.h = pl.dims;
      F.nprobe = p;
      if (static_cast<uint64_t>(p) * ix->max_list > pl.cap) {
        // a buffer can overflow (the coarse product's terms and distances have
        // been read)
        F.over = reinterpret_cast<uint32_t *>(bound);
        F.over_key = reinterpret_cast<unsigned long long *>(ws + pl.off_qterm);
        F.over_list = reinterpret_cast<uint32_t *>(cd);
        F.over_n = reinterpret_cast<uint32_t *>(ws + pl.off_over);
        if ((rc = rescan_overflows(F, qcount, nq, st))) return rc;
        g_launches += 2;
      }
    }
    mark(tm, 8, st);  // the survivor merge is part of the refinement kernel
    rc = finish(F, nq, st);
  }
  if (rc) return rc;
  ++g_launches;
  if (full) mark(tm, 8, st);
  mark(tm, 9, st);
  if (tm && tm->used < tm->max_passes) ++tm->used;
  return KATO_OK;
}

int search(const katoann_gpu_index *ix, const float *queries, uint32_t nq, uint32_t k, uint32_t p,
           int ranking, uint32_t survivors, uint32_t max_batch, void *ws, size_t ws_bytes,
           uint32_t *out_ids, float *out_dists, const Budget &budget, cudaStream_t st,
           void *timer) {
  if (nq == 0) return KATO_OK;
  if (max_batch == 0) return invalid("max_batch must be positive");
  // with a budget, the selection depth covers the cap and the model's features
  uint32_t depth = p;
  if (budget.active()) {
    if (budget.model) {
      if (int rc = check_probe_model(*budget.model)) return rc;
      depth = std::max(depth, budget.model->depth);
    }
    if (depth > kSortMax) return invalid("a per-query nprobe needs nprobe (and model depth) <= 4096");
  }
  Plan pl{};
  int rc = make_plan(ix, std::min(nq, max_batch), k, depth, ranking, survivors, &pl);
  if (rc) return rc;
  if (ws_bytes < pl.total) {
    set_error("search workspace too small");
    return KATO_ENOMEM;
  }
  unsigned char *w = static_cast<unsigned char *>(ws);
  KATO_CUDA(cudaMemsetAsync(w + pl.off_stats, 0, 48 * sizeof(unsigned long long), st));
  g_launches = 0;
  const Chain chain;
  for (uint32_t q0 = 0; q0 < nq; q0 += max_batch) {
    const uint32_t b = std::min(max_batch, nq - q0);
    Budget bud = budget;
    bud.cap = p;
    if (bud.nprobe_in) bud.nprobe_in += q0;
    if (bud.nprobe_out) bud.nprobe_out += q0;
    if ((rc = search_pass(ix, pl, queries + static_cast<size_t>(q0) * ix->dim, b, w,
                          out_ids + static_cast<size_t>(q0) * k,
                          out_dists + static_cast<size_t>(q0) * k, bud, st,
                          static_cast<PhaseTimer *>(timer))))
      return rc;
  }
  return KATO_OK;
}

static int features_plan(const katoann_gpu_index *ix, uint32_t B, uint32_t depth, Plan *pl) {
  if (depth == 0 || depth > ix->nlist || depth > kSortMax)
    return invalid("feature depth must be 1 to min(nlist, 4096)");
  return make_plan(ix, B, 1, depth, KATO_RANK_FULL, 1, pl, true);
}

size_t features_workspace(const katoann_gpu_index *ix, uint32_t max_batch, uint32_t depth) {
  Plan pl{};
  return features_plan(ix, max_batch, depth, &pl) ? 0 : pl.total;
}

// The probe-budget features of nq queries (phases 0-2, then the feature
// kernel), max_batch at a time.
int probe_features_search(const katoann_gpu_index *ix, const float *queries, uint32_t nq,
                          const uint32_t *rank, uint32_t depth, uint32_t max_batch, void *ws,
                          size_t ws_bytes, float *z, cudaStream_t st) {
  if (nq == 0) return KATO_OK;
  if (max_batch == 0) return invalid("max_batch must be positive");
  if (!rank) return invalid("null feature ranks");
  Plan pl{};
  int rc = features_plan(ix, std::min(nq, max_batch), depth, &pl);
  if (rc) return rc;
  if (ws_bytes < pl.total) {
    set_error("feature workspace too small");
    return KATO_ENOMEM;
  }
  unsigned char *w = static_cast<unsigned char *>(ws);
  g_launches = 0;
  for (uint32_t q0 = 0; q0 < nq; q0 += max_batch) {
    const uint32_t b = std::min(max_batch, nq - q0);
    if ((rc = coarse_pass(ix, pl, queries + static_cast<size_t>(q0) * ix->dim, b, w, depth,
                          nullptr, st, nullptr)))
      return rc;
    if ((rc = probe_features(reinterpret_cast<float *>(w + pl.off_cd), ix->nlist,
                             reinterpret_cast<uint32_t *>(w + pl.off_probed), depth, rank, b,
                             z + static_cast<size_t>(q0) * KATO_PROBE_FEATURES, st)))
      return rc;
  }
  return KATO_OK;
}

uint32_t last_launches() { return g_launches; }

// --------------------------------------------------------------- autotune
// Times one search of these queries under every candidate setting of the
// ranking pass's knobs - seed rows, CTA split weight, item width - and keeps
// the fastest. The knobs change the work and its schedule, never a result.
int autotune(const katoann_gpu_index *ix, const float *queries, uint32_t nq, uint32_t k, uint32_t p,
             int ranking, uint32_t survivors, uint32_t max_batch, const Budget &budget, void *ws,
             size_t ws_bytes, cudaStream_t st, uint32_t *out) {
  if (nq == 0) return invalid("autotune needs queries");
  // the batch the search runs, once: the buffers of the results
  uint32_t *ids = nullptr;
  float *dists = nullptr;
  KATO_CUDA(cudaMalloc(&ids, static_cast<size_t>(nq) * k * 4));
  const cudaError_t e2 = cudaMalloc(&dists, static_cast<size_t>(nq) * k * 4);
  if (e2 != cudaSuccess) {
    cudaFree(ids);
    return cuda_status(e2, "autotune buffers");
  }
  cudaEvent_t a = nullptr, b = nullptr;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const uint32_t seed0 = g_seed_rows.load(), beta0 = g_tc_beta.load(), width0 = g_tc_width.load();
  float best = 1e30f;
  uint32_t bs = seed0, bb = beta0, bw = width0;
  int rc = KATO_OK;
  for (uint32_t seed : {1024u, 2048u, 4096u})
    for (uint32_t beta : {0u, 1u, 2u, 4u})
      for (uint32_t width : {0u, 32u}) {
        g_seed_rows = seed;
        g_tc_beta = beta;
        g_tc_width = width;
        int r = search(ix, queries, nq, k, p, ranking, survivors, max_batch, ws, ws_bytes, ids,
                       dists, budget, st, nullptr);
        if (r == KATO_ENOMEM) continue;  // this setting needs a larger workspace
        if (r) {
          rc = r;
          break;
        }
        cudaEventRecord(a, st);
        for (int rep = 0; rep < 3 && !r; ++rep)
          r = search(ix, queries, nq, k, p, ranking, survivors, max_batch, ws, ws_bytes, ids, dists,
                     budget, st, nullptr);
        cudaEventRecord(b, st);
        if (r || cudaEventSynchronize(b) != cudaSuccess) {
          rc = r ? r : cuda_status(cudaGetLastError(), "autotune");
          break;
        }
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        if (ms < best) {
          best = ms;
          bs = seed;
          bb = beta;
          bw = width;
        }
      }
  g_seed_rows = rc ? seed0 : bs;
  g_tc_beta = rc ? beta0 : bb;
  g_tc_width = rc ? width0 : bw;
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(ids);
  cudaFree(dists);
  if (rc) return rc;
  out[0] = bs;
  out[1] = bb;
  out[2] = bw;
  out[3] = static_cast<uint32_t>(best / 3 * 1000.0f);
  return KATO_OK;
}

// ------------------------------------------------------------ CUDA graphs
struct SearchGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  uint32_t launches = 0;
};

int search_capture(const katoann_gpu_index *ix, const float *queries, uint32_t nq, uint32_t k,
                   uint32_t p, int ranking, uint32_t survivors, uint32_t max_batch, void *ws,
                   size_t ws_bytes, uint32_t *out_ids, float *out_dists, const Budget &budget,
                   cudaStream_t st, void **out) {
  *out = nullptr;
  if (!st || st == cudaStreamLegacy || st == cudaStreamPerThread)
    return invalid("graph capture needs a created stream");
  KATO_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  const int rc = search(ix, queries, nq, k, p, ranking, survivors, max_batch, ws, ws_bytes,
                        out_ids, out_dists, budget, st, nullptr);
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(st, &g);  // always ends the capture
  if (rc || e != cudaSuccess) {
    if (g) cudaGraphDestroy(g);
    return rc ? rc : cuda_status(e, "cudaStreamEndCapture");
  }
  cudaGraphExec_t ex = nullptr;
  const cudaError_t ei = cudaGraphInstantiate(&ex, g, 0);
  if (ei != cudaSuccess) {
    cudaGraphDestroy(g);
    return cuda_status(ei, "cudaGraphInstantiate");
  }
  *out = new SearchGraph{g, ex, g_launches};
  return KATO_OK;
}

int graph_launch(void *h, cudaStream_t st) {
  if (!h) return invalid("null graph");
  KATO_CUDA(cudaGraphLaunch(static_cast<SearchGraph *>(h)->exec, st));
  return KATO_OK;
}

uint32_t graph_launches(const void *h) {
  return h ? static_cast<const SearchGraph *>(h)->launches : 0;
}

void graph_destroy(void *h) {
  auto *g = static_cast<SearchGraph *>(h);
  if (!g) return;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  delete g;
}

void *timer_create(uint32_t max_passes) {
  auto *t = new PhaseTimer();
  t->max_passes = max_passes;
  t->ev.resize(static_cast<size_t>(max_passes) * kTimerStride);
  t->kdone.assign(max_passes, 0);
  for (auto &e : t->ev)
    if (cudaEventCreate(&e) != cudaSuccess) {
      delete t;
      return nullptr;
    }
  return t;
}

void timer_destroy(void *p) {
  auto *t = static_cast<PhaseTimer *>(p);
  if (!t) return;
  for (auto &e : t->ev) cudaEventDestroy(e);
  delete t;
}

int timer_read(void *p, float *ms, uint32_t *passes) {
  auto *t = static_cast<PhaseTimer *>(p);
  for (int i = 0; i < KATO_PHASES; ++i) ms[i] = 0.0f;
  *passes = t->used;
  for (int k = 0; k < KATO_TIMED_KERNELS; ++k) t->kms[k] = 0.0f, t->kn[k] = 0;
  if (t->used == 0) return KATO_OK;
  // the last phase event of the last pass follows every other event in it
  KATO_CUDA(cudaEventSynchronize(t->ev[(t->used - 1) * kTimerStride + KATO_PHASES]));
  for (uint32_t u = 0; u < t->used; ++u) {
    const cudaEvent_t *e = t->ev.data() + static_cast<size_t>(u) * kTimerStride;
    for (int i = 0; i < KATO_PHASES; ++i) {
      float x = 0;
      if (cudaEventElapsedTime(&x, e[i], e[i + 1]) == cudaSuccess) ms[i] += x;
    }
    for (int k = 0; k < KATO_TIMED_KERNELS; ++k) {
      float x = 0;
      if ((t->kdone[u] >> k & 1u) &&
          cudaEventElapsedTime(&x, e[KATO_PHASES + 1 + 2 * k], e[KATO_PHASES + 2 + 2 * k]) ==
              cudaSuccess) {
        t->kms[k] += x;
        ++t->kn[k];
      }
    }
    t->kdone[u] = 0;
  }
  t->used = 0;
  return KATO_OK;
}

void timer_kernels(void *p, float *ms, uint32_t *launches) {
  const auto *t = static_cast<const PhaseTimer *>(p);
  for (int k = 0; k < KATO_TIMED_KERNELS; ++k) {
    ms[k] = t->kms[k];
    launches[k] = t->kn[k];
  }
}

size_t search_workspace(const katoann_gpu_index *ix, uint32_t max_batch, uint32_t k, uint32_t p,
                        int ranking, uint32_t survivors) {
  Plan pl{};
  if (make_plan(ix, max_batch, k, p, ranking, survivors, &pl)) return 0;
  return pl.total;
}


}  // namespace kato
