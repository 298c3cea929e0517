// The end of a search: the exact best S candidates of each query by (ranking
// distance, id), their exact distances and the reference's top-k.
//
// Reference: the merge of the per-list heaps (src/index.cpp:1058-1080,
// :1205-1218), the refinement (:1081-1112), the top-k heap (:1113-1124) and
// emit_topk (:384-398).
#include <algorithm>

#include "finish.cuh"
#include "rank_tc.cuh"
#include "rows.cuh"
#include "scan.cuh"

namespace kato {

namespace {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr int kThreads = 256;

// ---------------------------------------------------- block selection helper
// Chooses the `p` smallest of n entries by (key, id), where entry i gives
// key = K(i) and id = I(i); keys == kEmpty are never chosen. Writes the chosen
// (key << 32 | id, position) pairs into sel/pos (unsorted) and returns how
// many were chosen (min(p, non-empty)). Radix selection over 8-bit digits,
// first of the key, then of the id among the entries tied at the boundary key.
template <class KeyF, class IdF>
__device__ uint32_t block_select(uint32_t n, uint32_t p, KeyF K, IdF I, unsigned long long *sel,
                                 uint32_t *pos, uint32_t *hist, uint32_t *scratch, uint32_t *wsum,
                                 bool *boundary_tie) {
  const uint32_t tid = threadIdx.x, nt = blockDim.x;
  // count non-empty
  if (tid == 0) scratch[0] = 0;
  __syncthreads();
  {
    uint32_t m = 0;
    for (uint32_t i = tid; i < n; i += nt) m += K(i) != kEmpty;
    atomicAdd(&scratch[0], m);
  }
  __syncthreads();
  const uint32_t valid = scratch[0];
  __syncthreads();
  const uint32_t want = min(p, valid);
  *boundary_tie = false;
  if (want == 0) return 0;
  uint32_t T = kEmpty, idmax = 0xFFFFFFFFu;
  if (want < valid) {
    // radix select of the want-th key
    uint32_t prefix = 0, rank = want - 1;
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (uint32_t i = tid; i < 256; i += nt) hist[i] = 0;
      __syncthreads();
      const uint32_t hm = shift == 24 ? 0u : (0xFFFFFFFFu << (shift + 8));
      for (uint32_t i = tid; i < n; i += nt) {
        const uint32_t k = K(i);
        if (k != kEmpty && (k & hm) == prefix) atomicAdd(&hist[(k >> shift) & 0xFFu], 1u);
      }
      __syncthreads();
      block_pick_digit(hist, rank, scratch + 1, wsum);
      rank -= scratch[2];
      prefix |= scratch[1] << shift;
      __syncthreads();
    }
    T = prefix;
    const uint32_t need = rank + 1;
    if (tid == 0) scratch[3] = 0;
    __syncthreads();
    {
      uint32_t m = 0;
      for (uint32_t i = tid; i < n; i += nt) m += K(i) == T;
      atomicAdd(&scratch[3], m);
    }
    __syncthreads();
    const uint32_t neq = scratch[3];
    *boundary_tie = neq > need;
    if (neq > need) {
      uint32_t ip = 0, ir = need - 1;
      for (int shift = 24; shift >= 0; shift -= 8) {
        for (uint32_t i = tid; i < 256; i += nt) hist[i] = 0;
        __syncthreads();
        const uint32_t hm = shift == 24 ? 0u : (0xFFFFFFFFu << (shift + 8));
        for (uint32_t i = tid; i < n; i += nt) {
          if (K(i) != T) continue;
          const uint32_t id = I(i);
          if ((id & hm) == ip) atomicAdd(&hist[(id >> shift) & 0xFFu], 1u);
        }
        __syncthreads();
        block_pick_digit(hist, ir, scratch + 1, wsum);
        ir -= scratch[2];
        ip |= scratch[1] << shift;
        __syncthreads();
      }
      idmax = ip;
    }
  }
  if (tid == 0) scratch[4] = 0;
  __syncthreads();
  for (uint32_t i = tid; i < n; i += nt) {
    const uint32_t k = K(i);
    if (k == kEmpty) continue;
    bool take = k < T;
    uint32_t id = 0;
    if (!take && k == T) {
      id = I(i);
      take = id <= idmax;
    } else if (take) {
      id = I(i);
    }
    if (take) {
      const uint32_t at = atomicAdd(&scratch[4], 1u);
      if (at < want) {
        sel[at] = (static_cast<unsigned long long>(k) << 32) | id;
        pos[at] = i;
      }
    }
  }
  __syncthreads();
  return want;
}

// In-shared-memory bitonic sort of n (key, payload) pairs, ascending by key.
__device__ void block_sort_pairs(unsigned long long *key, uint32_t *val, uint32_t n) {
  uint32_t np2 = 1;
  while (np2 < n) np2 <<= 1;
  for (uint32_t i = n + threadIdx.x; i < np2; i += blockDim.x) {
    key[i] = ~0ull;
    val[i] = 0;
  }
  __syncthreads();
  for (uint32_t size = 2; size <= np2; size <<= 1)
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x) {
        const uint32_t jx = i ^ stride;
        if (jx > i) {
          const bool up = (i & size) == 0;
          const unsigned long long a = key[i], b = key[jx];
          if ((a > b) == up) {
            key[i] = b;
            key[jx] = a;
            const uint32_t tv = val[i];
            val[i] = val[jx];
            val[jx] = tv;
          }
        }
      }
      __syncthreads();
    }
}

// --------------------------------------------------------------- full mode
// Per query: the k smallest of its slot entries by (distance, id), ascending,
// padded.
__global__ void __launch_bounds__(kThreads) merge_kernel(
    const uint2 *slots, uint32_t per_query, uint32_t per_probe, const uint32_t *qcount,
    const uint32_t *qprobes, const uint32_t *__restrict__ ids, uint32_t k, uint32_t *out_ids,
    float *out_dists, unsigned long long *tie_count) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t hist[256], scratch[8], wsum[8];
  __shared__ bool tie;
  unsigned long long *sel = reinterpret_cast<unsigned long long *>(smem);
  uint32_t np2 = 1;
  while (np2 < k) np2 <<= 1;
  uint32_t *pos = reinterpret_cast<uint32_t *>(sel + np2);
  const uint32_t q = blockIdx.x;
  const uint2 *e = slots + static_cast<size_t>(q) * per_query;
  // counted entries, or its probes' slots (rank-major), of which the first
  // budget ones were written
  const uint32_t n = qcount    ? min(qcount[q], per_query)
                     : qprobes ? min(per_query, qprobes[q] * per_probe)
                               : per_query;
  auto K = [&](uint32_t i) { return e[i].x; };
  auto I = [&](uint32_t i) { return ids[e[i].y]; };
  const uint32_t got = block_select(n, k, K, I, sel, pos, hist, scratch, wsum, &tie);
  if (threadIdx.x == 0 && tie && tie_count) atomicAdd(tie_count, 1ull);
  block_sort_pairs(sel, pos, got);
  for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
    uint32_t id = 0xFFFFFFFFu;
    float dd = 3.402823466e+38f;
    if (i < got) {
      id = static_cast<uint32_t>(sel[i] & 0xFFFFFFFFu);
      dd = __uint_as_float(static_cast<uint32_t>(sel[i] >> 32));
    }
    out_ids[static_cast<size_t>(q) * k + i] = id;
    out_dists[static_cast<size_t>(q) * k + i] = dd;
  }
}

// --------------------------------------------------------- overflow rescan
// A query whose buffer overflowed (more than `cap` rows within its seed bound,
// or dropped records; the buffer holds the first of them) is rescanned by its
// own CTA, in rounds:
//   * K = the S-th smallest key (distance bits << 32 | id) among the rows in
//     its buffer - an upper bound on the query's true S-th best key, as they
//     are some of its candidates;
//   * the rows of its probed lists with key <= K go into the buffer. If they
//     fit, it holds every row that can be selected. Otherwise the next round's
//     K comes from the new buffer and is strictly smaller (its cap > S
//     distinct keys are all <= K), which shrinks the count by about cap / S;
//   * after kRescanRounds rounds, the S smallest keys by 8-bit radix selection
//     over all of its candidates.
// Distances are recomputed from the codes; results never depend on the buffer
// size. Returns the entries in the buffer.
constexpr int kRescanRounds = 2;

// Candidates that K looks at: a subset's S-th smallest key is a bound as well,
// and eight times S leave about an eighth of the rows (with S = 4,000, 2,048 left
// all of them to a selection by digits over every row: 256 queries of 700 lists at
// 300k x 128 363 ms, 2.5 now).
constexpr uint32_t kBoundLook = 2048;
__device__ __forceinline__ uint32_t bound_look(uint32_t in, uint32_t S) {
  return min(in, max(kBoundLook, 8 * S));
}

__device__ uint32_t rescan(const FinishArgs &A, uint32_t q, uint32_t n, uint2 *buf, uint32_t *qw,
                           uint32_t *hist, uint32_t *sel, uint32_t *count) {
  const RowKey key{A.xhi, A.rank_xnorm, A.ids, A.dc, A.h, A.scale};
  const uint32_t cap = A.per_query, tid = threadIdx.x;
  load_query_words(A.qhi, q, A.dc, A.h, qw);
  __syncthreads();
  const int64_t qn = A.rank_qnorm[q];
  const uint32_t *pq = A.probed + static_cast<size_t>(q) * A.nprobe;
  const uint32_t np = A.qprobes ? A.qprobes[q] : A.nprobe;  // the query's own budget
  uint32_t in = min(n & ~kDropped, cap);
  unsigned long long K;
  for (int round = 0; round < kRescanRounds; ++round) {
    const uint32_t look = bound_look(in, A.S);
    K = look < A.S ? ~0ull
                   : block_select64(
                         look, A.S - 1,
                         [&](uint32_t i) {
                           const uint2 e = buf[i];
                           return (static_cast<unsigned long long>(e.x) << 32) | A.ids[e.y];
                         },
                         hist, sel);
    if (tid == 0) *count = 0;
    __syncthreads();
    for (uint32_t r = 0; r < np; ++r) {
      const uint32_t r0 = A.list_off[pq[r]];
      for_rows_split(
          A.xhi, A.dc, A.h, qw, r0, A.list_off[pq[r] + 1] - r0,
          [&](uint32_t i, uint32_t dot, int64_t xn) {
            const int64_t l2 = qn + xn - 2 * static_cast<int64_t>(dot);
            const unsigned long long k =
                (static_cast<unsigned long long>(__float_as_uint(dist_value(l2, A.scale))) << 32) |
                A.ids[r0 + i];
            if (k <= K) {
              const uint32_t at = atomicAdd(count, 1u);
              if (at < cap) buf[at] = make_uint2(static_cast<uint32_t>(k >> 32), r0 + i);
            }
          },
          [&](uint32_t i) { return A.rank_xnorm[r0 + i]; });
    }
    __syncthreads();
    in = min(*count, cap);
    if (*count <= cap) return in;
    __syncthreads();
  }
  uint32_t total = 0;
  for (uint32_t r = 0; r < np; ++r) total += A.list_off[pq[r] + 1] - A.list_off[pq[r]];
  // more than cap >= S candidates, so the S-th smallest key exists
  K = block_select64(
      total, A.S - 1,
      [&](uint32_t i) {
        uint32_t r = 0;
        for (;;) {
          const uint32_t len = A.list_off[pq[r] + 1] - A.list_off[pq[r]];
          if (i < len) break;
          i -= len;
          ++r;
        }
        return key(A.list_off[pq[r]] + i, qw, qn);
      },
      hist, sel);
  if (tid == 0) *count = 0;
  __syncthreads();
  for (uint32_t r = 0; r < np; ++r)
    for (uint32_t row = A.list_off[pq[r]] + tid; row < A.list_off[pq[r] + 1]; row += blockDim.x) {
      const unsigned long long k = key(row, qw, qn);
      if (k <= K) {
        const uint32_t at = atomicAdd(count, 1u);  // exactly S rows (distinct ids)
        if (at < cap) buf[at] = make_uint2(static_cast<uint32_t>(k >> 32), row);
      }
    }
  __syncthreads();
  return min(*count, cap);
}

// The first round for all overflowing queries at once, before finish_kernel,
// where p times the longest list is above cap: a round by one CTA reads its
// query's rows at some 30 GB/s (5 ms for 224 lists at 10M), the grid shares them.
// What bounds the round is a chain of latencies for each query: the bound's
// candidates are read once into shared memory (eight digits of a selection over
// them in global memory took 95 us), a list of the queries is kept instead of
// searching their flags, and the CTAs find their rows through the sums of 256
// lists at a time, where walking list by list took 60 us. The phase with two queries
// of 512 probes at 10M: 79 us, 680 before; with nothing to do 9 us, its events included.
__global__ void __launch_bounds__(kThreads) overflow_bound_kernel(const __grid_constant__ FinishArgs A,
                                                                  uint32_t *qcount, uint32_t nq) {
  after_previous();
  __shared__ unsigned long long keys[kBoundLook];
  __shared__ uint32_t hist[256], sel[2], list[kThreads], n_list;
  const uint32_t tid = threadIdx.x, cap = A.per_query;
  // thread t looks at the CTA's t-th query
  for (uint32_t q0 = blockIdx.x; q0 < nq; q0 += gridDim.x * kThreads) {
    const uint32_t mine = q0 + tid * gridDim.x;
    const bool full = mine < nq && qcount[mine] > cap;
    if (mine < nq) A.over[mine] = full;
    if (tid == 0) n_list = 0;
    if (!__syncthreads_or(full)) continue;
    if (full) list[atomicAdd(&n_list, 1u)] = mine;
    __syncthreads();
    for (uint32_t i = 0; i < n_list; ++i) {
      const uint32_t q = list[i], n = qcount[q];
      const uint2 *buf = A.slots + static_cast<size_t>(q) * cap;
      const uint32_t look = bound_look(min(n & ~kDropped, cap), A.S);
      unsigned long long K = ~0ull;
      if (look > kBoundLook) {
        K = block_select64(
            look, A.S - 1,
            [&](uint32_t j) {
              const uint2 e = buf[j];
              return (static_cast<unsigned long long>(e.x) << 32) | A.ids[e.y];
            },
            hist, sel);
      } else if (look >= A.S) {
#pragma unroll
        for (uint32_t j = 0; j < kBoundLook; j += kThreads)
          if (j + tid < look) {
            const uint2 e = buf[j + tid];
            keys[j + tid] = (static_cast<unsigned long long>(e.x) << 32) | A.ids[e.y];
          }
        __syncthreads();
        K = block_select64(look, A.S - 1, [&](uint32_t j) { return keys[j]; }, hist, sel);
      }
      __syncthreads();  // every thread has read the count
      if (tid == 0) {
        A.over_key[q] = K;
        A.over_list[atomicAdd(A.over_n, 1u)] = q;
        qcount[q] = 0;
        atomicMax(A.rescans + 1, static_cast<unsigned long long>(n & ~kDropped));
        atomicAdd(A.rescans, 1ull);
      }
    }
    __syncthreads();  // n_list is written again
  }
}

__global__ void __launch_bounds__(kThreads) overflow_rows_kernel(const __grid_constant__ FinishArgs A,
                                                                 uint32_t *qcount) {
  after_previous();
  const uint32_t found = *A.over_n;
  if (found == 0) return;
  __shared__ __align__(16) uint32_t qw[1024 / 4];
  __shared__ uint32_t first[kThreads], upto[kThreads], rows[kThreads], wsum[kThreads / 32];
  const uint32_t cap = A.per_query, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t turn = blockIdx.x;  // pieces of 256 rows until this CTA's next one
  for (uint32_t i = 0; i < found; ++i) {
    const uint32_t q = A.over_list[i];
    load_query_words(A.qhi, q, A.dc, A.h, qw);
    const int64_t qn = A.rank_qnorm[q];
    const unsigned long long K = A.over_key[q];
    const uint32_t *pq = A.probed + static_cast<size_t>(q) * A.nprobe;
    const uint32_t np = A.qprobes ? A.qprobes[q] : A.nprobe;
    uint2 *buf = A.slots + static_cast<size_t>(q) * cap;
    for (uint32_t rb = 0; rb < np; rb += kThreads) {
      uint32_t at = 0, n = 0;
      if (rb + tid < np) {
        const uint32_t c = pq[rb + tid];
        at = A.list_off[c];
        n = A.list_off[c + 1] - at;
      }
      uint32_t incl = div_up(n, kThreads);  // the list's pieces, then those up to its end
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) wsum[warp] = incl;
      __syncthreads();  // (the query's words are there too)
      for (uint32_t w = 0; w < warp; ++w) incl += wsum[w];
      first[tid] = at;
      rows[tid] = n;
      upto[tid] = incl;
      __syncthreads();
      const uint32_t pieces = upto[kThreads - 1];
      for (; turn < pieces; turn += gridDim.x) {
        uint32_t lo = 0, hi = kThreads - 1;  // the first list that ends after piece `turn`
        while (lo < hi) {
          const uint32_t mid = (lo + hi) / 2;
          if (upto[mid] > turn) hi = mid;
          else lo = mid + 1;
        }
        const uint32_t at0 = (turn - (lo ? upto[lo - 1] : 0)) * kThreads, r0 = first[lo] + at0;
        for_rows_split(
            A.xhi, A.dc, A.h, qw, r0, min(rows[lo] - at0, static_cast<uint32_t>(kThreads)),
            [&](uint32_t j, uint32_t dot, int64_t xn) {
              const int64_t l2 = qn + xn - 2 * static_cast<int64_t>(dot);
              const uint32_t d = __float_as_uint(dist_value(l2, A.scale));
              if (((static_cast<unsigned long long>(d) << 32) | A.ids[r0 + j]) > K) return;
              const uint32_t to = atomicAdd(qcount + q, 1u);
              if (to < cap) buf[to] = make_uint2(d, r0 + j);
            },
            [&](uint32_t j) { return A.rank_xnorm[r0 + j]; });
      }
      turn -= pieces;
      __syncthreads();  // the lists and the query's words are written again
    }
  }
}

// ------------------------------------------------------------- tied top-k
// The reference's heap (:1113-1124) over the survivors in its order, for a
// query whose k-th exact distance ties with the next: the first k enter; a
// later one replaces the largest (distance, id) when its distance is strictly
// smaller; then ascending by (distance, id). kid: distance bits << 32 | id
// (~0 for an id without a row), skey: ranking distances; both are reordered.
__device__ void tied_topk(const FinishArgs &A, uint32_t ns, unsigned long long *kid, uint32_t *val,
                          uint32_t *skey, float *hd, uint32_t *out_ids, float *out_dists) {
  const uint32_t k = A.k;
  for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x) {
    const unsigned long long v = kid[i];
    val[i] = static_cast<uint32_t>(v >> 32);
    kid[i] = (static_cast<unsigned long long>(skey[i]) << 32) | static_cast<uint32_t>(v);
  }
  __syncthreads();
  block_sort_pairs(kid, val, ns);  // ascending by (ranking distance, id): fed from the end
  if (k <= 32) {
    // one warp holds the heap sorted descending by (distance, id) across its
    // lanes - lane 0 is the largest, the one the reference evicts - so an
    // insertion is one ballot and one shift; unused lanes sort below all
    if (threadIdx.x >= 32) return;
    const uint32_t u = threadIdx.x;
    float d = -1.0f;
    uint32_t id = 0u, n = 0;
    for (uint32_t s = ns; s-- > 0;) {
      const float dd = __uint_as_float(val[s]);
      const uint32_t ii = static_cast<uint32_t>(kid[s]);
      if (ii >= A.npts) continue;  // ids without a row are skipped (:1091-1094)
      const bool gt = d > dd || (d == dd && id > ii);  // this slot sorts above the new one
      if (n < k) {
        // enters after the g larger ones; the rest move up one lane
        const uint32_t g = __popc(__ballot_sync(0xffffffffu, gt && u < n));
        const float ud = __shfl_up_sync(0xffffffffu, d, 1);
        const uint32_t uid = __shfl_up_sync(0xffffffffu, id, 1);
        if (u == g) {
          d = dd;
          id = ii;
        } else if (u > g && u <= n) {
          d = ud;
          id = uid;
        }
        ++n;
        continue;
      }
      if (!(dd < __shfl_sync(0xffffffffu, d, 0))) continue;  // strictly below the largest
      // the largest leaves; the g larger ones below it move down one lane
      const uint32_t g = __popc(__ballot_sync(0xffffffffu, gt && u >= 1 && u < k));
      const float nd = __shfl_down_sync(0xffffffffu, d, 1);
      const uint32_t nid = __shfl_down_sync(0xffffffffu, id, 1);
      if (u < g) {
        d = nd;
        id = nid;
      } else if (u == g) {
        d = dd;
        id = ii;
      }
    }
    if (u < n) {  // ascending: lane u is the (n - 1 - u)-th
      out_ids[n - 1 - u] = id;
      out_dists[n - 1 - u] = d;
    }
    return;
  }
  if (threadIdx.x != 0) return;
  uint32_t *hid = skey;
  uint32_t n = 0;
  for (uint32_t s = ns; s-- > 0;) {
    const float dd = __uint_as_float(val[s]);
    const uint32_t id = static_cast<uint32_t>(kid[s]);
    if (id >= A.npts) continue;
    if (n < k) {
      hd[n] = dd;
      hid[n] = id;
      ++n;
      continue;
    }
    uint32_t mi = 0;  // the largest (distance, id)
    for (uint32_t i = 1; i < n; ++i)
      if (hd[i] > hd[mi] || (hd[i] == hd[mi] && hid[i] > hid[mi])) mi = i;
    if (dd < hd[mi]) {
      hd[mi] = dd;
      hid[mi] = id;
    }
  }
  // ascending by (distance, id)
  for (uint32_t i = 1; i < n; ++i) {
    const float d0 = hd[i];
    const uint32_t i0 = hid[i];
    uint32_t m = i;
    while (m > 0 && (hd[m - 1] > d0 || (hd[m - 1] == d0 && hid[m - 1] > i0))) {
      hd[m] = hd[m - 1];
      hid[m] = hid[m - 1];
      --m;
    }
    hd[m] = d0;
    hid[m] = i0;
  }
  for (uint32_t i = 0; i < n; ++i) {
    out_ids[i] = hid[i];
    out_dists[i] = hd[i];
  }
}

// ------------------------------------------------------- survivors to top-k
// One CTA per query, from the candidates to the results: the survivors never
// leave shared memory (two kernels, a sorted survivor list through memory and
// a heap replayed by one warp, or one thread for k > 32, took 174 us at 10M
// and 332 us for 113 queries with k = 100 and 128 survivors).
//   1. the best S candidates by (ranking distance, id), as a set: up to 256
//      candidates by counting, per candidate, the smaller ones (one broadcast
//      read serves four comparisons and there are no barriers; a radix
//      selection needs 24), more by radix selection;
//   2. the survivors' dot products: rows of up to 256 dimensions by 4, 8 or 16
//      lanes, four rows of each such group in flight, longer ones two at a time
//      by a warp (64 registers, four CTAs per SM); the distances then by one
//      thread each. A warp per row, with its distance worked out by one lane
//      before the next was read, waited on memory between rows: 2000 queries,
//      128 survivors of 768 dimensions, took 153 us instead of 104, 333 queries
//      with 400 of 102 took 65 instead of 35, 1024 with 64 of 128 took 32
//      instead of 23; 4096 with 32 of 3,072 (118 us of HBM time) 145 as before;
//   3. the k smallest by (exact distance, id), again by counting or, above 256
//      survivors, a bitonic sort.
// Step 3 is what the reference's heap leaves unless a distance ties across the
// k boundary: it keeps the first k and replaces the largest (distance, id) by
// a strictly smaller distance, so only the order in which tied entries came
// can matter. Then the heap is replayed, survivors in the reference's order
// (descending ranking distance, id).
constexpr uint32_t kCount = 256;  // entries ranked by counting, one per thread

__global__ void __launch_bounds__(kThreads, 4) finish_kernel(const __grid_constant__ FinishArgs A) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) uint32_t hist[256];
  __shared__ uint32_t scratch[8], wsum[8], nsel, bound[2];
  __shared__ bool tie;
  const uint32_t q = blockIdx.x, tid = threadIdx.x, S = A.S, k = A.k;
  const uint32_t n16 = A.dc / 16;  // 16-byte words of a plane row
  uint32_t np2 = 1;
  while (np2 < S) np2 <<= 1;
  np2 = max(np2, kCount);
  uint4 *sq = reinterpret_cast<uint4 *>(smem);                                        // [2][n16]
  unsigned long long *kid = reinterpret_cast<unsigned long long *>(sq + 2 * n16);     // [np2]
  uint32_t *srow = reinterpret_cast<uint32_t *>(kid + np2);                           // [np2] rows
  uint32_t *skey = srow + np2;                                                        // [np2] ranking distances
  uint2 *e = A.slots + static_cast<size_t>(q) * A.per_query;
  uint32_t n = A.qcount    ? A.qcount[q]
               : A.qprobes ? min(A.per_query, A.qprobes[q] * A.per_probe)
                           : A.per_query;
  if (A.qcount) {
    if (tid == 0) atomicMax(A.rescans + 1, static_cast<unsigned long long>(n & ~kDropped));
    if (n > A.per_query) {
      if (tid == 0 && !(A.over && A.over[q])) atomicAdd(A.rescans, 1ull);
      n = rescan(A, q, n, e, reinterpret_cast<uint32_t *>(sq), hist, scratch, scratch + 4);
      __syncthreads();
    }
  }
  for (uint32_t i = tid; i < n16; i += kThreads) {
    sq[i] = reinterpret_cast<const uint4 *>(A.qhi + static_cast<size_t>(q) * A.dc)[i];
    sq[n16 + i] = reinterpret_cast<const uint4 *>(A.qlo + static_cast<size_t>(q) * A.dc)[i];
  }
  // 1. survivors
  uint32_t ns;
  if (A.qcount && n <= kCount) {
    uint2 mine = make_uint2(kEmpty, 0);
    if (tid < n) mine = e[tid];
    ns = min(n, S);
    if (n <= S) {
      if (tid < n) srow[tid] = mine.y, skey[tid] = mine.x;
    } else {
      hist[tid] = mine.x;  // kEmpty past n: never below a key
      if (tid == 0) nsel = 0, tie = false;
      __syncthreads();
      if (tid < n) {
        uint32_t lt = 0, eq = 0;
        for (uint32_t j = 0; j < n; j += 4) {
          const uint4 o = *reinterpret_cast<const uint4 *>(hist + j);
          lt += (o.x < mine.x) + (o.y < mine.x) + (o.z < mine.x) + (o.w < mine.x);
          eq += (o.x == mine.x) + (o.y == mine.x) + (o.z == mine.x) + (o.w == mine.x);
        }
        bool in = lt + eq <= S;
        if (lt < S && lt + eq > S) {  // ties across the boundary: by id
          const uint32_t id = A.ids[mine.y];
          for (uint32_t j = 0; j < n; ++j)
            if (hist[j] == mine.x) {
              const uint32_t oid = A.ids[e[j].y];
              lt += oid < id || (oid == id && j < tid);
            }
          in = lt < S;
          tie = true;
        }
        if (in) {
          const uint32_t at = atomicAdd(&nsel, 1u);
          srow[at] = mine.y, skey[at] = mine.x;
        }
      }
      __syncthreads();
      if (tid == 0 && tie && A.ties) atomicAdd(A.ties, 1ull);
    }
  } else {
    auto K = [&](uint32_t i) { return e[i].x; };
    auto I = [&](uint32_t i) { return A.ids[e[i].y]; };
    ns = block_select(n, S, K, I, kid, srow, hist, scratch, wsum, &tie);
    if (tid == 0 && tie && A.ties) atomicAdd(A.ties, 1ull);
    for (uint32_t i = tid; i < ns; i += kThreads) {
      skey[i] = static_cast<uint32_t>(kid[i] >> 32);
      srow[i] = e[srow[i]].y;
    }
  }
  __syncthreads();
  // 2. exact distances: kid = the dot products, then distance bits << 32 | id
  const uint32_t lane = tid & 31, warp = tid >> 5;
  // what the distances need besides arrives meanwhile
  const int64_t qn = A.qnorm[q];
  uint32_t id0 = 0;
  int64_t xn0 = 0;
  if (tid < ns) {
    id0 = A.ids[srow[tid]];
    xn0 = A.xnorm[srow[tid]];
  }
  auto dot_of = [](uint32_t hh, uint32_t mx, uint32_t ll) {
    return (static_cast<unsigned long long>(hh) << 16) + (static_cast<unsigned long long>(mx) << 8) + ll;
  };
  auto products = [](uint4 ah, uint4 al, uint4 bh, uint4 bl, uint32_t &hh, uint32_t &mx, uint32_t &ll) {
    hh = dp4(ah.x, bh.x, dp4(ah.y, bh.y, dp4(ah.z, bh.z, dp4(ah.w, bh.w, hh))));
    mx = dp4(ah.x, bl.x, dp4(ah.y, bl.y, dp4(ah.z, bl.z, dp4(ah.w, bl.w, mx))));
    mx = dp4(al.x, bh.x, dp4(al.y, bh.y, dp4(al.z, bh.z, dp4(al.w, bh.w, mx))));
    ll = dp4(al.x, bl.x, dp4(al.y, bl.y, dp4(al.z, bl.z, dp4(al.w, bl.w, ll))));
  };
  if (n16 <= 16) {
    // short rows: 4, 8 or 16 lanes to a row, four rows of each group in flight
    const uint32_t lg = n16 <= 4 ? 2 : n16 <= 8 ? 3 : 4, gl = lane & ((1u << lg) - 1), rows = 32 >> lg;
    const uint32_t u = min(gl, n16 - 1);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const uint4 ah = gl < n16 ? sq[u] : zero, al = gl < n16 ? sq[n16 + u] : zero;
    for (uint32_t s0 = warp * rows * 4; s0 < ns; s0 += kThreads / 32 * rows * 4) {
      uint4 bh[4], bl[4];
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const size_t at = static_cast<size_t>(srow[min(s0 + j * rows + (lane >> lg), ns - 1)]) * A.dc;
        bh[j] = reinterpret_cast<const uint4 *>(A.xhi + at)[u];
        bl[j] = reinterpret_cast<const uint4 *>(A.xlo + at)[u];
      }
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        uint32_t hh = 0, mx = 0, ll = 0;
        products(ah, al, bh[j], bl[j], hh, mx, ll);
        for (uint32_t o = 1; o < 1u << lg; o <<= 1) {
          hh += __shfl_xor_sync(0xffffffffu, hh, o);
          mx += __shfl_xor_sync(0xffffffffu, mx, o);
          ll += __shfl_xor_sync(0xffffffffu, ll, o);
        }
        const uint32_t s = s0 + j * rows + (lane >> lg);
        if (gl == 0 && s < ns) kid[s] = dot_of(hh, mx, ll);
      }
    }
  } else {
    // a warp takes two rows at a time
    for (uint32_t s0 = warp * 2; s0 < ns; s0 += kThreads / 32 * 2) {
      const size_t r0 = static_cast<size_t>(srow[s0]) * A.dc, r1 = static_cast<size_t>(srow[min(s0 + 1, ns - 1)]) * A.dc;
      uint32_t hh0 = 0, mx0 = 0, ll0 = 0, hh1 = 0, mx1 = 0, ll1 = 0;
#pragma unroll 1
      for (uint32_t u = lane; u < n16; u += 32) {
        const uint4 h0 = reinterpret_cast<const uint4 *>(A.xhi + r0)[u], h1 = reinterpret_cast<const uint4 *>(A.xhi + r1)[u];
        const uint4 l0 = reinterpret_cast<const uint4 *>(A.xlo + r0)[u], l1 = reinterpret_cast<const uint4 *>(A.xlo + r1)[u];
        const uint4 ah = sq[u], al = sq[n16 + u];
        products(ah, al, h0, l0, hh0, mx0, ll0);
        products(ah, al, h1, l1, hh1, mx1, ll1);
      }
      hh0 = __reduce_add_sync(0xffffffffu, hh0);
      mx0 = __reduce_add_sync(0xffffffffu, mx0);
      ll0 = __reduce_add_sync(0xffffffffu, ll0);
      hh1 = __reduce_add_sync(0xffffffffu, hh1);
      mx1 = __reduce_add_sync(0xffffffffu, mx1);
      ll1 = __reduce_add_sync(0xffffffffu, ll1);
      if (lane == 0) kid[s0] = dot_of(hh0, mx0, ll0);
      if (lane == 1 && s0 + 1 < ns) kid[s0 + 1] = dot_of(hh1, mx1, ll1);
    }
  }
  __syncthreads();
  for (uint32_t i = tid; i < ns; i += kThreads) {
    if (i >= kThreads) {
      id0 = A.ids[srow[i]];
      xn0 = A.xnorm[srow[i]];
    }
    const uint32_t d = __float_as_uint(dist_value(qn + xn0 - 2 * static_cast<int64_t>(kid[i]), A.scale));
    // ids without a row are skipped (:1091-1094): they sort last
    kid[i] = id0 < A.npts ? (static_cast<unsigned long long>(d) << 32) | id0 : ~0ull;
  }
  if (tid < 2) bound[tid] = kEmpty;
  __syncthreads();
  // 3. top-k
  uint32_t *out_ids = A.out_ids + static_cast<size_t>(q) * k;
  float *out_dists = A.out_dists + static_cast<size_t>(q) * k;
  auto emit = [&](uint32_t at, unsigned long long v) {
    out_ids[at] = v == ~0ull ? 0xFFFFFFFFu : static_cast<uint32_t>(v);
    out_dists[at] = v == ~0ull ? 3.402823466e+38f : __uint_as_float(static_cast<uint32_t>(v >> 32));
  };
  if (ns <= kCount) {
    const unsigned long long v = tid < ns ? kid[tid] : ~0ull;
    uint32_t rank = 0;
    for (uint32_t j = 0; j < ns; ++j) {
      const unsigned long long o = kid[j];
      rank += o < v || (o == v && j < tid);
    }
    // the distances on the two sides of the boundary
    if (tid < ns && (rank == k - 1 || rank == k) && v != ~0ull) bound[rank == k] = static_cast<uint32_t>(v >> 32);
    if (tid < ns && rank < k) emit(rank, v);
  } else {
    block_sort_pairs(kid, skey, ns);
    if (tid < 2 && k - 1 + tid < ns && kid[k - 1 + tid] != ~0ull)
      bound[tid] = static_cast<uint32_t>(kid[k - 1 + tid] >> 32);
    for (uint32_t i = tid; i < min(ns, k); i += kThreads) emit(i, kid[i]);
  }
  for (uint32_t i = ns + tid; i < k; i += kThreads) emit(i, ~0ull);
  __syncthreads();
  if (bound[0] == kEmpty || bound[0] != bound[1]) return;
  tied_topk(A, ns, kid, srow, skey, reinterpret_cast<float *>(skey + np2), out_ids, out_dists);
}

}  // namespace

int rescan_overflows(const FinishArgs &A, uint32_t *qcount, uint32_t nq, cudaStream_t st) {
  int sms = 0;
  if (const int rc = current_sms(&sms)) return rc;
  // (so few CTAs that the next kernel's are placed at once)
  launch(overflow_bound_kernel, std::min(nq, kFewCtas - 1), kThreads, 0, st, A, qcount, nq);
  KATO_LAUNCHED("overflow_bound_kernel");
  launch(overflow_rows_kernel, 4 * sms, kThreads, 0, st, A, qcount);
  KATO_LAUNCHED("overflow_rows_kernel");
  return KATO_OK;
}

int finish(const FinishArgs &A, uint32_t nq, cudaStream_t st) {
  if (nq == 0) return KATO_OK;
  uint32_t np2 = 1;
  while (np2 < A.S) np2 <<= 1;
  np2 = std::max(np2, kCount);
  const size_t smem = static_cast<size_t>(A.dc) * 2 + static_cast<size_t>(np2) * 16 +
                      static_cast<size_t>(A.k) * 4;
  if (const int rc = smem_limit(reinterpret_cast<const void *>(finish_kernel), static_cast<int>(smem),
                                "finish_kernel shared memory"))
    return rc;
  launch(finish_kernel, nq, kThreads, smem, st, A);
  KATO_LAUNCHED("finish_kernel");
  return KATO_OK;
}

int merge_topk(const uint2 *slots, uint32_t per_query, uint32_t per_probe, const uint32_t *qcount,
               const uint32_t *qprobes, const uint32_t *ids, uint32_t nq, uint32_t k, uint32_t *out_ids, float *out_dists,
               unsigned long long *ties, cudaStream_t st) {
  uint32_t np2 = 1;
  while (np2 < k) np2 <<= 1;
  const size_t smem = static_cast<size_t>(np2) * 12;
  if (const int rc = smem_limit(reinterpret_cast<const void *>(merge_kernel), static_cast<int>(smem),
                                "merge_kernel shared memory"))
    return rc;
  launch(merge_kernel, nq, kThreads, smem, st, slots, per_query, per_probe, qcount, qprobes, ids, k, out_ids,
                                           out_dists, ties);
  KATO_LAUNCHED("merge_kernel");
  return KATO_OK;
}

}  // namespace kato
