// Ranking pass on the tensor cores.
//
// The reference scores every row of every probed list against the queries
// that probe it with the high bytes of the leading h rotated dimensions
// (sq16_high_l2, src/kernels.cpp:216-243, called from src/index.cpp:1016-1042)
// and keeps each query's best S by (distance, id) (:63-97 / :101-135). Here:
//   1. rank_seed_kernel gives every query an upper bound on its final S-th
//      ranking l2: the S-th smallest one over the first rows of its nearest
//      lists (any S of its candidates bound its S-th best from above), widened
//      so that every l2 with the same float distance stays inside;
//   2. rank_tc_kernel scores (row, query) pairs and appends those that may lie
//      within the bound to per-CTA record lists (below);
//   3. tc_bucket_kernel completes the records' l2, drops those beyond the
//      bound and sorts the rest into per-query buffers with their float
//      distances;
//   4. finish_kernel (finish.cu) takes the exact best S by (distance, id) from
//      each buffer, after an exact rescan of a query whose buffer overflowed,
//      so results never depend on the bound or the buffer size.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "kcommon.cuh"
#include "rank_tc.cuh"
#include "rows.cuh"
#include "scan.cuh"
#include "tc.cuh"

namespace kato {

namespace {

constexpr uint32_t kSeedCap = 4096;  // rows a seed bound looks at, at most
constexpr uint32_t kSeedMany = 65536;  // probed rows from which it looks at twice as many

// rank_tc_kernel: one CTA per SM takes an equal share, by cost, of all 64-row
// slabs of all work items (an item is a list and up to N of the queries
// probing it).
//
// What bounds it is DRAM: each probed row's ranking bytes are read once per
// item, and a row meets few queries (10M x 1,024, nlist 16,384, nprobe 72:
// 8 to 18 per list), so the products are cheap for any matrix path. mma.sync
// m16n8k16 is taken over tcgen05 because the work comes in groups of 8
// queries and its operands stay in registers: 1,024 fp16 products per clock
// per SM measured, against 54 to 108 cycles for each tcgen05.mma of 128 rows,
// 16 to 64 queries and 16 dimensions, whose operands also had to pass through
// tensor memory between five roles of warps.
//
//   - eight scoring warps, each with its own ring of stages of two TMA boxes
//     (32 rows x `IN` bytes each: a slab's two halves, or two chunks of one
//     half), filled by the warp's own lane 0 ahead of their use. A lane turns the bytes of its four
//     rows into fp16 A fragments, sums each row's norm, and multiplies with
//     the item's queries, eight at a time. A dot product is the same over any
//     order of its dimensions, so the fragments take the dimensions in the
//     order that 16-byte reads deliver them;
//   - four staging warps, each with its own query buffer: every nB-th item's
//     description, bounds and the fp16 rows of its queries, copied ahead of
//     the scoring warps.
// The products of 32 rows x 128 bytes with 16 queries take 109 cycles of an
// SM when nothing else runs (157 when each step is guarded for four query
// groups, so there is a body for two); the rest is what a slab costs besides:
// with 32-row slabs, runtime divisions and 64-bit addresses it was 490 more.
// Exactness. For h <= 256 a row byte b enters as the fp16 bit pattern 0x00bb,
// the subnormal b 2^-24 (one byte permute makes two of them), and a query byte
// as itself: sums of up to 256 * 255^2 < 2^24 such products are exact in fp32
// (kScale undoes the 2^-24). Beyond 256 dimensions both are re-centred to
// (byte - 128), which leaves every squared distance unchanged and bounds a
// product by 2^14: up to 1,024 dimensions add up exactly.
// A pair passes if l2 = qn + xn - 2 dot is at most the query's bound, that is
// if dot - xn / 2 >= -(bound - qn) / 2; rounding is monotone, so no pair within
// the bound fails the float compare, and tc_bucket_kernel drops the few beyond
// it that pass.
//
// Filtered items: a squared distance over the leading f < h dimensions never
// exceeds the one over h, so an item may be scored over its rows' first f
// bytes alone; what passes is recorded with its partial l2 and completed by
// tc_bucket_kernel. On rotated vectors the leading dimensions hold most of
// the distance, and the pass then reads f instead of h bytes per row (10M x
// 1,024, h = 256, f = 128: 0.50 against 0.71 ms). Data whose distance is spread
// evenly would pass nearly everything, so each CTA watches the records its
// slabs give and filters only while completing them costs less.
constexpr int kScoreWarps = kTcScoreWarps, kStageWarps = 4;
constexpr int kTcThreads = (kScoreWarps + kStageWarps) * 32;

static_assert(kStageWarps >= static_cast<int>(kTcMaxBufs), "roles");

// An item as the scoring warps see it: its slabs, rows, queries and chunks of
// IN dimensions.
struct __align__(16) Desc {
  uint32_t s0, s1, row0, nrows;
  uint32_t ne, nch, partial, pad;
};
static_assert(sizeof(Desc) == kTcDesc, "item slot size");

// Shared-memory accesses by 32-bit address.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 lds_float2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16-byte asynchronous global -> shared copy (L2 only).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// A word of shared memory that other warps write meanwhile, as lane 0 reads it:
// the lanes of a warp must not differ in what they do next.
__device__ __forceinline__ uint32_t warp_read(const volatile uint32_t *p) {
  return __shfl_sync(0xffffffffu, *p, 0);
}

// One arrival on `bar` once this thread's copies so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_addr(bar))
               : "memory");
}

// Two bytes of a word (selector) as fp16: the subnormals b 2^-24, or
// (byte - 128) by way of 1024 + byte.
template <bool kCentred>
__device__ __forceinline__ uint32_t half2_of(uint32_t w, uint32_t selector) {
  if (!kCentred) return __byte_perm(w, 0, selector);
  const uint32_t a = __byte_perm(w, 0x64646464u, selector);
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&a), __floats2half2_rn(1152.0f, 1152.0f));
  return *reinterpret_cast<const uint32_t *>(&h);
}

// sum over 16 bytes of b^2
__device__ __forceinline__ uint32_t sq_sum16(const uint32_t *w, uint32_t acc) {
  return dp4(w[0], w[0], dp4(w[1], w[1], dp4(w[2], w[2], dp4(w[3], w[3], acc))));
}

// IN: bytes of a row in one chunk, 128, or 64 where the pass has only 64.
template <uint32_t IN, bool kCentred>
__global__ void __launch_bounds__(kTcThreads, 1)
    rank_tc_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ RankTcArgs A,
                   const __grid_constant__ TcShape S) {
  after_previous();
  constexpr uint32_t NI = IN / 64;        // 16-byte reads per row, lane and chunk
  constexpr uint32_t kBox = kTcBoxRows * IN, kStage = 2 * kBox;
  // row bytes enter as multiples of kScale
  constexpr float kScale = kCentred ? 1.0f : 0x1p-24f;
  extern __shared__ __align__(1024) unsigned char sm[];
  const uint32_t h = A.h, N = S.N, nB = S.Bs, depth = S.Rs;
  const TcSmem L = tc_smem_layout(h, S);
  uint64_t *full = reinterpret_cast<uint64_t *>(sm + L.bars);  // per scoring warp and stage
  uint64_t *d_full = full + kScoreWarps * kTcMaxStages;        // per query buffer: described,
  uint64_t *b_full = d_full + kTcMaxBufs;                      // copied,
  uint64_t *b_empty = b_full + kTcMaxBufs;                     // used by every scoring warp
  volatile uint32_t *err = reinterpret_cast<volatile uint32_t *>(sm + L.err);
  uint32_t *rcount = reinterpret_cast<uint32_t *>(sm + L.rcount);
  // slabs scored; filtered pairs staged, and those of them whose item has been left
  uint32_t *slabs = rcount + 1, *fstaged = rcount + 2, *fpairs = rcount + 3;
  uint32_t *qids = reinterpret_cast<uint32_t *>(sm + L.qids);
  // -(bound - qn) / 2 of each query slot, in units of kScale
  float *qbv = reinterpret_cast<float *>(sm + L.qbv);
  Desc *desc = reinterpret_cast<Desc *>(sm + L.desc);
  const uint32_t nkc = (h + IN - 1) / IN, brow = nkc * IN * 2, btile = N * brow;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (uint32_t s = 0; s < kScoreWarps * kTcMaxStages; ++s) tc::mbar_init(full + s, 1);
    for (uint32_t s = 0; s < kTcMaxBufs; ++s) {
      tc::mbar_init(d_full + s, 1);
      tc::mbar_init(b_full + s, 64);
      tc::mbar_init(b_empty + s, kScoreWarps);
    }
    rcount[0] = rcount[1] = rcount[2] = rcount[3] = 0;
    // the TMA swizzle pattern repeats every 1024 bytes of shared address
    *err = (tc::smem_addr(sm + L.raw) & 1023u) ? 2u : 0u;
    tc::fence_barrier_init();
  }
  __syncthreads();
  // this CTA's slabs t0 .. t1 - 1 and items it0 .. it1
  const uint2 share = A.share[blockIdx.x], upto = A.share[blockIdx.x + 1];
  const uint32_t t0 = share.x, t1 = upto.x, it0 = share.y;
  // per-role cycle profile (first thread of each role): waits, then total
  unsigned long long pw[2] = {0, 0};
  const long long tstart = clock64();
  // a bounded wait by the whole warp on the barrier at shared address b
  // calling meanwhile() between its tries
  auto wait_for = [&](uint32_t b, uint32_t phase, unsigned long long &acc, auto meanwhile) -> bool {
    if (__all_sync(0xffffffffu, tc::mbar_test(b, phase))) return true;
    const long long t = clock64();
    bool ok = false, late = false;
    long long took = 0;
    do {
      ok = __all_sync(0xffffffffu, meanwhile(b, phase));
      took = clock64() - t;
      late = __any_sync(0xffffffffu, took > A.wait);
    } while (!ok && !late && !warp_read(err));
    if (late) *err = 1, ok = false;
    acc += took;
    return ok;
  };
  auto wait = [&](uint32_t b, uint32_t phase, unsigned long long &acc) -> bool {
    return wait_for(b, phase, acc, [](uint32_t x, uint32_t p) { return tc::mbar_try(x, p); });
  };

  if (t0 < t1 && !warp_read(err)) {
    // the item after the last one may start inside the next share
    const uint32_t n_li = upto.y - it0 + (A.tile_off[upto.y] < t1);
    const uint32_t d_full_a = tc::smem_addr(d_full), b_full_a = tc::smem_addr(b_full);
    const uint32_t b_empty_a = tc::smem_addr(b_empty), desc_a = tc::smem_addr(desc);
    if (warp < kScoreWarps) {
      // ---- scoring: slabs t0 + warp, t0 + warp + kScoreWarps, ...
      const uint32_t g = lane >> 2, tig = lane & 3;
      const uint32_t ring = tc::smem_addr(sm + L.raw) + warp * depth * kStage;
      const uint32_t bar = tc::smem_addr(full + warp * kTcMaxStages);
      const uint32_t qbv_a = tc::smem_addr(qbv) + tig * 8, qid_a = tc::smem_addr(qids) + tig * 8;
      const uint32_t b_a = tc::smem_addr(sm + L.b) + g * brow;
      uint4 *rec = A.rec + static_cast<size_t>(blockIdx.x) * A.rec_cap;
      // fetch side: the next stage to fetch (slab tn, its cn-th), its item (the
      // i_n-th, in buffer i_bf) and ring stage
      uint32_t inflight = 0, tn = t0 + warp, cn = 0, is = 0;
      uint32_t i_n = 0, i_bf = nB - 1, i_ph = 1, i_end = 0, i_row = 0, i_nch = 1, i_pairs = 1;
      // score side: the item being scored (the c_n-th), ring stage and phase
      uint32_t c_n = 0, c_bf = nB - 1, c_ph = 1, c_end = 0, cs = 0, cph = 0;
      uint4 d0 = make_uint4(0, 0, 0, 0), d1 = d0;
      // fetches ahead as far as the ring and the described items allow; the
      // item of the chunk to be read next is always described
      auto fetch = [&]() {
        while (inflight < depth && tn < t1) {
          while (tn >= i_end) {
            const uint32_t bf = i_bf + 1 == nB ? 0 : i_bf + 1, ph = i_ph ^ (bf == 0);
            if (!__all_sync(0xffffffffu, tc::mbar_test(d_full_a + bf * 8, ph))) return;
            const uint4 n0 = lds128(desc_a + bf * kTcDesc);
            i_nch = lds32(desc_a + bf * kTcDesc + 20);
            i_end = n0.y, i_row = n0.z - n0.x * kTcSlab, i_pairs = (i_nch + 1) / 2;
            ++i_n, i_bf = bf, i_ph = ph;
          }
          if (lane == 0) {
            const uint32_t dst = ring + is * kStage, b = bar + is * 8;
            const int32_t y = static_cast<int32_t>(i_row + tn * kTcSlab);
            if (i_nch == 1) {  // the slab's two halves
              tc::mbar_expect_tx(b, kStage);
              tc::tma_load_2d(dst, &tmap, 0, y, b);
              tc::tma_load_2d(dst + kBox, &tmap, 0, y + static_cast<int32_t>(kTcBoxRows), b);
            } else {           // two chunks of the first, then of the second half
              const uint32_t half = cn >= i_pairs, ch = 2 * (half ? cn - i_pairs : cn);
              const int32_t yh = y + static_cast<int32_t>(half * kTcBoxRows);
              const bool both = ch + 1 < i_nch;
              tc::mbar_expect_tx(b, both ? kStage : kBox);
              tc::tma_load_2d(dst, &tmap, static_cast<int32_t>(ch * IN), yh, b);
              if (both) tc::tma_load_2d(dst + kBox, &tmap, static_cast<int32_t>((ch + 1) * IN), yh, b);
            }
          }
          ++inflight;
          if (++is == depth) is = 0;
          if (i_nch == 1 || ++cn == 2 * i_pairs) cn = 0, tn += kScoreWarps;
        }
      };
      uint32_t xa[4][4 * NI];             // raw words of the lane's rows g, g + 8, g + 16, g + 24
      auto read = [&](uint32_t st) {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
#pragma unroll
          for (uint32_t i = 0; i < NI; ++i) {
            // 16-byte unit of the row, where the TMA's swizzle put it
            const uint32_t u = IN == 128 ? ((2 * tig + i) ^ g) : (tig ^ ((g >> 1) & 3));
            const uint4 v = lds128(st + (g + 8 * q) * IN + u * 16);
            xa[q][4 * i] = v.x, xa[q][4 * i + 1] = v.y, xa[q][4 * i + 2] = v.z, xa[q][4 * i + 3] = v.w;
          }
      };
      // the stage has been read by every lane: on to the next, and refill
      auto release = [&]() {
        __syncwarp();
        if (++cs == depth) cs = 0, cph ^= 1;
        --inflight;
        fetch();
      };
      // the lane's part of its rows' norms
      auto norms = [&](uint32_t (&xn)[4]) {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
#pragma unroll
          for (uint32_t i = 0; i < NI; ++i) {
            const uint32_t *w = xa[q] + 4 * i;
            if (kCentred) xn[q] += static_cast<uint32_t>(tc::centred_sq_sum16(make_uint4(w[0], w[1], w[2], w[3])));
            else xn[q] = sq_sum16(w, xn[q]);
          }
      };
      // the rows' norms from their four lanes' parts, and -xn / 2; `left` rows
      // of the list remain from the lane's first row on, those past its end
      // never pass
      auto finish = [&](uint32_t (&xn)[4], float (&xh)[4], int32_t left) {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
          xn[q] += __shfl_xor_sync(0xffffffffu, xn[q], 1);
          xn[q] += __shfl_xor_sync(0xffffffffu, xn[q], 2);
          xh[q] = static_cast<int32_t>(8 * q) < left
                      ? static_cast<float>(static_cast<int32_t>(xn[q])) * (-0.5f * kScale)
                      : -INFINITY;
        }
      };
      // dimensions 32 s .. of the chunk times the kG query groups at bq
      auto step = [&](auto kg, uint32_t s, uint32_t bq, float (&c)[decltype(kg)::value][2][4]) {
        uint32_t a[2][2][4];
#pragma unroll
        for (uint32_t m = 0; m < 2; ++m)
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j) {
            // A fragments of rows g + 16 m, g + 16 m + 8
            a[m][j][0] = half2_of<kCentred>(xa[2 * m][2 * s + j], 0x4140);
            a[m][j][1] = half2_of<kCentred>(xa[2 * m + 1][2 * s + j], 0x4140);
            a[m][j][2] = half2_of<kCentred>(xa[2 * m][2 * s + j], 0x4342);
            a[m][j][3] = half2_of<kCentred>(xa[2 * m + 1][2 * s + j], 0x4342);
          }
        // the B fragments of two 16-dimension steps: one 16-byte unit of the
        // query's row, swizzled so that eight lanes meet eight banks
        uint32_t u;
        if (IN == 128) {
          u = 4 * tig + s;
          u = u ^ ((u >> 3) & 1) ^ ((g & 1) << 1);
        } else {
          u = (2 * tig + s) ^ (g & 1);
        }
#pragma unroll
        for (uint32_t gr = 0; gr < decltype(kg)::value; ++gr) {
          const uint4 b = lds128(bq + gr * 8 * brow + u * 16);
#pragma unroll
          for (uint32_t m = 0; m < 2; ++m) mma_16816(c[gr][m], a[m][0], b.x, b.y);
#pragma unroll
          for (uint32_t m = 0; m < 2; ++m) mma_16816(c[gr][m], a[m][1], b.z, b.w);
        }
      };
      // tests a group's pairs (query slots at `slot`) and records those that pass
      auto test = [&](const float (&c)[2][4], const float (&xh)[4], const uint32_t (&xn)[4],
                      uint32_t slot, uint32_t row) {
        const float2 th = lds_float2(qbv_a + slot * 4);
        bool hit = false;
#pragma unroll
        for (uint32_t b = 0; b < 8; ++b)
          hit |= c[b >> 2][b & 3] + xh[b >> 1] >= ((b & 1) ? th.y : th.x);
        if (hit) {
          uint32_t mask = 0;
#pragma unroll
          for (uint32_t b = 0; b < 8; ++b)
            mask |= static_cast<uint32_t>(c[b >> 2][b & 3] + xh[b >> 1] >= ((b & 1) ? th.y : th.x)) << b;
          // records (query, xn - 2 dot, row, partial) go to this CTA's list;
          // few lanes have any, so each reserves its own places
          uint32_t at = atomicAdd(rcount, __popc(mask));
          do {
            const uint32_t b = __ffs(mask) - 1;
            mask &= mask - 1;
            const float v0 = b & 4 ? c[1][0] : c[0][0], v1 = b & 4 ? c[1][1] : c[0][1];
            const float v2 = b & 4 ? c[1][2] : c[0][2], v3 = b & 4 ? c[1][3] : c[0][3];
            const float w0 = b & 2 ? v2 : v0, w1 = b & 2 ? v3 : v1;
            const uint32_t x0 = b & 4 ? xn[2] : xn[0], x1 = b & 4 ? xn[3] : xn[1];
            const uint32_t qid = lds32(qid_a + (slot + (b & 1)) * 4);
            const int32_t l2 = static_cast<int32_t>(b & 2 ? x1 : x0) +
                               __float2int_rn((b & 1 ? w1 : w0) * (-2.0f / kScale));
            if (at < A.rec_cap) rec[at] = make_uint4(qid, static_cast<uint32_t>(l2), row + 8 * (b >> 1), d1.z);
            else atomicOr(A.qcount + qid, kDropped);
            ++at;
          } while (mask);
        }
      };
      bool ok = true;
      for (uint32_t t = t0 + warp; ok && t < t1; t += kScoreWarps) {
        while (t >= c_end) {  // on to the slab's item, handing back those before it
          __syncwarp();       // every lane has done with the item's queries
          if (c_n && lane == 0) tc::mbar_arrive(b_empty_a + c_bf * 8);
          c_bf = c_bf + 1 == nB ? 0 : c_bf + 1;
          c_ph ^= c_bf == 0;
          ++c_n;
          // rows are fetched as soon as their item is described
          if (!wait_for(b_full_a + c_bf * 8, c_ph, pw[1], [&](uint32_t x, uint32_t p) {
                fetch();
                return __all_sync(0xffffffffu, tc::mbar_test(x, p)) != 0;
              })) {
            ok = false;
            break;
          }
          d0 = lds128(desc_a + c_bf * kTcDesc);
          d1 = lds128(desc_a + c_bf * kTcDesc + 16);
          c_end = d0.y;
          // the fetch side never falls behind: a buffer handed back may
          // already describe a later item
          if (i_n < c_n) {
            i_n = c_n, i_bf = c_bf, i_ph = c_ph, i_end = d0.y;
            i_row = d0.z - d0.x * kTcSlab, i_nch = d1.y, i_pairs = (i_nch + 1) / 2;
          }
        }
        if (!ok) break;
        if (inflight == 0) fetch();
        const uint32_t ng = (d1.x + 7) / 8;
        const uint32_t first = (t - d0.x) * kTcSlab, row = d0.z + first + g;
        const int32_t left = static_cast<int32_t>(d0.w - first) - static_cast<int32_t>(g);
        const uint32_t bq = b_a + c_bf * btile, slot = c_bf * N;
        const uint32_t nch = d1.y;
        const bool two = d0.w - first > kTcBoxRows;  // the slab's second half has rows
        // one chunk: a stage is the slab's two halves, and the second is left
        // out of a slab without it; several: two chunks of a half
        const uint32_t halves = nch == 1 && !two ? 1 : 2;
        uint32_t box = 0, half = 0;
        uint32_t xn[4];
        float xh[4];
        // the half's 32 rows against groups g0 .. g0 + kG - 1. A group past the
        // first ones meets the same rows again (one chunk then: N = 64 only
        // with h <= 128)
        auto score = [&](auto kg, uint32_t g0) -> bool {
          constexpr uint32_t kG = decltype(kg)::value;
          float c[kG][2][4];
#pragma unroll
          for (uint32_t gr = 0; gr < kG; ++gr)
#pragma unroll
            for (uint32_t m = 0; m < 2; ++m)
#pragma unroll
              for (uint32_t e = 0; e < 4; ++e) c[gr][m][e] = 0.0f;
          for (uint32_t ch = 0;;) {
            if (g0 == 0) {
              if (box == 0 && !wait(bar + cs * 8, cph, pw[0])) return false;
              read(ring + cs * kStage + box * kBox);
              box = box || (nch == 1 ? halves == 1 : ch + 1 == nch) ? 0 : 1;
              if (box == 0) release();
            }
#pragma unroll
            for (uint32_t s = 0; s < 2 * NI; ++s) step(kg, s, bq + g0 * 8 * brow + ch * IN * 2, c);
            // the last chunk may hold 64 dimensions only
            if (g0 == 0 && ((ch + 1) * IN <= h || ch * IN + tig * (IN / 4) < h)) norms(xn);
            if (++ch == nch) break;
          }
          if (g0 == 0) finish(xn, xh, left - static_cast<int32_t>(kTcBoxRows * half));
#pragma unroll
          for (uint32_t gr = 0; gr < kG; ++gr)
            test(c[gr], xh, xn, slot + (g0 + gr) * 8, row + kTcBoxRows * half);
          return true;
        };
#pragma unroll 1
        for (; ok && half < halves; ++half) {
          xn[0] = xn[1] = xn[2] = xn[3] = 0;
          // a body for each count of groups: guarding every step of one for
          // four costs 42 cycles of the 150 that two groups take
#pragma unroll 1
          for (uint32_t g0 = 0; ok && g0 < ng; g0 += 4) {
            const uint32_t n = ng - g0;
            ok = n >= 4   ? score(std::integral_constant<uint32_t, 4>{}, g0)
                 : n == 1 ? score(std::integral_constant<uint32_t, 1>{}, g0)
                 : n == 2 ? score(std::integral_constant<uint32_t, 2>{}, g0)
                          : score(std::integral_constant<uint32_t, 3>{}, g0);
          }
        }
        if (!ok) break;
        if (IN == 128 && lane == 0) atomicAdd(slabs, 1u);
      }
      // hand back the remaining items' buffers, so that the staging warps end
      __syncwarp();
      while (ok && !warp_read(err)) {
        if (c_n && lane == 0) tc::mbar_arrive(b_empty_a + c_bf * 8);
        if (++c_n > n_li) break;
        c_bf = c_bf + 1 == nB ? 0 : c_bf + 1;
        c_ph ^= c_bf == 0;
        ok = wait(b_full_a + c_bf * 8, c_ph, pw[1]);
      }
      // copies still in flight land before the CTA exits
      for (; inflight; --inflight) {
        for (uint32_t i = 0; i < (1u << 26) && !tc::mbar_try(bar + cs * 8, cph); ++i) {
        }
        if (++cs == depth) cs = 0, cph ^= 1;
      }
    } else {
      // ---- query staging: warp sw takes the CTA's items sw, sw + nB, ...
      const uint32_t sw = warp - kScoreWarps;
      const uint32_t b0 = tc::smem_addr(sm + L.b + sw * btile);
      if (sw < nB) {
        // loads run ahead: an item's queries while the one before it is
        // copied, the description of the one after while both are
        auto item_at = [&](uint32_t li) { return li < n_li ? A.items[it0 + li] : TcItem{0, 0, 0, 0}; };
        auto slab_at = [&](uint32_t li) { return li <= n_li ? A.tile_off[it0 + li] : 0u; };
        auto entry = [&](const TcItem &it, uint32_t j) { return j < it.ne ? A.entries[it.e0 + j] : 0u; };
        TcItem cur = item_at(sw), nxt = item_at(sw + nB);
        uint32_t s0 = slab_at(sw), s1 = slab_at(sw + 1);
        uint32_t staged = 0;  // filtered pairs of the buffer's item
        uint32_t q0 = entry(cur, lane) / A.nprobe, q1 = entry(cur, lane + 32) / A.nprobe;
        for (uint32_t li = sw, use = 0; li < n_li; li += nB, ++use) {
          const uint32_t e0 = entry(nxt, lane), e1 = entry(nxt, lane + 32);
          const uint32_t n0 = slab_at(li + nB), n1 = slab_at(li + nB + 1);
          const TcItem nxt2 = item_at(li + 2 * nB);
          const int2 cn0 = A.qcn[q0], cn1 = N > 32 ? A.qcn[q1] : make_int2(0, 0);
          const int32_t bd0 = A.bound[q0], bd1 = N > 32 ? A.bound[q1] : 0;
          // (rows of 64 dimensions are never filtered)
          bool filt = IN == 128 && A.f < h && cur.nrows * cur.ne <= 2 * A.rec_cap;
          // pairs of the item's rows that are the CTA's
          const uint32_t rows = min(cur.nrows, (min(s1, t1) - s0) * kTcSlab) - (max(s0, t0) - s0) * kTcSlab;
          const uint32_t pairs = filt ? rows * cur.ne : 0;
          if (!wait(b_empty_a + sw * 8, (use & 1) ^ 1, pw[0])) break;
          // Filtered while few records come of it. A slab saves about 0.15 us
          // of an SM against all of h = 256, and completing a record costs an
          // SM about 5 ns: on while the CTA's slabs gave below 16 each, whatever
          // their items were (10M x 1,024 of one spread-out cloud: 3 per slab,
          // 0.50 ms against 0.71; of tight clusters, 20 and more, 1.16 ms with
          // its records for 1.30 with 32 as the line and 1.07 without a
          // filter). The first items go ahead, those after 8 slabs await their count.
          // Partial records must leave the CTA's list room (whoever's records
          // do not fit is rescanned): an eighth of an item's pairs may pass,
          // which keeps a server's batches of a hundred or so off long lists
          // (400k searches/s at 10M: p99 8.4 -> 4.2 ms; with half the pairs, the
          // 384-probe batches' long lists went unfiltered, 245 -> 265 us). And the
          // pairs in the other buffers with this item's have to fit into what is left
          // of it, but for an eighth: all of them, or at twice the records there were
          // so far to a filtered pair (a flat spectrum, 512 queries of 16 lists,
          // h = 512: 243 us a search, 806 with rescans)
          if constexpr (IN == 128) {
            if (lane == 0) {
              // (four accesses in flight together: 10M x 1,024 493.9 us, one after
              // another 495.7; without the room's rule 490.8, and 2,000 queries of
              // 2M x 768, whose first items do not all fit, 242 for 248)
              const uint32_t have = *static_cast<volatile uint32_t *>(rcount);
              const uint32_t scored = *static_cast<volatile uint32_t *>(slabs);
              // this buffer's last item has been scored
              const uint32_t seen = atomicAdd(fpairs, staged) + staged;
              const uint32_t ahead = atomicAdd(fstaged, pairs) + pairs - seen;
              const uint32_t room = A.rec_cap / 8 * 7 - have;  // have is a quarter at most
              filt = filt && have <= min(scored >= 8 ? 16 * scored : ~0u, A.rec_cap / 4) &&
                     (ahead <= room || (seen && 2ull * have * ahead <= static_cast<uint64_t>(room) * seen));
              staged = filt ? pairs : 0;
              if (pairs != staged) atomicSub(fstaged, pairs);
            }
            filt = __shfl_sync(0xffffffffu, filt, 0);
          }
          const uint32_t dims = filt ? A.f : h;
          if (lane == 0) {
            desc[sw] = Desc{s0, s1, cur.row0, cur.nrows, cur.ne, (dims + IN - 1) / IN, filt, 0};
            tc::mbar_arrive(d_full + sw);
          }
          // the queries' fp16 rows, `per` 16-byte units each, the ids shuffled
          const uint32_t per = (dims + IN - 1) / IN * (IN / 8), steps = (cur.ne * per + 31) / 32;
          uint32_t j = lane / per, u = lane % per;
          for (uint32_t i = 0; i < steps; ++i) {
            const uint32_t ql = __shfl_sync(0xffffffffu, q0, j & 31);
            const uint32_t qh = N > 32 ? __shfl_sync(0xffffffffu, q1, j & 31) : 0;
            if (j < cur.ne) {
              const uint32_t pos = IN == 128 ? (u ^ ((u >> 3) & 1) ^ ((j & 1) << 1)) : (u ^ (j & 1));
              cp_async16(b0 + j * brow + pos * 16,
                         A.qr16 + static_cast<size_t>(j < 32 ? ql : qh) * (brow / 2) + u * 8);
            }
            for (u += 32; u >= per; u -= per) ++j;
          }
#pragma unroll
          for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t slot = lane + 32 * k;
            if (slot < N) {
              // a slot without a query never passes (its row of the buffer may
              // hold any bits, infinities among them)
              const int2 cn = k ? cn1 : cn0;
              const float qb = static_cast<float>(static_cast<int64_t>(filt ? cn.x : cn.y) - (k ? bd1 : bd0));
              qids[sw * N + slot] = k ? q1 : q0;
              qbv[sw * N + slot] = slot < cur.ne ? qb * (0.5f * kScale) : NAN;
            }
          }
          cp_async_arrive(b_full + sw);
          tc::mbar_arrive(b_full + sw);
          cur = nxt, nxt = nxt2, s0 = n0, s1 = n1;
          q0 = e0 / A.nprobe, q1 = e1 / A.nprobe;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
      }
    }
  }
  if (A.prof && lane == 0 && (warp == 0 || warp == kScoreWarps)) {
    // slots: first scoring warp's waits for rows, for items, its total; first
    // staging warp's wait for a buffer, its total
    const int base = warp == 0 ? 0 : 12;
    atomicAdd(A.prof + base, pw[0]);
    if (warp == 0) atomicAdd(A.prof + 1, pw[1]);
    atomicAdd(A.prof + base + (warp == 0 ? 2 : 1), static_cast<unsigned long long>(clock64() - tstart));
  }
  __syncthreads();
  if (tid == 0) {
    if (*err) atomicAdd(A.timeouts, 1u);
    A.rec_n[blockIdx.x] = min(*rcount, A.rec_cap);
    // the longest CTA (cycles): against the average it shows the schedule's imbalance
    if (A.prof) atomicMax(A.prof + 15, static_cast<unsigned long long>(clock64() - tstart));
  }
}

// ------------------------------------------------------------- seed bounds
// One CTA per query. It looks at the first `want` rows of the query's probed
// lists (probe order, nearest list first). When there are more than `full` of
// them, a sketch picks the ones to score: the squared distance over the first
// 32 head dimensions (the leading rotated dimensions, which carry most of the
// variance), of which the `full` smallest, and any others in the last one's
// bin, are scored over all h dimensions.
// The bound is the S-th smallest scored l2, widened to L + (L >> 22) + 1: the
// distance value is monotone in l2 and two l2 that far apart never round to
// the same float, so every row whose distance can tie the S-th best is still
// inside. Any S of a query's candidates bound its S-th best from above, so
// the rows the sketch picks change no result, only how tight the bound is
// and how many bytes it costs: 1,024 sketched rows (32 bytes each) and 2S
// scored rows read 4 times fewer bytes than 1,024 scored rows of 256 bytes. Fewer than S rows: no bound.

// sum x (x - 2 q) over 16 bytes: the squared distance less the query's own sum
__device__ __forceinline__ uint32_t sketch16(uint4 x, uint4 q) {
  const uint32_t xx = dp4(x.x, x.x, dp4(x.y, x.y, dp4(x.z, x.z, dp4(x.w, x.w, 0))));
  const uint32_t xq = dp4(x.x, q.x, dp4(x.y, q.y, dp4(x.z, q.z, dp4(x.w, q.w, 0))));
  return xx - 2 * xq;
}

// The bin of half a sketch distance (32 255^2 < 2^21, so half of it is below
// 2^20): 32 bins per power of two, so that one histogram of 512 bins resolves
// every distance to 3%.
constexpr uint32_t kSketchBins = 512;
__device__ __forceinline__ uint32_t sketch_bin(uint32_t d) {
  if (d < 32) return d;
  const uint32_t e = 31 - __clz(d);
  return (e - 4) * 32 + ((d >> (e - 5)) & 31);
}

// The sketch loads bound it: 32-byte pieces of rows h or more bytes apart. Two
// lanes to a row halve the L1's work (2,048 rows: 148 -> 127 us for 4096 queries
// at 1M; the squares as x (x - 2 q) by dp4a instead of a byte-wise difference
// among it), eight of them are in flight to a thread; at 10M it is the DRAM's, and
// more CTAs on an SM than three slow it down (206, 254, 276 us at three, four,
// five). The rest is a chain of latencies, kept short: offsets read 32 lists at a
// time, keys kept in registers, one histogram for the picked bin, and a last
// selection that ranks by counting where there are few.
__global__ void __launch_bounds__(256, 3) rank_seed_kernel(
    const uint8_t *__restrict__ xhi, const int64_t *__restrict__ xnorm,
    const uint8_t *qhi, const int64_t *qnorm, const uint32_t *probed, const uint32_t *qprobes,
    const uint32_t *__restrict__ list_off, uint32_t p,
    uint32_t dc, uint32_t h, uint32_t S, uint32_t want, uint32_t more, SeedBound kind, DistScale scale,
    int32_t *bound) {
  after_previous();
  // rowof: the rows looked at. Where all are scored, l2s gets their distances;
  // where some are, l2s gets those rows and rowof their distances.
  __shared__ __align__(16) uint32_t rowof[kSeedCap];
  __shared__ __align__(16) uint32_t l2s[kSeedCap];
  __shared__ __align__(16) uint32_t qw[2048 / 4];
  __shared__ uint32_t hist[kSketchBins], sel[2], wsum[8], npick;
  const uint32_t q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint32_t i = tid; i < h / 4; i += 256)
    qw[i] = reinterpret_cast<const uint32_t *>(qhi + static_cast<size_t>(q) * dc)[i];
  for (uint32_t i = tid; i < kSketchBins; i += 256) hist[i] = 0;
  if (tid == 0) npick = 0;
  // the rows, 32 lists at a time: every warp reads their offsets, and writes
  // the rows of every eighth
  const uint32_t pq = qprobes ? qprobes[q] : p;  // the query's own budget
  uint32_t count = 0, full = min(want, 2 * S);
  for (uint32_t r = 0; r < pq && count < want; r += 32) {
    uint32_t r0 = 0, n = 0;
    if (r + lane < pq) {
      const uint32_t c = probed[static_cast<size_t>(q) * p + r + lane];
      r0 = list_off[c];
      n = list_off[c + 1] - r0;
    }
    if (r == 0) {
      // rows that the query probes, by its nearest lists: of many the bound
      // lets more through, and more rows are looked at (default_seed_rows)
      const uint32_t lists = min(pq, 32u), rows = __reduce_add_sync(0xffffffffu, min(n, 1u << 20));
      if (static_cast<uint64_t>(rows) * pq > static_cast<uint64_t>(kSeedMany) * lists) {
        want = more;
        full = min(want, 3 * S);
      }
    }
    uint32_t incl = min(n, want);  // (sums stay below 32 want)
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t at = count + incl - min(n, want), total = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t l = warp; l < 32; l += 8) {
      const uint32_t first = __shfl_sync(0xffffffffu, at, l), row = __shfl_sync(0xffffffffu, r0, l);
      const uint32_t rows = __shfl_sync(0xffffffffu, n, l);
      if (first >= want) break;
      const uint32_t m = min(rows, want - first);
      for (uint32_t i = lane; i < m; i += 32) rowof[first + i] = row + i;
    }
    count = min(want, count + total);
  }
  __syncthreads();
  if (count < S) {
    if (tid == 0) bound[q] = 0x7FFFFFFF;
    return;
  }
  uint32_t n = count;
  const uint32_t *rows = rowof;
  uint32_t *l2 = l2s;
  if (count > full) {
    // Every row in or below the bin of the full-th smallest sketch distance is
    // scored: at least `full`, a few more when the bin holds several. Two lanes
    // read a row's 32 bytes, which is one line of a load's 32 for each pair
    // instead of one for each lane; even lanes keep the rows of the even loads,
    // odd lanes those of the odd ones: row 32 (8 j + warp) + 16 (lane & 1) +
    // lane / 2 is key j.
    constexpr uint32_t kPer = kSeedCap / 256;
    const uint32_t odd = lane & 1;
    const uint4 qv = reinterpret_cast<const uint4 *>(qw)[odd];
    const uint32_t qq = dp4(qv.x, qv.x, dp4(qv.y, qv.y, dp4(qv.z, qv.z, dp4(qv.w, qv.w, 0))));
    const uint32_t q2 = qq + __shfl_xor_sync(0xffffffffu, qq, 1);
    const uint32_t r0 = 32 * warp + lane / 2, mine0 = r0 + 16 * odd;
    uint32_t bins[kPer / 2];  // two 16-bit bins to a word
#pragma unroll
    for (uint32_t j0 = 0; j0 < kPer; j0 += 4) {
      if (j0 * 256 >= count) break;
      uint4 v[8];
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) {
        const uint32_t i = (j0 + j / 2) * 256 + r0 + 16 * (j & 1);
        v[j] = __ldg(reinterpret_cast<const uint4 *>(xhi + static_cast<size_t>(rowof[min(i, count - 1)]) * dc) + odd);
      }
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t t0 = sketch16(v[2 * j], qv), t1 = sketch16(v[2 * j + 1], qv);
        const uint32_t d2 = q2 + (odd ? t1 : t0) + __shfl_xor_sync(0xffffffffu, odd ? t0 : t1, 1);
        const uint32_t bin = sketch_bin(d2 / 2);
        if ((j0 + j) * 256 + mine0 < count) atomicAdd(&hist[bin], 1u);
        if (j & 1) bins[(j0 + j) / 2] |= bin << 16;
        else bins[(j0 + j) / 2] = bin;
      }
    }
    __syncthreads();
    // the bin of rank full - 1: thread t has bins 2 t and 2 t + 1
    const uint32_t ha = hist[2 * tid], hb = hist[2 * tid + 1];
    uint32_t incl = ha + hb;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t below = incl - ha - hb;
    for (uint32_t w = 0; w < warp; ++w) below += wsum[w];
    if (full - 1 >= below && full - 1 < below + ha + hb) sel[0] = 2 * tid + (full - 1 >= below + ha);
    __syncthreads();
    const uint32_t last = sel[0];
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
      if (j * 256 >= count) break;
      const bool take = j * 256 + mine0 < count && ((bins[j / 2] >> (16 * (j & 1))) & 0xFFFFu) <= last;
      const uint32_t votes = __ballot_sync(0xffffffffu, take);
      uint32_t at = 0;
      if (lane == 0 && votes) at = atomicAdd(&npick, __popc(votes));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(votes & ((1u << lane) - 1));
      if (take) l2s[at] = rowof[j * 256 + mine0];
    }
    __syncthreads();
    n = npick;
    rows = l2s;
    l2 = rowof;
  }
  const int64_t qn = qnorm[q];
  for_rows_at(
      xhi, dc, h, qw, [&](uint32_t i) { return rows[i]; }, n,
      [&](uint32_t i, uint32_t dot, int64_t xn) {
        l2[i] = static_cast<uint32_t>(qn + xn - 2 * static_cast<int64_t>(dot));
      },
      [&](uint32_t i) { return xnorm[rows[i]]; });
  // the S-th smallest
  uint32_t L2 = 0;
  bool have = false;
  if (n <= 256) {
    if (tid >= n && tid < (n + 3) / 4 * 4) l2[tid] = 0xFFFFFFFFu;
    __syncthreads();
    const uint32_t v = l2[min(tid, n - 1)];
    uint32_t lt = 0, le = 0;
    for (uint32_t j = 0; j < n; j += 4) {
      const uint4 o = *reinterpret_cast<const uint4 *>(l2 + j);
      lt += (o.x < v) + (o.y < v) + (o.z < v) + (o.w < v);
      le += (o.x <= v) + (o.y <= v) + (o.z <= v) + (o.w <= v);
    }
    L2 = v;
    have = tid < n && lt < S && S <= le;  // equal values: each of them says the same
  } else {
    __syncthreads();
    // radix selection by 8-bit digits (l2 < 255^2 h: no top digit for h up to 258)
    uint32_t prefix = 0, rank = S - 1;
    for (int shift = h * 65025u < (1u << 24) ? 16 : 24; shift >= 0; shift -= 8) {
      if (tid < 256) hist[tid] = 0;
      __syncthreads();
      const uint32_t hm = shift == 24 ? 0u : (0xFFFFFFFFu << (shift + 8));
      for (uint32_t i = tid; i < n; i += 256)
        if ((l2[i] & hm) == prefix) atomicAdd(&hist[(l2[i] >> shift) & 0xFFu], 1u);
      __syncthreads();
      block_pick_digit(hist, rank, sel, wsum);
      rank -= sel[1];
      prefix |= sel[0] << shift;
      __syncthreads();
    }
    L2 = prefix;
    have = tid == 0;
  }
  if (have) {
    const int32_t v = static_cast<int32_t>(L2);
    if (kind == SeedBound::kRanking) {
      bound[q] = v + (v >> 22) + 1;
    } else {
      // as the bits of a distance. For exact distances over all h dimensions:
      // codes whose high bytes differ by e differ by at most 256 e + 255, and
      // the sum of e is at most sqrt(h sum e^2)
      int64_t u = v;
      if (kind == SeedBound::kExactKey)
        u = 65536ll * v + 65025ll * h + 1 +
            static_cast<int64_t>(130560.0 * sqrt(static_cast<double>(h) * static_cast<double>(v)));
      bound[q] = __float_as_int(dist_value(u, scale));
    }
  }
}

constexpr uint32_t kBucketCtas = 8;

// The pass's candidate records (query, xn - 2 dot, row, partial) into per-query
// buffers of (distance bits, row); kBucketCtas CTAs share each ranking CTA's
// list, so that enough records (each a global atomic and a scattered store)
// are in flight per SM; those without records leave after one load (2M x 768,
// 64 lists, with eight CTAs and with one: 1 query 78.5 and 78.3 us a search, 64 142 and
// 147, 511 226 and 243, 1,024 318 and 355). A partial record covers the first f dimensions:
// eight lanes add the rest, 16 bytes of the row and of the query each, with
// the loads of a warp's 32 records in flight together.
__global__ void __launch_bounds__(256) tc_bucket_kernel(
    const uint4 *rec, const uint32_t *rec_n, uint32_t rec_cap, const uint8_t *__restrict__ xhi,
    const uint8_t *qhi, const int2 *qcn, const int32_t *bound, uint32_t dc, uint32_t f, uint32_t h,
    uint32_t *qcount, uint2 *qbuf, uint32_t cap, DistScale scale, unsigned long long *found) {
  after_previous();
  const uint4 *r = rec + static_cast<size_t>(blockIdx.x) * rec_cap;
  const uint32_t n = rec_n[blockIdx.x], lane = threadIdx.x & 31, grp = lane >> 3, gl = lane & 7;
  const uint32_t nw = gridDim.y * (blockDim.x >> 5);
  uint32_t kept = 0;
  for (uint32_t i0 = (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; i0 < n;
       i0 += nw * 32) {
    const bool valid = i0 + lane < n;
    const uint4 e = valid ? r[i0 + lane] : make_uint4(0, 0, 0, 0);
    const int2 cn = valid ? qcn[e.x] : make_int2(0, 0);
    int32_t l2 = static_cast<int32_t>(e.y) + (e.w ? cn.x : cn.y);
    if (__any_sync(0xffffffffu, e.w != 0)) {
      uint32_t tail = 0;
      for (uint32_t u0 = f / 16; u0 < h / 16; u0 += 8) {
        const bool in = u0 + gl < h / 16;
        uint4 x[8], q[8];
#pragma unroll
        for (uint32_t it = 0; it < 8; ++it) {
          const uint32_t src = it * 4 + grp;
          const uint32_t eq = __shfl_sync(0xffffffffu, e.x, src), er = __shfl_sync(0xffffffffu, e.z, src);
          const bool on = __shfl_sync(0xffffffffu, e.w, src) != 0 && in;
          x[it] = on ? __ldg(reinterpret_cast<const uint4 *>(xhi + static_cast<size_t>(er) * dc) + u0 + gl)
                     : make_uint4(0, 0, 0, 0);
          q[it] = on ? reinterpret_cast<const uint4 *>(qhi + static_cast<size_t>(eq) * dc)[u0 + gl]
                     : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (uint32_t it = 0; it < 8; ++it) {
          const uint32_t a[4] = {x[it].x, x[it].y, x[it].z, x[it].w};
          const uint32_t b[4] = {q[it].x, q[it].y, q[it].z, q[it].w};
          uint32_t sq = 0, xq = 0;
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            sq = dp4(a[w], a[w], dp4(b[w], b[w], sq));
            xq = dp4(a[w], b[w], xq);
          }
          uint32_t d2 = sq - 2 * xq;
#pragma unroll
          for (uint32_t o = 1; o < 8; o <<= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, o);
          const uint32_t t = __shfl_sync(0xffffffffu, d2, (lane & 3) * 8);
          if (lane >> 2 == it) tail += t;
        }
      }
      l2 += static_cast<int32_t>(tail);
    }
    const bool keep = valid && l2 <= bound[e.x];
    kept += __popc(__ballot_sync(0xffffffffu, keep));
    if (keep) {
      const uint32_t at = atomicAdd(qcount + e.x, 1u) & ~kDropped;
      if (at < cap)
        qbuf[static_cast<size_t>(e.x) * cap + at] =
            make_uint2(__float_as_uint(dist_value(l2, scale)), e.z);
    }
  }
  if (lane == 0 && kept) atomicAdd(found, static_cast<unsigned long long>(kept));
}

}  // namespace

uint32_t rank_tc_ctas() {
  int sms = 0;
  if (current_sms(&sms) != KATO_OK) sms = 1;
  return static_cast<uint32_t>(std::max(sms, 1));
}

std::atomic<uint32_t> g_tc_width{0}, g_tc_beta{0};
std::atomic<unsigned long long> g_tc_wait{0};

bool rank_tc_plan(uint32_t h, uint32_t dc, bool rotated, TcShape *s) {
  if (h == 0 || h % 64 || h > 1024 || h > dc || dc % 64) return false;
  TcShape t{};
  // items narrow as the queries' rows widen, so that several query buffers fit
  t.N = h <= 128 ? 64 : (h <= 512 ? 32 : 16);
  const uint32_t cap = g_tc_width.load();
  if (cap >= 16 && cap < t.N) t.N = cap;
  t.inner = h == 64 ? 64 : 128;
  // without a rotation the leading dimensions are like any others: nearly every
  // pair passes on 128 of them, and what does not fit the lists is rescanned
  // (high bytes of 300k flat vectors, 512 queries of 33 lists, without the filter
  // and with it: 576 dimensions 222 and 594 us, 1,024 291 and 625; where they
  // decay as i^-1, 832 dimensions 277 and 296, 320 151 and 146)
  t.f = rotated ? std::min(h, kTcFilterDims) : h;
  t.centred = h > 256;
  constexpr uint32_t shapes[][2] = {{4, 4}, {4, 2}, {3, 2}, {2, 2}, {1, 2}};
  for (const auto &b : shapes) {
    t.Bs = b[0];
    t.Rs = b[1];
    t.smem = tc_smem_layout(h, t).total;
    if (t.smem <= 227 * 1024) {
      *s = t;
      return true;
    }
  }
  return false;
}

int rank_tc(const RankTcArgs &A, const uint8_t *xhi, uint32_t npts, const TcShape &s,
            cudaStream_t st) {
  const PFN_cuTensorMapEncodeTiled_v12000 encode = tc::tensor_map_encoder();
  if (!encode) return cuda_status(cudaErrorNotSupported, "cuTensorMapEncodeTiled");
  // the high-byte plane as a 2-D tensor of bytes: x = byte in row, y = row
  CUtensorMap tmap;
  const cuuint64_t dims[2] = {A.dc, npts};
  const cuuint64_t strides[1] = {A.dc};
  const cuuint32_t box[2] = {s.inner, kTcBoxRows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult cr = encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t *>(xhi), dims,
                             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             s.inner == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                             s.inner == 128 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B
                                            : CU_TENSOR_MAP_L2_PROMOTION_L2_64B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed for the high-byte plane (error " + std::to_string(cr) + ")");
    return KATO_ERUNTIME;
  }
  const uint32_t ctas = rank_tc_ctas();
  auto go = [&](auto kern) -> int {
    if (const int rc = smem_limit(reinterpret_cast<const void *>(kern), static_cast<int>(s.smem),
                                  "rank_tc_kernel shared memory"))
      return rc;
    launch(kern, ctas, kTcThreads, s.smem, st, tmap, A, s);
    KATO_LAUNCHED("rank_tc_kernel");
    return KATO_OK;
  };
  if (s.inner == 64) return go(rank_tc_kernel<64, false>);
  return s.centred ? go(rank_tc_kernel<128, true>) : go(rank_tc_kernel<128, false>);
}

int rank_tc_bucket(const uint4 *rec, const uint32_t *rec_n, uint32_t rec_cap, uint32_t ctas,
                   const uint8_t *xhi, const uint8_t *qhi, const int2 *qcn, const int32_t *bound,
                   uint32_t dc, uint32_t f, uint32_t h, uint32_t *qcount, uint2 *qbuf, uint32_t cap,
                   DistScale scale, unsigned long long *found, cudaStream_t st) {
  launch(tc_bucket_kernel, dim3(ctas, kBucketCtas), 256, 0, st, rec, rec_n, rec_cap, xhi, qhi, qcn, bound, dc, f, h,
                                                  qcount, qbuf, cap, scale, found);
  KATO_LAUNCHED("tc_bucket_kernel");
  return KATO_OK;
}

int rank_seed(const uint8_t *xhi, const int64_t *xnorm, const uint8_t *qhi, const int64_t *qnorm,
              const uint32_t *probed, const uint32_t *qprobes, const uint32_t *list_off, uint32_t B,
              uint32_t p, uint32_t dc, uint32_t h, uint32_t S, uint32_t rows, SeedBound kind,
              DistScale scale, int32_t *bound, cudaStream_t st) {
  if (h > 2048 || h % 64) return invalid("seed bounds need h <= 2048, a multiple of 64");
  if (B == 0) return KATO_OK;
  // `rows` for a query of few rows, twice as many for one of many
  const uint32_t want = std::min(std::max(rows, S), kSeedCap);
  const uint32_t more = std::min(std::max(2 * rows, S), kSeedCap);
  launch(rank_seed_kernel, B, 256, 0, st, xhi, xnorm, qhi, qnorm, probed, qprobes, list_off, p, dc, h,
                                      S, want, more, kind, scale, bound);
  KATO_LAUNCHED("rank_seed_kernel");
  return KATO_OK;
}

}  // namespace kato
