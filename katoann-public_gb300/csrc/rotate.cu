// Rotation and 16-bit coding of rows on the GPU, bit-identical to the
// reference's float arithmetic.
//
// The reference computes every rotated value out[i][j] = <x_i, r_j> with 16
// lane accumulators: lane l sums x[k] * r[k] over k = l, l + 16, ... by fused
// multiply-add in k order, the 16 lanes are added as (l, l+8), (l, l+4),
// (l, l+2), (0, 1), and the last d % 16 dimensions follow one by one
// (src/index.cpp:139-208). Here 16 consecutive threads of a warp play the 16
// lanes: each thread keeps the lane sums of a block of outputs, and the lane
// reduction is a butterfly of shuffles (8, 4, 2, 1), which adds the same pairs
// in the same order, so every output ends with the reference's bits. The scalar parts are replayed with explicit rounding: the reference's
// compiler evaluates those chains four products at a time with the products
// rounded, then fuses the last (length % 4) terms.
#include "kcommon.cuh"
#include "rank_tc.cuh"
#include "tc.cuh"

namespace kato {

namespace {

constexpr int kRotRows = 32;     // output rows per CTA
constexpr int kRotCols = 32;     // output columns per CTA
constexpr int kRotK = 64;        // k-chunk staged in shared memory
constexpr int kRotStride = 36;   // floats per staged k (rows/columns 0..31 + pad: 16-byte
                                 // aligned and conflict-free for 128-bit reads)

// Scalar tail of one output: dimensions [k0, d), the first ((d - k0) & ~3) of
// them with rounded products, the rest fused.
__device__ __forceinline__ float rot_tail(float s, const float *x, const float *r, uint32_t k0,
                                          uint32_t d) {
  const uint32_t m = k0 + ((d - k0) & ~3u);
  uint32_t k = k0;
  for (; k < m; ++k) s = __fadd_rn(s, __fmul_rn(x[k], r[k]));
  for (; k < d; ++k) s = __fmaf_rn(x[k], r[k], s);
  return s;
}

// 4-byte asynchronous global -> shared copy; src_bytes 0 writes a zero.
__device__ __forceinline__ void cp_async4(float *dst, const float *src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(src_bytes)
               : "memory");
}

// Lane reduction as a reduce-scatter: at each step (lane distance 8, 4, 2, 1)
// a lane keeps half of its NV outputs and adds its partner's partial sums of
// them. Every output meets the same pairs in the same order as in the
// reference's horizontal add (IEEE addition is commutative). Lane l ends with
// the NV / 16 outputs from the returned one on: against an all-reduce a quarter
// of the shuffles, and no spills.
template <int NV>
__device__ __forceinline__ int lane_scatter(float (&v)[NV], int l) {
#pragma unroll
  for (int step = 0, half = NV / 2, m = 8; step < 4; ++step, half >>= 1, m >>= 1) {
    const bool hi = (l & m) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = hi ? v[i] : v[i + half];
      const float keep = hi ? v[i + half] : v[i];
      v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, m));
    }
  }
  return ((l >> 3) & 1) * (NV / 2) + ((l >> 2) & 1) * (NV / 4) + ((l >> 1) & 1) * (NV / 8) +
         (l & 1) * (NV / 16);
}

// The four outputs of row i from column j on: the scalar tail, then the store.
__device__ __forceinline__ void store_outputs(const float *v, uint32_t i, uint32_t j, uint32_t nrows,
                                              uint32_t d, const float *in, const float *rot,
                                              float *out) {
  if (i >= nrows) return;
  const uint32_t d4 = d & ~3u, d16 = d & ~15u;
  const float *x = in + static_cast<size_t>(i) * d;
  float *o = out + static_cast<size_t>(i) * d + j;
  if (d16 == d && j + 4 <= d4 && (reinterpret_cast<uintptr_t>(o) & 15u) == 0) {
    *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (j + e < d4) o[e] = rot_tail(v[e], x, rot + static_cast<size_t>(j + e) * d, d16, d);
  }
}

// Rows as they are (an index's rows at load): 32 x 32 outputs per CTA, 8 x 8
// per thread, chunks of 64 dimensions copied 4 bytes at a time into a
// double-buffered k-major staging.
__global__ void __launch_bounds__(256, 2) rotate_lanes_kernel(const float *__restrict__ in,
                                                              uint32_t nrows, uint32_t d,
                                                              const float *__restrict__ rot,
                                                              float *__restrict__ out) {
  // two stages, each staged k-major (xs[k][row], rs[k][column]) so that a
  // thread reads its 8 rows and 8 columns at one k with four 128-bit loads;
  // the next chunk is copied asynchronously while the current one is used
  __shared__ __align__(16) float xs[2][kRotK * kRotStride];
  __shared__ __align__(16) float rs[2][kRotK * kRotStride];
  const uint32_t d4 = d & ~3u, d16 = d & ~15u;
  const uint32_t i0 = blockIdx.x * kRotRows, j0 = blockIdx.y * kRotCols;
  const int t = threadIdx.x, l = t & 15, g = t >> 4;
  const int rb = (g >> 2) * 8, cb = (g & 3) * 8;
  float acc[8][8];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[a][b] = 0.0f;

  auto stage = [&](uint32_t k0, int buf) {
    for (int idx = t; idx < kRotRows * kRotK; idx += 256) {
      const int r = idx / kRotK, c = idx % kRotK;
      const uint32_t gk = k0 + c;
      const uint32_t gi = i0 + r, gj = j0 + r;
      const bool okx = gi < nrows && gk < d16, okr = gj < d4 && gk < d16;
      cp_async4(&xs[buf][c * kRotStride + r], okx ? in + static_cast<size_t>(gi) * d + gk : in,
                okx ? 4u : 0u);
      cp_async4(&rs[buf][c * kRotStride + r], okr ? rot + static_cast<size_t>(gj) * d + gk : rot,
                okr ? 4u : 0u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int buf = 0;
  if (d16) stage(0, 0);
  for (uint32_t k0 = 0; k0 < d16; k0 += kRotK, buf ^= 1) {
    if (k0 + kRotK < d16) {
      stage(k0 + kRotK, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const uint32_t kend = min(static_cast<uint32_t>(kRotK), d16 - k0);
    // this lane's dimension of each 16-dimension step: fixed offsets from one
    // base per chunk, the four steps unrolled (kend is a multiple of 16)
    const float *xl = xs[buf] + l * kRotStride + rb, *rl = rs[buf] + l * kRotStride + cb;
#pragma unroll
    for (uint32_t c = 0; c < kRotK; c += 16) {
      if (c < kend) {
        const float4 x0 = *reinterpret_cast<const float4 *>(xl + c * kRotStride);
        const float4 x1 = *reinterpret_cast<const float4 *>(xl + c * kRotStride + 4);
        const float4 r0 = *reinterpret_cast<const float4 *>(rl + c * kRotStride);
        const float4 r1 = *reinterpret_cast<const float4 *>(rl + c * kRotStride + 4);
        const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
        const float rv[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
          for (int b = 0; b < 8; ++b) acc[a][b] = __fmaf_rn(xv[a], rv[b], acc[a][b]);
      }
    }
    __syncthreads();  // the buffer is refilled by the next iteration's copies
  }
  float v[64];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) v[a * 8 + b] = acc[a][b];
  const int at = lane_scatter<64>(v, l);
  store_outputs(v, i0 + rb + at / 8, j0 + cb + at % 8, nrows, d, in, rot, out);
}

// The queries of a search. What bounds it is the FP32 pipe: d^2 products per
// row in the reference's order, so no tensor cores; the same inner loop over
// data already in place reaches 113 of 128 FMA per clock and SM, and 92 with a
// barrier every 32 dimensions. Copying the staged parts with 16-byte cp.async,
// 64 dimensions at a time, left 65: its address arithmetic and the chunk's
// hand-over each cost as much as a third of the products. So the parts come by
// TMA, 128 dimensions to a chunk (64: 12% slower), from thread 0: 128-byte rows
// of the k-major copies, in the 128-byte swizzle, which leaves the 16-byte
// reads of eight consecutive lanes (eight consecutive k) free of bank
// conflicts. Products are packed two columns to an fma.rn.f32x2, which halves
// their issue slots and rounds each as the scalar one does.
//   kRows false: tiles of 32 x 32 outputs, 8 x 16 per thread (96 bytes read per
//     128 products instead of 64 per 64), the queries' k-major copy by TMA too;
//     two CTAs of 128 threads per SM hide each other's hand-overs (one of 256
//     over 32 x 64: 8% slower). With the transpose, 4096 x 1024: 171 us (262
//     before), 4096 x 3072: 1,331 us (2,118);
//   kRows true (few queries): tiles of 8 rows x 32 columns, so that one query
//     spreads over d / 32 CTAs of 64 threads; the CTA transposes its 8 rows
//     into shared memory itself.
constexpr int kRotChunk = 128, kRotStages = 3, kRotAhead = kRotStages - 1;
constexpr uint32_t kRotBox = kRotChunk * 128;  // kRotChunk dimensions x 32 floats
constexpr uint32_t kSlabRows = 8, kSlabStride = 12;  // floats per k: 16-byte reads without conflicts

template <bool kRows>
__host__ __device__ constexpr uint32_t rot_stage_bytes() {
  return kRows ? kRotBox : 2 * kRotBox;
}

template <bool kRows>
__host__ __device__ constexpr int rot_threads() {
  return kRows ? 64 : 128;
}

template <bool kRows>
__global__ void __launch_bounds__(rot_threads<kRows>(), kRows ? 1 : 2)
    rotate_tma_kernel(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tr,
                      const float *__restrict__ in, uint32_t nrows, uint32_t d,
                      const float *__restrict__ rot, float *out, uint32_t *timeouts) {
  after_previous();
  constexpr int TB = kRows ? 8 : 16, CG = kRows ? 4 : 2;
  constexpr uint32_t kStage = rot_stage_bytes<kRows>();
  constexpr uint32_t kRowTile = kRows ? kSlabRows : 32, kColTile = 32;
  constexpr int kWarps = rot_threads<kRows>() / 32;
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char *sm = smraw + ((1024 - (tc::smem_addr(smraw) & 1023u)) & 1023u);
  __shared__ uint64_t full[kRotStages], empty[kRotStages];
  __shared__ volatile uint32_t err;
  const uint32_t d16 = d & ~15u, nk = (d16 + kRotChunk - 1) / kRotChunk;
  // one grid dimension: the second ends at 65,535, two million rows
  const uint32_t across = div_up(d & ~3u, kColTile);
  const uint32_t i0 = blockIdx.x / across * kRowTile, j0 = blockIdx.x % across * kColTile;
  const int t = threadIdx.x, lane = t & 31;
  if (t == 0) {
    for (int s = 0; s < kRotStages; ++s) {
      tc::mbar_init(full + s, 1);
      tc::mbar_init(empty + s, kWarps);
    }
    err = 0;
    tc::fence_barrier_init();
  }
  __syncthreads();
  const int l = t & 15, g = t >> 4;
  const uint32_t rb = kRows ? 0 : (g / CG) * 8, cb = (g % CG) * TB;
  float *slab = reinterpret_cast<float *>(sm + kRotStages * kStage);  // [k][row], kRows only
  // chunk c into its stage, once every warp has read the one before in it
  auto issue = [&](uint32_t c) -> bool {
    const uint32_t s = c % kRotStages, use = c / kRotStages;
    if (use && !tc::mbar_test(tc::smem_addr(empty + s), (use & 1) ^ 1) &&
        !tc::mbar_wait_or(empty + s, (use & 1) ^ 1, &err))
      return false;
    unsigned char *st = sm + s * kStage;
    const int32_t k = static_cast<int32_t>(c * kRotChunk), j = static_cast<int32_t>(j0);
    tc::mbar_expect_tx(full + s, kStage);
    tc::tma_load_2d(st, &tr, j, k, full + s);
    if (!kRows) tc::tma_load_2d(st + kRotBox, &tx, static_cast<int32_t>(i0), k, full + s);
    return true;
  };
  uint32_t issued = 0;  // thread 0's
  bool ok = true;
  if (t == 0)
    for (; issued < nk && issued < kRotAhead; ++issued) issue(issued);
  if (kRows) {
    // thread t takes row t % 8, four dimensions at a time
    const uint32_t r = t % kSlabRows;
    const bool in_rows = i0 + r < nrows;
    const float *x = in + static_cast<size_t>(in_rows ? i0 + r : 0) * d;
    const bool vec = d % 4 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
#pragma unroll 16
    for (uint32_t k = t / kSlabRows * 4; k < d16; k += kWarps * 16) {
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (in_rows) v = vec ? __ldg(reinterpret_cast<const float4 *>(x + k)) : make_float4(x[k], x[k + 1], x[k + 2], x[k + 3]);
      float *o = slab + k * kSlabStride + r;
      o[0] = v.x, o[kSlabStride] = v.y, o[2 * kSlabStride] = v.z, o[3 * kSlabStride] = v.w;
    }
    __syncthreads();
  }
  // this lane's dimension is l of every 16: its 128-byte row of a box, and
  // its 16-byte units where the swizzle put them
  const unsigned char *xo[2], *ro[TB / 4];
#pragma unroll
  for (int u = 0; u < 2; ++u)
    xo[u] = kRows ? reinterpret_cast<const unsigned char *>(slab + l * kSlabStride + 4 * u)
                  : sm + kRotBox + l * 128 + (((rb / 4 + u) ^ (l & 7)) << 4);
#pragma unroll
  for (int u = 0; u < TB / 4; ++u)
    ro[u] = sm + l * 128 + (((cb / 4 + u) ^ (l & 7)) << 4);
  unsigned long long acc[8][TB / 2];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < TB / 2; ++b) acc[a][b] = 0ull;
  uint32_t s = 0, ph = 0;
  for (uint32_t c = 0; c < nk; ++c) {
    if (t == 0 && issued < nk && (ok = issue(issued))) ++issued;
    if (ok && !tc::mbar_test(tc::smem_addr(full + s), ph))
      ok = tc::mbar_wait_or(full + s, ph, &err);
    if (!__all_sync(0xffffffffu, ok)) break;
    // one 16-dimension step: this lane's products of the 8 rows and TB columns
    auto step = [&](uint32_t k) {
      const uint32_t so = s * kStage + k * 128;
      float xv[8];
      unsigned long long rv[TB / 2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float4 v = *reinterpret_cast<const float4 *>(xo[u] + (kRows ? (c * kRotChunk + k) * kSlabStride * 4 : so));
        xv[4 * u] = v.x, xv[4 * u + 1] = v.y, xv[4 * u + 2] = v.z, xv[4 * u + 3] = v.w;
      }
#pragma unroll
      for (int u = 0; u < TB / 4; ++u) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(ro[u] + so);
        rv[2 * u] = v.x, rv[2 * u + 1] = v.y;
      }
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        unsigned long long xx;
        asm("mov.b64 %0, {%1,%1};" : "=l"(xx) : "f"(xv[a]));
#pragma unroll
        for (int b = 0; b < TB / 2; ++b)
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[a][b]) : "l"(xx), "l"(rv[b]));
      }
    };
    if ((c + 1) * kRotChunk <= d16) {  // whole chunks without a test per step
#pragma unroll
      for (uint32_t k = 0; k < kRotChunk; k += 16) step(k);
    } else {
#pragma unroll 1
      for (uint32_t k = 0; c * kRotChunk + k < d16; k += 16) step(k);
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(empty + s);
    if (++s == kRotStages) s = 0, ph ^= 1;
  }
  float v[8 * TB];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < TB / 2; ++b)
      asm("mov.b64 {%0,%1}, %2;" : "=f"(v[a * TB + 2 * b]), "=f"(v[a * TB + 2 * b + 1]) : "l"(acc[a][b]));
  const int at = lane_scatter<8 * TB>(v, l);
  if (!err) {
#pragma unroll
    for (int e = 0; e < TB / 2; e += 4)
      store_outputs(v + e, i0 + rb + at / TB, j0 + cb + at % TB + e, nrows, d, in, rot, out);
  }
  if (t == 0 && err)  // copies still in flight land before the CTA exits
    for (uint32_t c = issued < kRotStages ? 0 : issued - kRotStages; c < issued; ++c)
      tc::mbar_wait(full + c % kRotStages, (c / kRotStages) & 1);
  __syncthreads();
  if (t == 0 && err && timeouts) atomicAdd(timeouts, 1u);
}

// out[k * ld + r] = in[r * d + k] for r < rows (zero for rows <= r < ld),
// k < kn: 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) transpose_pad_kernel(const float *__restrict__ in,
                                                            uint32_t rows, uint32_t d, uint32_t kn,
                                                            float *out, uint32_t ld) {
  after_previous();
  __shared__ float tile[32][33];
  const uint32_t r0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (uint32_t y = ty; y < 32; y += 8) {
    const uint32_t r = r0 + y, k = k0 + tx;
    tile[y][tx] = (r < rows && k < kn) ? in[static_cast<size_t>(r) * d + k] : 0.0f;
  }
  __syncthreads();
  for (uint32_t y = ty; y < 32; y += 8) {
    const uint32_t k = k0 + y, r = r0 + tx;
    if (k < kn && r < ld) out[static_cast<size_t>(k) * ld + r] = tile[tx][y];
  }
}

// The same transpose with 16-byte accesses on both sides (d % 4 == 0, `in`
// 16-byte aligned, ld % 32 == 0): 64 x 64 tiles, four float4 loads and four
// float4 stores per thread.
__global__ void __launch_bounds__(256) transpose_pad4_kernel(const float *__restrict__ in,
                                                             uint32_t rows, uint32_t d, uint32_t kn,
                                                             float *out, uint32_t ld) {
  after_previous();
  __shared__ float tile[64][65];
  const uint32_t r0 = blockIdx.x * 64, k0 = blockIdx.y * 64;
  const uint32_t t = threadIdx.x;
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i) {
    const uint32_t idx = t + 256 * i, rr = idx >> 4, k = k0 + (idx & 15) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (r0 + rr < rows && k < kn)
      v = *reinterpret_cast<const float4 *>(in + static_cast<size_t>(r0 + rr) * d + k);
    float *dst = &tile[rr][(idx & 15) * 4];
    dst[0] = v.x, dst[1] = v.y, dst[2] = v.z, dst[3] = v.w;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i) {
    const uint32_t idx = t + 256 * i, kk = idx >> 4, r = (idx & 15) * 4;
    if (k0 + kk < kn && r0 + r < ld)
      *reinterpret_cast<float4 *>(out + static_cast<size_t>(k0 + kk) * ld + r0 + r) =
          make_float4(tile[r][kk], tile[r + 1][kk], tile[r + 2][kk], tile[r + 3][kk]);
  }
}

// out (kn x ld, k-major) from in (rows x d, row-major), zero-padded rows.
void transpose_pad(const float *in, uint32_t rows, uint32_t d, uint32_t kn, float *out, uint32_t ld,
                   cudaStream_t st) {
  if (d % 4 == 0 && ld % 32 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0)
    launch(transpose_pad4_kernel, dim3(div_up(ld, 64), div_up(kn, 64)), 256, 0, st, in, rows, d, kn, out,
                                                                                ld);
  else
    launch(transpose_pad_kernel, dim3(ld / 32, div_up(kn, 32)), 256, 0, st, in, rows, d, kn, out, ld);
}

// The last d % 4 output columns: one chain over all d dimensions
// (src/index.cpp:171-179, :247-257).
__global__ void rotate_seq_kernel(const float *__restrict__ in, uint32_t nrows, uint32_t d,
                                  const float *__restrict__ rot, float *out) {
  after_previous();
  const uint32_t d4 = d & ~3u, nc = d - d4;
  const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<uint64_t>(nrows) * nc) return;
  const uint32_t i = static_cast<uint32_t>(idx / nc), j = d4 + static_cast<uint32_t>(idx % nc);
  out[static_cast<size_t>(i) * d + j] =
      rot_tail(0.0f, in + static_cast<size_t>(i) * d, rot + static_cast<size_t>(j) * d, 0, d);
}

__global__ void minmax_init_kernel(uint32_t *keys) {
  keys[0] = 0xFFFFFFFFu;  // min
  keys[1] = 0u;           // max
}

__global__ void minmax_kernel(const float *__restrict__ x, size_t n, uint32_t *keys) {
  uint32_t mn = 0xFFFFFFFFu, mx = 0u;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t k = float_order_key(x[i]);
    mn = min(mn, k);
    mx = max(mx, k);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(keys, mn);
    atomicMax(keys + 1, mx);
  }
}

// One warp per row: codes, byte planes (padding zero) and the three norms.
__global__ void quantize_rows_kernel(const float *__restrict__ x, uint32_t nrows, uint32_t d,
                                     uint32_t dc, float lo, double inv_step, uint32_t head,
                                     uint8_t *__restrict__ hi, uint8_t *__restrict__ lop,
                                     int64_t *__restrict__ norm, int64_t *__restrict__ hinorm,
                                     int64_t *__restrict__ headnorm) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
  const QuantScale qs = quant_scale(lo, inv_step);
  for (uint64_t row = warp; row < nrows; row += nwarps) {
    const float *xr = x + row * d;
    uint8_t *hr = hi + row * dc;
    uint8_t *lr = lop + row * dc;
    uint64_t s = 0, sh = 0, s0 = 0;
    for (uint32_t k = lane; k < dc; k += 32) {
      uint32_t v = 0;
      if (k < d) v = quantize1(xr[k], qs);
      const uint32_t vh = v >> 8;
      hr[k] = static_cast<uint8_t>(vh);
      lr[k] = static_cast<uint8_t>(v & 0xFFu);
      s += static_cast<uint64_t>(v) * v;
      sh += vh * vh;
      if (k < head) s0 += vh * vh;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      sh += __shfl_xor_sync(0xffffffffu, sh, o);
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    }
    if (lane == 0) {
      norm[row] = static_cast<int64_t>(s);
      hinorm[row] = static_cast<int64_t>(sh);
      if (headnorm) headnorm[row] = static_cast<int64_t>(s0);
    }
  }
}

// A query's codes and everything the search derives from them, one warp per
// row, four dimensions per lane and step: the byte planes and their norms
// (quantize_rows_kernel's), the centred fp16 planes and term of the coarse
// product and the rows of the ranking pass (centre_planes_kernel's). Also
// clears `zeros` words at `zero` (the inversion's and the candidates' counts).
__global__ void __launch_bounds__(256) query_planes_kernel(const float *x, uint32_t nrows,
                                                           uint32_t d, float lo, double inv_step,
                                                           bool vec, const QueryPlanes P,
                                                           const RankRows rr) {
  after_previous();
  const uint32_t lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.zeros; i += gridDim.x * blockDim.x)
    P.zero[i] = 0;
  if (row >= nrows) return;
  const QuantScale qs = quant_scale(lo, inv_step);
  const float *xr = x + static_cast<size_t>(row) * d;
  uint64_t s = 0;
  uint32_t sh = 0, s0 = 0;
  int32_t ch = 0, cl = 0, rf = 0, rh = 0;  // centred byte sums; the ranking rows' norms
  for (uint32_t k = lane * 4; k < P.dc; k += 128) {
    float f[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (vec && k < d) {
      const float4 v = *reinterpret_cast<const float4 *>(xr + k);
      f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
    }
    uint32_t hw = 0, lw = 0;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      if (k + j >= d) break;  // padding dimensions are 0
      const uint32_t v = quantize1(vec ? f[j] : xr[k + j], qs);
      hw |= (v >> 8) << (8 * j);
      lw |= (v & 0xFFu) << (8 * j);
      s += static_cast<uint64_t>(v) * v;
    }
    const size_t at = static_cast<size_t>(row) * P.dc + k;
    *reinterpret_cast<uint32_t *>(P.hi + at) = hw;
    *reinterpret_cast<uint32_t *>(P.lo + at) = lw;
    const uint32_t h2 = dp4(hw, hw, 0), h1 = dp4(hw, 0x01010101u, 0);
    sh += h2;
    if (k < P.head) s0 += h2;
    if (P.hi16) {
      auto halves = [](uint32_t w, uint32_t bias2) {  // four bytes as fp16 (byte - bias)
        const uint32_t a = __byte_perm(w, 0x64646464u, 0x4140), b = __byte_perm(w, 0x64646464u, 0x4342);
        const __half2 bias = *reinterpret_cast<const __half2 *>(&bias2);
        const __half2 ha = __hsub2(*reinterpret_cast<const __half2 *>(&a), bias);
        const __half2 hb = __hsub2(*reinterpret_cast<const __half2 *>(&b), bias);
        return make_uint2(*reinterpret_cast<const uint32_t *>(&ha), *reinterpret_cast<const uint32_t *>(&hb));
      };
      constexpr uint32_t k1152 = 0x64806480u, k1024 = 0x64006400u;  // pairs of fp16 1152 and 1024
      *reinterpret_cast<uint2 *>(P.hi16 + at) = halves(hw, k1152);
      *reinterpret_cast<uint2 *>(P.lo16 + at) = halves(lw, k1152);
      ch += static_cast<int32_t>(h1) - 512;
      cl += static_cast<int32_t>(dp4(lw, 0x01010101u, 0)) - 512;
      if (rr.rows && k < rr.width) {  // f <= h <= width, multiples of 64
        uint2 r = make_uint2(0, 0);
        if (k < rr.h) {
          r = halves(hw, rr.centred ? k1152 : k1024);
          // sum (b - 128)^2 = sum b^2 - 256 sum b + 4 * 16384
          const int32_t c = static_cast<int32_t>(h2) -
                            (rr.centred ? 256 * static_cast<int32_t>(h1) - 4 * 16384 : 0);
          rh += c;
          if (k < rr.f) rf += c;
        }
        *reinterpret_cast<uint2 *>(rr.rows + static_cast<size_t>(row) * rr.width + k) = r;
      }
    }
  }
  // a chunk that ends past the row meets zeros (the scan multiplies all of it, and
  // the row bytes there are out of range: -128 when centred)
  if (P.hi16 && rr.rows)
    for (uint32_t k = P.dc + lane * 4; k < rr.width; k += 128)
      *reinterpret_cast<uint2 *>(rr.rows + static_cast<size_t>(row) * rr.width + k) = make_uint2(0, 0);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    sh += __shfl_xor_sync(0xffffffffu, sh, o);
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    ch += __shfl_xor_sync(0xffffffffu, ch, o);
    cl += __shfl_xor_sync(0xffffffffu, cl, o);
    rf += __shfl_xor_sync(0xffffffffu, rf, o);
    rh += __shfl_xor_sync(0xffffffffu, rh, o);
  }
  if (lane == 0) {
    P.norm[row] = static_cast<int64_t>(s);
    P.hinorm[row] = sh;
    P.headnorm[row] = s0;
    if (P.hi16) P.term[row] = static_cast<int64_t>(s) - 256 * (65792ll * ch + 257ll * cl) - 16384ll * P.dc * 66049ll;
    if (P.hi16 && rr.rows) rr.norms[row] = make_int2(rf, rh);
  }
}

}  // namespace

int query_planes(const float *x, uint32_t nrows, uint32_t d, float lo, double inv_step,
                 const QueryPlanes &P, const RankRows &rr, cudaStream_t st) {
  if (nrows == 0) return KATO_OK;
  const bool vec = d % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0;
  launch(query_planes_kernel, div_up(nrows, 8), 256, 0, st, x, nrows, d, lo, inv_step, vec, P, rr);
  KATO_LAUNCHED("query_planes_kernel");
  return KATO_OK;
}

int rotate_rows(const float *in, uint32_t nrows, uint32_t d, const float *rot, float *out,
                cudaStream_t st) {
  if (nrows == 0) return KATO_OK;
  const uint32_t d4 = d & ~3u;
  if (d4) {
    dim3 grid(div_up(nrows, kRotRows), div_up(d4, kRotCols));
    rotate_lanes_kernel<<<grid, 256, 0, st>>>(in, nrows, d, rot, out);
    KATO_LAUNCHED("rotate_lanes_kernel");
  }
  if (d4 < d) {
    const uint64_t n = static_cast<uint64_t>(nrows) * (d - d4);
    launch(rotate_seq_kernel, static_cast<uint32_t>((n + 255) / 256), 256, 0, st, in, nrows, d, rot, out);
    KATO_LAUNCHED("rotate_seq_kernel");
  }
  return KATO_OK;
}

size_t rotate_scratch_bytes(uint32_t nrows, uint32_t d) {
  const size_t ldx = (static_cast<size_t>(nrows) + 31) / 32 * 32;
  const size_t ldr = (static_cast<size_t>(d & ~3u) + 31) / 32 * 32;
  return (ldx + ldr) * (d & ~15u) * 4 + 256;
}

size_t rotation_kmajor_bytes(uint32_t d) {
  const size_t ldr = (static_cast<size_t>(d & ~3u) + 31) / 32 * 32;
  return ldr * (d & ~15u) * 4;
}

int rotation_kmajor(const float *rot, uint32_t d, float *out, cudaStream_t st) {
  const uint32_t d4 = d & ~3u, d16 = d & ~15u;
  if (d16 == 0) return KATO_OK;
  transpose_pad(rot, d4, d, d16, out, div_up(d4, 32) * 32, st);
  KATO_LAUNCHED("transpose_pad_kernel");
  return KATO_OK;
}

// A k-major copy (k rows of ld floats) in boxes of 32 floats x kRotChunk k.
static int encode_kmajor(CUtensorMap *map, const float *base, uint32_t ld, uint32_t k) {
  const PFN_cuTensorMapEncodeTiled_v12000 encode = tc::tensor_map_encoder();
  if (!encode) return cuda_status(cudaErrorNotSupported, "cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {ld, k};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 4};
  const cuuint32_t box[2] = {32, kRotChunk};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), dims,
                            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed for the rotation (error " + std::to_string(r) + ")");
    return KATO_ERUNTIME;
  }
  return KATO_OK;
}

// Few rows of few dimensions: tiles of 8 rows, which need no transpose (with tiles
// of 32 and the transpose in brackets, 16 rows: d = 128 8.5 us (9.0), 256 8.8
// (10.4)). From 512 dimensions on the rows' slab in shared memory leaves an SM few
// CTAs and its filling is not hidden: 64 rows of 512 12.4 us (11.8), of 1,024 18.1
// (15.2), of 3,072 269 (44).
constexpr uint32_t kRotFewRows = 64, kRotFewDims = 512;

int rotate_rows_kmajor(const float *in, uint32_t nrows, uint32_t d, const float *rot,
                       const float *rot_kmajor, void *scratch, float *out, uint32_t *timeouts,
                       uint32_t *launches, cudaStream_t st) {
  if (nrows == 0) return KATO_OK;
  const uint32_t d4 = d & ~3u, d16 = d & ~15u;
  if (d16 == 0) {
    *launches += (d4 ? 1 : 0) + (d4 < d ? 1 : 0);
    return rotate_rows(in, nrows, d, rot, out, st);
  }
  const uint32_t ldx = div_up(nrows, 32) * 32, ldr = div_up(d4, 32) * 32;
  float *xt = static_cast<float *>(scratch);
  const float *rt = rot_kmajor;
  // 1 KiB of slack: the stages start on a 1 KiB boundary
  const size_t slab_smem =
      kRotStages * rot_stage_bytes<true>() + static_cast<size_t>(d16) * kSlabStride * 4 + 1024;
  const bool few = nrows <= kRotFewRows && d16 < kRotFewDims;
  if (!few) {
    transpose_pad(in, nrows, d, d16, xt, ldx, st);
    ++*launches;
  }
  if (!rt) {  // no copy made at load: transpose the rotation here
    float *t = xt + static_cast<size_t>(ldx) * d16;
    transpose_pad(rot, d4, d, d16, t, ldr, st);
    ++*launches;
    rt = t;
  }
  KATO_LAUNCHED("transpose_pad_kernel");
  CUtensorMap tx{}, tr;
  int rc;
  if ((rc = encode_kmajor(&tr, rt, ldr, d16)) || (!few && (rc = encode_kmajor(&tx, xt, ldx, d16)))) return rc;
  auto go = [&](auto kern, uint32_t row_tile, int threads, size_t smem) -> int {
    if (const int r = smem_limit(reinterpret_cast<const void *>(kern), static_cast<int>(smem),
                                 "rotate_tma_kernel shared memory"))
      return r;
    launch(kern, div_up(d4, 32) * div_up(nrows, row_tile), threads, smem, st,
        tx, tr, in, nrows, d, rot, out, timeouts);
    KATO_LAUNCHED("rotate_tma_kernel");
    return KATO_OK;
  };
  rc = few ? go(rotate_tma_kernel<true>, kSlabRows, rot_threads<true>(), slab_smem)
           : go(rotate_tma_kernel<false>, 32, rot_threads<false>(),
                kRotStages * rot_stage_bytes<false>() + 1024);
  if (rc) return rc;
  ++*launches;
  if (d4 < d) {
    const uint64_t n = static_cast<uint64_t>(nrows) * (d - d4);
    launch(rotate_seq_kernel, static_cast<uint32_t>((n + 255) / 256), 256, 0, st, in, nrows, d, rot, out);
    KATO_LAUNCHED("rotate_seq_kernel");
    ++*launches;
  }
  return KATO_OK;
}

int minmax(const float *x, size_t n, uint32_t *d_keys, float *h_out, cudaStream_t st) {
  minmax_init_kernel<<<1, 1, 0, st>>>(d_keys);
  KATO_LAUNCHED("minmax_init_kernel");
  if (n) {
    const uint32_t blocks = static_cast<uint32_t>(std::min<size_t>((n + 255) / 256, 152 * 16));
    minmax_kernel<<<blocks, 256, 0, st>>>(x, n, d_keys);
    KATO_LAUNCHED("minmax_kernel");
  }
  uint32_t keys[2];
  KATO_CUDA(cudaMemcpyAsync(keys, d_keys, sizeof(keys), cudaMemcpyDeviceToHost, st));
  KATO_CUDA(cudaStreamSynchronize(st));
  h_out[0] = float_from_order_key(keys[0]);
  h_out[1] = float_from_order_key(keys[1]);
  return KATO_OK;
}

int quantize_rows(const float *x, uint32_t nrows, uint32_t d, uint32_t dc, float lo,
                  double inv_step, uint32_t head, uint8_t *hi, uint8_t *lop, int64_t *norm,
                  int64_t *hinorm, int64_t *headnorm, cudaStream_t st) {
  if (nrows == 0) return KATO_OK;
  const uint32_t blocks = std::min<uint32_t>(div_up(nrows, 8), 152 * 64);
  quantize_rows_kernel<<<blocks, 256, 0, st>>>(x, nrows, d, dc, lo, inv_step, head, hi, lop, norm,
                                              hinorm, headnorm);
  KATO_LAUNCHED("quantize_rows_kernel");
  return KATO_OK;
}

}  // namespace kato
