// chi2.cu -- the FP32C chi-square matrix over histograms (distance.cu has the
// other distance matrices and the definition).
//
// Three launches:
//   pack     every value rounded to FP32 once and laid out tile-major,
//            [64-row block][bin][64 rows], rows past the end zero, so that a
//            chunk of 32 bins of a block is 8 KB in one piece;
//   tiles    one CTA per 64 x 64 tile of the upper triangle and bin split:
//            chunks of both row blocks come by bulk async copy into a two-stage
//            ring, a thread owns 4 x 4 entries and reads its rows and its
//            column pairs with one 16-byte load each per bin; two terms per
//            packed f32x2 instruction, one MUFU reciprocal per term.  Each chunk
//            is summed plainly and Kahan-added (Kahan 1965) into a running
//            (sum, compensation) pair per entry;
//   merge    the splits' pairs added in split order (TwoSum, the rounding errors and
//            the compensations beside the sum, their own rounding errors as a third
//            float: more bits than a double holds), halved, and written to the entry
//            and its mirror image through shared memory.
//            With one split the tile kernel writes the matrix itself.
// Sums stay in floats until the double additions at the end: an FP64 warp
// instruction holds a scheduler's FP64 pipe for 64 cycles, and 48 of them per
// thread (conversions included) were a quarter of the time.
// Bound: the MUFU reciprocals, one per term: a warp's takes a scheduler's unit 8
// cycles, and a loop of this body on registers alone 16.9 cycles per pair of terms
// (10.3 without the reciprocals); two terms can't share one, 1 / (s t) rounds
// differently.  1,024 histograms of 400 bins: pack 3, tiles 60 (51 at 16.9 cycles),
// merge 11 us, 78 us per call; 96 before, with row-major staging and the splits summed
// in double.  A call with 3 or 4 CTAs per SM and 1, 2 or 4 bins per turn: 3 and 2
// 78 us, 3 and 1 86, 3 and 4 82, 4 and 1 to 4 82 to 84; 2 x 4 and 4 x 2 entries per
// thread, and 32 x 16 tiles in one pass without splits, up to 6 us longer.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "common.cuh"
#include "kernels.cuh"

namespace cpetgb {
namespace {

constexpr int kTile = 64;
constexpr int kThreads = 256;  // 16 x 16 threads, 4 x 4 entries each
constexpr int kChunk = 32;     // bins per Kahan-added sum and per stage
constexpr int kStages = 2;
constexpr int kEntries = kTile * kTile;

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Reciprocal of a bin's sum a + b by the MUFU; 0 for a sum of zero, whose bin does
// not contribute whatever a - b is, and for a subnormal one, which the MUFU takes for
// zero (the values it comes from have a square that vanishes).  The reciprocal cut off
// at FLT_MAX instead, which is enough where no value is negative, runs 2% faster on
// large matrices (3,000 x 900 980 us against 998) and alike on 1,024 x 400 (78 us).
__device__ __forceinline__ float rcp_sum(float s) {
  return fabsf(s) >= FLT_MIN ? rcp_mufu(s) : 0.f;
}

__device__ __forceinline__ double pair_value(float s, float c) { return __dsub_rn(widen(s), widen(c)); }

// Upper-triangle tile t, column by column: t = jb (jb + 1) / 2 + ib, ib <= jb.
__device__ __forceinline__ void tile_of(uint32_t t, int& ib, int& jb) {
  uint32_t j = static_cast<uint32_t>(0.5f * (sqrtf(8.f * static_cast<float>(t) + 1.f) - 1.f));
  while (uint64_t(j) * (j + 1) / 2 > t) --j;
  while (uint64_t(j + 1) * (j + 2) / 2 <= t) ++j;
  jb = static_cast<int>(j);
  ib = static_cast<int>(t - uint64_t(j) * (j + 1) / 2);
}

// One row block x 32 bins per step, all of a thread's loads in flight at once.
__global__ void __launch_bounds__(kThreads)
    chi2_pack_kernel(int n, int bins, const double* __restrict__ in, float* __restrict__ out) {
  constexpr int kBins = 32, kLoads = kTile * kBins / kThreads;
  __shared__ float t[kBins][kTile + 1];
  const int tid = threadIdx.x, rb = blockIdx.x;
  for (int64_t k0 = int64_t(blockIdx.y) * kBins; k0 < bins; k0 += int64_t(gridDim.y) * kBins) {
    const int64_t k = k0 + tid % kBins;
    double v[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int64_t row = int64_t(rb) * kTile + tid / kBins + u * (kThreads / kBins);
      v[u] = row < n && k < bins ? in[row * bins + k] : 0.0;
    }
    __syncthreads();  // the previous step's reads
#pragma unroll
    for (int u = 0; u < kLoads; ++u) t[tid % kBins][tid / kBins + u * (kThreads / kBins)] = narrow(v[u]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int e = tid + u * kThreads;
      if (k0 + e / kTile < bins) out[(int64_t(rb) * bins + k0) * kTile + e] = t[e / kTile][e % kTile];
    }
  }
}

// part: [tile][split][16 entries][256 threads] pairs, or null (one split).
__global__ void __launch_bounds__(kThreads, 3)
    chi2_tile_kernel(int n, int bins, int per, const float* __restrict__ rows, double* __restrict__ out,
                     float2* __restrict__ part, int* __restrict__ status) {
  __shared__ alignas(16) float sA[kStages][kChunk][kTile];
  __shared__ alignas(16) float sB[kStages][kChunk][kTile];
  __shared__ uint64_t full[kStages];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  int ib, jb;
  tile_of(blockIdx.x, ib, jb);
  const int kb = blockIdx.y * per, ke = min(bins, kb + per);
  const int n_chunks = ke > kb ? (ke - kb + kChunk - 1) / kChunk : 0;
  const float* rows_a = rows + (int64_t(ib) * bins + kb) * kTile;
  const float* rows_b = rows + (int64_t(jb) * bins + kb) * kTile;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  auto issue = [&](int t) {
    const int s = t % kStages;
    const uint32_t bytes = static_cast<uint32_t>(min(kChunk, ke - kb - t * kChunk)) * kTile * sizeof(float);
    mbar_arrive_expect_tx(&full[s], 2 * bytes);
    bulk_g2s(&sA[s][0][0], rows_a + int64_t(t) * kChunk * kTile, bytes, &full[s]);
    bulk_g2s(&sB[s][0][0], rows_b + int64_t(t) * kChunk * kTile, bytes, &full[s]);
  };
  if (tid == 0)
    for (int t = 0; t < min(kStages, n_chunks); ++t) issue(t);

  float sum[4][4], cmp[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) sum[r][c] = cmp[r][c] = 0.f;

  for (int t = 0; t < n_chunks; ++t) {
    const int s = t % kStages;
    const bool mine = mbar_wait(&full[s], static_cast<uint32_t>((t / kStages) & 1), status);
    // also: every thread is done with chunk t - 1, whose stage takes the next copy
    if (!__syncthreads_and(mine)) {
      // a copy that never came: wait (with the same limit) for what else is in flight
      if (tid == 0)
        for (int u = t; u < min(t - 1 + kStages, n_chunks); ++u)
          mbar_wait(&full[u % kStages], static_cast<uint32_t>((u / kStages) & 1), status);
      return;
    }
    if (tid == 0 && t >= 1 && t - 1 + kStages < n_chunks) issue(t - 1 + kStages);
    const int kn = min(kChunk, ke - kb - t * kChunk);
    const float4* a4 = reinterpret_cast<const float4*>(&sA[s][0][0]) + ty;
    const ulonglong2* b4 = reinterpret_cast<const ulonglong2*>(&sB[s][0][0]) + tx;
    uint64_t p[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) p[r][0] = p[r][1] = 0ull;
#pragma unroll 2
    for (int k = 0; k < kn; ++k) {
      const float4 av = a4[k * (kTile / 4)];
      const ulonglong2 bv = b4[k * (kTile / 4)];
      const float a[4] = {av.x, av.y, av.z, av.w};
      const uint64_t b[2] = {bv.x, bv.y};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint64_t aa = pk2(a[r], a[r]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint64_t d = sub2(aa, b[h]);
          float s0, s1;
          upk2(add2(aa, b[h]), s0, s1);
          p[r][h] = fma2(mul2(d, d), pk2(rcp_sum(s0), rcp_sum(s1)), p[r][h]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float lo, hi;
        upk2(p[r][h], lo, hi);
        kahan_add(sum[r][2 * h], cmp[r][2 * h], lo);
        kahan_add(sum[r][2 * h + 1], cmp[r][2 * h + 1], hi);
      }
  }

  if (part) {
    float2* dst = part + (int64_t(blockIdx.x) * gridDim.y + blockIdx.y) * kEntries + tid;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) dst[(4 * r + c) * kThreads] = make_float2(sum[r][c], cmp[r][c]);
    return;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int64_t i = int64_t(ib) * kTile + 4 * ty + r, j = int64_t(jb) * kTile + 4 * tx + c;
      if (i >= n || j >= n) continue;
      const double v = i == j ? 0.0 : 0.5 * pair_value(sum[r][c], cmp[r][c]);
      out[i * n + j] = v;
      if (ib != jb) out[j * n + i] = v;
    }
}

// A sum of pairs (value hi - lo) in three floats: s, the rounding errors and the
// compensations c, and the rounding errors of those.
struct Sum3 {
  float s = 0.f, c = 0.f, d = 0.f;
  __device__ __forceinline__ void add(float hi, float lo) {
    float e, w, ew, ec;
    two_sum(s, hi, s, e);
    two_sum(e, -lo, w, ew);
    two_sum(c, w, c, ec);
    d = __fadd_rn(d, __fadd_rn(ew, ec));
  }
  __device__ __forceinline__ double value() const {
    return __dadd_rn(widen(s), __dadd_rn(widen(c), widen(d)));
  }
};

constexpr int kManySplits = 16;  // (see chi2_merge_kernel)

// blockIdx.y = part g of the tile: its rows ROWS g .. ROWS g + ROWS - 1, so that both
// the rows and their mirror columns are written in runs.  G groups of threads take the
// splits z, z + G, ..., and the first adds the others' sums in order.  One group and 16
// rows (runs of 128 bytes) for few splits; for many, which come with few tiles, the
// chain over the splits is what counts.  A call with <16, 1> and with <4, 8>: 100
// histograms of 20,000 bins (3 tiles, 203 splits) 137 and 86 us, 60 of 20,000 137 and 61,
// 100 of 3,000 (46 splits) 41 and 30; 300 of 800 (12 splits) 39 and 38, 500 of 900 (14)
// 59 and 61.
template <int ROWS, int G>
__global__ void __launch_bounds__(16 * ROWS * G)
    chi2_merge_kernel(int n, int splits, const float2* __restrict__ part, double* __restrict__ out) {
  constexpr int kGroup = 16 * ROWS, kOwners = 4 * ROWS;  // threads of a group; tile threads it stands for
  __shared__ double t[ROWS][kTile + 1];
  __shared__ Sum3 others[G > 1 ? G - 1 : 1][G > 1 ? 4 : 1][kGroup];
  const int tid = threadIdx.x % kGroup, group = threadIdx.x / kGroup, g = blockIdx.y;
  const int owner = tid % kOwners, r = tid / kOwners;
  int ib, jb;
  tile_of(blockIdx.x, ib, jb);
  const float2* src = part + int64_t(blockIdx.x) * splits * kEntries + 4 * r * kThreads + kOwners * g + owner;
  Sum3 sum[4];
#pragma unroll 4
  for (int z = group; z < splits; z += G)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 v = src[int64_t(z) * kEntries + k * kThreads];
      sum[k].add(v.x, v.y);
    }
  if constexpr (G > 1) {
    if (group > 0)
#pragma unroll
      for (int k = 0; k < 4; ++k) others[group - 1][k][tid] = sum[k];
    __syncthreads();
    if (group == 0)
      for (int o = 0; o < G - 1; ++o)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const Sum3 v = others[o][k][tid];
          sum[k].add(v.s, -v.c);
          sum[k].add(v.d, 0.f);
        }
  }
  if (group == 0)
#pragma unroll
    for (int k = 0; k < 4; ++k) t[4 * (owner >> 4) + r][4 * (owner & 15) + k] = 0.5 * sum[k].value();
  __syncthreads();
  const int64_t i0 = int64_t(ib) * kTile + ROWS * g, j0 = int64_t(jb) * kTile;
  for (int e = threadIdx.x; e < ROWS * kTile; e += kGroup * G) {
    const int64_t i = i0 + e / kTile, j = j0 + e % kTile;
    if (i < n && j < n) out[i * n + j] = i == j ? 0.0 : t[e / kTile][e % kTile];
  }
  if (ib == jb) return;
  for (int e = threadIdx.x; e < ROWS * kTile; e += kGroup * G) {
    const int64_t i = i0 + e % ROWS, j = j0 + e / ROWS;
    if (i < n && j < n) out[j * n + i] = t[e % ROWS][e / ROWS];
  }
}

template <int ROWS, int G>
cudaError_t launch_merge(int n, int splits, unsigned tiles, const float2* part, double* out, cudaStream_t s) {
  chi2_merge_kernel<ROWS, G><<<dim3(tiles, kTile / ROWS), 16 * ROWS * G, 0, s>>>(n, splits, part, out);
  return cudaGetLastError();
}

}  // namespace

int64_t chi2_row_blocks(int n) { return (int64_t(n) + kTile - 1) / kTile; }
size_t chi2_rows_bytes(int n, int bins) { return size_t(chi2_row_blocks(n)) * kTile * size_t(bins) * sizeof(float); }
size_t chi2_partial_bytes(int n, int splits) {
  const int64_t nb = chi2_row_blocks(n);
  return size_t(nb * (nb + 1) / 2) * size_t(splits) * kEntries * sizeof(float2);
}

cudaError_t launch_chi2_f32(int n, int bins, const double* hists, double* out, int splits, void* partial,
                            void* rows, int* status, cudaStream_t s) {
  const int64_t nb = chi2_row_blocks(n);
  float* fr = static_cast<float*>(rows);
  if (bins > 0) {
    const int by = static_cast<int>(std::min<int64_t>((int64_t(bins) + 31) / 32, 65535));
    chi2_pack_kernel<<<dim3(static_cast<unsigned>(nb), by), kThreads, 0, s>>>(n, bins, hists, fr);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (splits < 1 || bins == 0) splits = 1;
  const int per = (bins + splits - 1) / splits;
  float2* pairs = splits > 1 ? static_cast<float2*>(partial) : nullptr;
  const unsigned tiles = static_cast<unsigned>(nb * (nb + 1) / 2);
  chi2_tile_kernel<<<dim3(tiles, splits), kThreads, 0, s>>>(n, bins, per, fr, out, pairs, status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || splits == 1) return e;
  return splits < kManySplits ? launch_merge<16, 1>(n, splits, tiles, pairs, out, s)
                              : launch_merge<4, 8>(n, splits, tiles, pairs, out, s);
}

}  // namespace cpetgb
