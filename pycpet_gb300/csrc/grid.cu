// grid.cu -- all-pairs Coulomb sums on point sets (K1 field, K2 potential).
//
// Replaces compute_looped_field (CPET/utils/math_module.c:405-451, field with
// r^2 clamped at 1e-6), calc_field (math_module.c:255-293, unclamped field at
// a point) and calc_esp_base (math_module.c:453-486, potential), which the
// reference evaluates one point at a time on one CPU core.
//
// Work decomposition: a CTA owns a tile of a frame's points (kGridThreads
// threads, PPT points each, kept in registers) and a contiguous chunk of that
// frame's charges.  The charges stream through a ring of shared memory stages
// filled by 1-D bulk async copies (cp.async.bulk) that complete on mbarriers;
// every thread reads each staged charge as a broadcast and applies it to its
// PPT points.
//
// Lattices: the points of a volume are a mesh, x slowest.  The preparation
// kernel looks for the stride S at which x changes and (y, z) repeat, and for meshes a
// thread takes PPT points of one (y, z) column: dy, dz and dy^2 + dz^2 are formed
// once per charge instead of once per point and charge, in the same order of
// operations, so the sums are the same bits.  That is 9 instead of 12 FP32-pipe
// operations per pair (4 instead of 7 for the potential, which is then bound by
// the MUFU alone), 9 FP64-pipe instructions instead of 12.  The points that do
// not fill a column's last group are evaluated as points without a mesh.
//
// Precision forms:
//   FP32C  pair terms in FP32 with the MUFU rsqrt; each stage's contribution is
//          summed plainly in FP32 and then Kahan-added (compensated) into a
//          running (sum, compensation) pair per component; the result leaves
//          the CTA as a double.
//   FP64   every operation in IEEE double (plain sums), the drop-in form.
// A frame whose charges are split over several items writes per-split partial
// sums (doubles) that grid_final_kernel adds in a fixed order: deterministic.
// A frame of at most kGridFewPoints points (point fields) goes to
// grid_few_kernel, whose threads take (point, run of charges) units instead of
// points, with the same runs and order.
//
// The r^2 >= 1e-6 clamp of compute_looped_field only changes a pair term when
// a point lies within 1e-3 A of a charge.  A CTA takes the bounding box of its
// points once, tests each staged tile of charges against it (distance below
// kNearA) and runs the clamped loop only for tiles that hold such a charge;
// every other tile runs the unclamped loop, which gives the same values there.
//
// FP32C field refinement: where the field nearly cancels, FP32 rounding of the
// pair terms (about 1e-7 of each term) is a large fraction of |E|.  After the
// FP32C pass, grid_final_kernel (which counts a histogram of |E|^2 and takes the
// median from it) and grid_flag_kernel find, per frame, the points whose |E| is
// below tau times the frame's median |E| and grid_refine_kernel recomputes those
// points over all of the frame's charges in double-float arithmetic (pairs of
// floats, about 48 significant bits, on the FP32 pipe: GB300's FP64 pipe is
// 1/64 of its FP32 pipe).
#include <algorithm>
#include <cstddef>
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.cuh"
#include "point_map.cuh"

namespace cpetgb {
namespace {

constexpr int kStages = 4;

// static_cast<Real>, FP32C without the FP64 pipe.
template <typename Real>
__device__ __forceinline__ Real to_real(double v) {
  if constexpr (sizeof(Real) == 4)
    return narrow(v);
  else
    return v;
}

template <int PREC>
struct GridCfg;
// FP32C charge record with every component duplicated, {x,x,y,y} {z,z,q,q}:
// one broadcast 16-byte shared load yields two ready f32x2 operands, and a
// packed instruction then evaluates the pair term for two grid points.
struct alignas(32) ChargeDup {
  ulonglong2 xy;
  ulonglong2 zq;
};
template <>
struct GridCfg<kFP32C> {
  using ChargeT = ChargeDup;
  using Real = float;
  static constexpr int kTile = 256;  // charges per stage (8 KiB)
};
template <>
struct GridCfg<kFP64> {
  using ChargeT = Charge64;
  using Real = double;
  static constexpr int kTile = 256;  // charges per stage (8 KiB)
};

// FP64: q r^-3 (field) or q r^-1 (potential).
template <int KIND>
__device__ __forceinline__ double weight_f64(const Charge64& c, double r2) {
  return KIND == kField ? weight_r3_f64(c.q, r2) : weight_r1_f64(c.q, r2);
}
// {v, v} as one packed 64-bit value.
__device__ __forceinline__ uint64_t dup2(float v) {
  const uint64_t b = __float_as_uint(v);
  return b | (b << 32);
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// Kahan accumulation on both lanes of packed pairs.
__device__ __forceinline__ void kahan_add2(uint64_t& s, uint64_t& c, uint64_t t) {
  const uint64_t y = sub2(t, c);
  const uint64_t u = add2(s, y);
  c = sub2(sub2(u, s), y);
  s = u;
}

constexpr int kKahanRun = 32;  // FP32C: charges summed plainly between Kahan steps

// A staged charge closer than kNearA to the CTA's point box sends its tile
// through the clamped loop.  The clamp acts below 1e-3 A; the margin covers the
// FP32 rounding of coordinates up to 1e4 A.
constexpr float kNearA = 0.01f;

__device__ __forceinline__ void charge_xyz(const ChargeDup& c, float& x, float& y, float& z) {
  x = __uint_as_float(static_cast<uint32_t>(c.xy.x));
  y = __uint_as_float(static_cast<uint32_t>(c.xy.y));
  z = __uint_as_float(static_cast<uint32_t>(c.zq.x));
}
__device__ __forceinline__ void charge_xyz(const Charge64& c, float& x, float& y, float& z) {
  x = static_cast<float>(c.x);
  y = static_cast<float>(c.y);
  z = static_cast<float>(c.z);
}
// Squared distance from (x, y, z) to the box [lo, hi] (0 inside).
__device__ __forceinline__ float box_dist2(const float (&lo)[3], const float (&hi)[3], float x,
                                           float y, float z) {
  const float dx = fmaxf(fmaxf(lo[0] - x, x - hi[0]), 0.f);
  const float dy = fmaxf(fmaxf(lo[1] - y, y - hi[1]), 0.f);
  const float dz = fmaxf(fmaxf(lo[2] - z, z - hi[2]), 0.f);
  return dx * dx + dy * dy + dz * dz;
}

// One charge against this thread's G packed point pairs, added to part[].
template <int KIND, bool CLAMP, int G>
__device__ __forceinline__ void pair_terms_f32x2(const ChargeDup& ch, const uint64_t (&px)[G],
                                                 const uint64_t (&py)[G], const uint64_t (&pz)[G],
                                                 uint64_t (&part)[(KIND == kField) ? 3 : 1][G]) {
  const ulonglong2 xy = ch.xy;
  const ulonglong2 zq = ch.zq;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const uint64_t dx = sub2(px[g], xy.x);
    const uint64_t dy = sub2(py[g], xy.y);
    const uint64_t dz = sub2(pz[g], zq.x);
    uint64_t r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    if constexpr (CLAMP) {  // compute_looped_field's fmaxf(r^2, 1e-6f)
      float a, b;
      upk2(r2, a, b);
      r2 = pk2(fmaxf(a, 1e-6f), fmaxf(b, 1e-6f));
    }
    const uint64_t ri = rsqrt2(r2);
    if constexpr (KIND == kField) {
      const uint64_t w = mul2(mul2(zq.y, ri), mul2(ri, ri));
      part[0][g] = fma2(w, dx, part[0][g]);
      part[1][g] = fma2(w, dy, part[1][g]);
      part[2][g] = fma2(w, dz, part[2][g]);
    } else {
      part[0][g] = fma2(zq.y, ri, part[0][g]);
    }
  }
}

// One charge against G packed point pairs of one (y, z) column: the same
// operations as pair_terms_f32x2, those of y and z once.
template <int KIND, int G>
__device__ __forceinline__ void column_terms_f32x2(const ChargeDup& ch, const uint64_t (&px)[G], float py,
                                                   float pz, uint64_t (&part)[(KIND == kField) ? 3 : 1][G]) {
  const ulonglong2 xy = ch.xy;
  const ulonglong2 zq = ch.zq;
  const float dy = __fsub_rn(py, __uint_as_float(static_cast<uint32_t>(xy.y)));
  const float dz = __fsub_rn(pz, __uint_as_float(static_cast<uint32_t>(zq.x)));
  const float t = __fmaf_rn(dy, dy, __fmul_rn(dz, dz));
  const uint64_t t2 = pk2(t, t), dy2 = pk2(dy, dy), dz2 = pk2(dz, dz);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const uint64_t dx = sub2(px[g], xy.x);
    const uint64_t ri = rsqrt2(fma2(dx, dx, t2));
    if constexpr (KIND == kField) {
      const uint64_t w = mul2(mul2(zq.y, ri), mul2(ri, ri));
      part[0][g] = fma2(w, dx, part[0][g]);
      part[1][g] = fma2(w, dy2, part[1][g]);
      part[2][g] = fma2(w, dz2, part[2][g]);
    } else {
      part[0][g] = fma2(zq.y, ri, part[0][g]);
    }
  }
}

// FP32C body: this thread's points as G packed pairs (points k = 2g, 2g+1).
// CLAMP = true is the rare path (a staged charge next to the point box): the
// same arithmetic with the clamp, in a loop that is not unrolled, so it adds
// few registers to the kernel.
// COLUMN: the points are of one (y, z) column.
template <int KIND, bool CLAMP, bool COLUMN, int G>
__device__ __forceinline__ void grid_tile_f32x2(const ChargeDup* __restrict__ tl, int cnt,
                                                const uint64_t (&px)[G], const uint64_t (&py)[G],
                                                const uint64_t (&pz)[G], uint64_t (&acc)[3][G],
                                                uint64_t (&cmp)[3][G]) {
  constexpr int NC = (KIND == kField) ? 3 : 1;
  for (int j0 = 0; j0 < cnt; j0 += kKahanRun) {
    const int j1 = min(cnt, j0 + kKahanRun);
    uint64_t part[NC][G];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int g = 0; g < G; ++g) part[c][g] = 0ull;
    if constexpr (CLAMP) {
#pragma unroll 1
      for (int j = j0; j < j1; ++j) pair_terms_f32x2<KIND, true, G>(tl[j], px, py, pz, part);
    } else if constexpr (COLUMN) {
      const float y = __uint_as_float(static_cast<uint32_t>(py[0]));
      const float z = __uint_as_float(static_cast<uint32_t>(pz[0]));
#pragma unroll 8
      for (int j = j0; j < j1; ++j) column_terms_f32x2<KIND, G>(tl[j], px, y, z, part);
    } else {
// (potential: 522 us per 101^3 points in no order x 2,000 charges, 528 with four)
#pragma unroll (KIND == kEsp ? 8 : 4)
      for (int j = j0; j < j1; ++j) pair_terms_f32x2<KIND, false, G>(tl[j], px, py, pz, part);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int g = 0; g < G; ++g) kahan_add2(acc[c][g], cmp[c][g], part[c][g]);
  }
}

// The frame of item / tile / preparation block `i`: the last one whose base (the
// int32 at byte offset OFF of the record) is <= i.  32 records per look, by a
// whole warp.
template <int OFF>
__device__ __forceinline__ int find_frame(const GridFrame* frames, int n_frames, int i) {
  const int lane = threadIdx.x & 31;
  auto base = [&](int f) {
    return *reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(frames + f) + OFF);
  };
  int lo = 0, span = n_frames;
  while (span > 1) {  // narrow [lo, lo + span) to one of 32 parts
    const int part = (span + 31) / 32;
    const int f = lo + lane * part;
    const unsigned below = __ballot_sync(0xffffffffu, lane * part < span && base(f) <= i);
    const int k = 31 - __clz(below);
    span = min(part, span - k * part);
    lo += k * part;
  }
  return lo;
}

// A kernel's view of its frame: the launch's only one, from the kernel's
// parameters, or the table's entry.
template <int OFF>
__device__ __forceinline__ GridFrame load_frame(const GridFrame* frames, int n_frames, const GridFrame& one,
                                                int i, int* f) {
  if (n_frames == 1) {
    *f = 0;
    return one;
  }
  *f = find_frame<OFF>(frames, n_frames, i);
  return frames[*f];
}

// FP32C with 4 points per thread: four CTAs (16 warps) per SM for the field,
// whose column loop needs more than 80 registers to keep the FP32 pipe fed (24
// frames: 2.09 ms, 2.20 with six CTAs), six for the potential.
template <int PREC, int KIND, bool CLAMP, int PPT>
__global__ void __launch_bounds__(kGridThreads, PREC == kFP32C && PPT == 4 ? (KIND == kField ? 4 : 6) : 0)
    grid_kernel(const GridFrame* __restrict__ frames, int n_frames, const GridFrame one, int item0,
                const int* __restrict__ stride, const int* __restrict__ broken, const void* __restrict__ packed,
                const double* __restrict__ points, double* __restrict__ out,
                double* __restrict__ partial, int* __restrict__ status) {
  using Cfg = GridCfg<PREC>;
  using ChargeT = typename Cfg::ChargeT;
  using Real = typename Cfg::Real;
  constexpr int TC = Cfg::kTile;
  constexpr int NC = (KIND == kField) ? 3 : 1;

  __shared__ alignas(128) ChargeT tile[kStages][TC];
  __shared__ alignas(8) uint64_t full[kStages];

  const int tid = threadIdx.x;
  const int item = item0 + static_cast<int>(blockIdx.x);
  int f;
  const GridFrame fr = load_frame<offsetof(GridFrame, item_base)>(frames, n_frames, one, item, &f);
  const int n_tiles_pt = fr.n_tiles;
  const int split = (item - fr.item_base) / n_tiles_pt;
  const int tile_id = (item - fr.item_base) - split * n_tiles_pt;
  const int n_begin = split * fr.chunk;
  const int n = min(fr.chunk, fr.n_charges - n_begin);
  const ChargeT* src = reinterpret_cast<const ChargeT*>(packed) + fr.charge_off + n_begin;
  const int n_tiles = (n + TC - 1) / TC;
  PointMap map;
  map.set<PPT>(stride && !broken[f] ? stride[f] : 0, fr.n_points);
  if (tile_id * kGridThreads >= map.threads<PPT>()) return;  // the table's last tile may be spare

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncthreads();

  auto issue = [&](int t) {
    const int s = t % kStages;
    const int cnt = min(TC, n - t * TC);
    const uint32_t bytes = static_cast<uint32_t>(cnt * sizeof(ChargeT));
    mbar_arrive_expect_tx(&full[s], bytes);
    bulk_g2s(&tile[s][0], src + static_cast<int64_t>(t) * TC, bytes, &full[s]);
  };
  if (tid == 0) {
    for (int t = 0; t < min(kStages, n_tiles); ++t) issue(t);
  }

  const int u = tile_id * kGridThreads + tid;
  const int64_t point_off = fr.point_off;
  const bool column = map.column(u);
  unsigned valid = 0;  // which of this thread's points exist
  // This thread's points, in registers (FP32C: packed in pairs).
  Real px[PPT], py[PPT], pz[PPT];
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int pl = map.point<PPT>(u, k);
    if (pl >= 0) {
      valid |= 1u << k;
      const double* pp = points + 3 * (point_off + pl);
      px[k] = to_real<Real>(pp[0]);
      py[k] = to_real<Real>(pp[1]);
      pz[k] = to_real<Real>(pp[2]);
    } else {
      px[k] = py[k] = pz[k] = static_cast<Real>(1.0e4);  // far away, never written
    }
  }
  constexpr int G = PPT / 2;
  [[maybe_unused]] uint64_t px2[G], py2[G], pz2[G], acc2[3][G], cmp2[3][G];
  if constexpr (PREC == kFP32C) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      px2[g] = pk2(px[2 * g], px[2 * g + 1]);
      py2[g] = pk2(py[2 * g], py[2 * g + 1]);
      pz2[g] = pk2(pz[2 * g], pz[2 * g + 1]);
#pragma unroll
      for (int c = 0; c < 3; ++c) acc2[c][g] = cmp2[c][g] = 0ull;
    }
  }

  // FP64 running sums.
  Real acc[NC][PPT];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int k = 0; k < PPT; ++k) acc[c][k] = Real(0);

  // Bounding box of this CTA's points (clamped kernels only), kept in shared
  // memory so it holds no registers during the pair loops.
  __shared__ float box_s[6];
  if constexpr (CLAMP) {
    __shared__ float box_part[kGridThreads / 32][6];
    float v[6] = {3.0e38f, 3.0e38f, 3.0e38f, -3.0e38f, -3.0e38f, -3.0e38f};
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      if ((valid >> k) & 1u) {
        const float c3[3] = {static_cast<float>(px[k]), static_cast<float>(py[k]),
                             static_cast<float>(pz[k])};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          v[a] = fminf(v[a], c3[a]);
          v[3 + a] = fmaxf(v[3 + a], c3[a]);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        v[a] = fminf(v[a], __shfl_xor_sync(0xffffffffu, v[a], o));
        v[3 + a] = fmaxf(v[3 + a], __shfl_xor_sync(0xffffffffu, v[3 + a], o));
      }
    if ((tid & 31) == 0)
#pragma unroll
      for (int a = 0; a < 6; ++a) box_part[tid >> 5][a] = v[a];
    __syncthreads();
    if (tid < 6) {
      float b = box_part[0][tid];
#pragma unroll
      for (int w = 1; w < kGridThreads / 32; ++w)
        b = tid < 3 ? fminf(b, box_part[w][tid]) : fmaxf(b, box_part[w][tid]);
      box_s[tid] = b;
    }
    __syncthreads();
  }

  const bool work = __any_sync(0xffffffffu, valid != 0);  // a warp without points only waits
  bool ok = true;
  for (int t = 0; t < n_tiles; ++t) {
    const int s = t % kStages;
    const bool mine = mbar_wait(&full[s], static_cast<uint32_t>((t / kStages) & 1), status);
    const int cnt = min(TC, n - t * TC);
    const ChargeT* tl = &tile[s][0];
    bool clamp_tile = false;
    if constexpr (CLAMP) {
      // Does this tile hold a charge next to the point box?  One barrier both
      // answers that and confirms every thread's wait (the common case).
      bool near = false;
      if (mine) {
        const float blo[3] = {box_s[0], box_s[1], box_s[2]};
        const float bhi[3] = {box_s[3], box_s[4], box_s[5]};
        for (int j = tid; j < cnt; j += kGridThreads) {
          float cx, cy, cz;
          charge_xyz(tl[j], cx, cy, cz);
          near |= box_dist2(blo, bhi, cx, cy, cz) < kNearA * kNearA;
        }
      }
      const int clean = __syncthreads_count(mine && !near);  // also: tile t-1 is done
      if (clean != kGridThreads) {
        ok = __syncthreads_and(mine) != 0;
        clamp_tile = true;
      }
    } else {
      ok = __syncthreads_and(mine) != 0;  // also: every thread is done with tile t-1
    }
    if (!ok) break;
    if (tid == 0 && t >= 1 && (t - 1) + kStages < n_tiles) issue((t - 1) + kStages);

    if (!work) continue;
    if constexpr (PREC == kFP32C) {
      if (CLAMP && clamp_tile)
        grid_tile_f32x2<KIND, true, false, G>(tl, cnt, px2, py2, pz2, acc2, cmp2);
      else if (column)
        grid_tile_f32x2<KIND, false, true, G>(tl, cnt, px2, py2, pz2, acc2, cmp2);
      else
        grid_tile_f32x2<KIND, false, false, G>(tl, cnt, px2, py2, pz2, acc2, cmp2);
    } else {
      Real part[NC][PPT];
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < PPT; ++k) part[c][k] = Real(0);
      auto term = [&](const ChargeT& ch, int k, Real dy, Real dz, Real t, auto clamped) {
        const Real dx = px[k] - ch.x;
        Real r2 = __fma_rn(dx, dx, t);
        if constexpr (clamped.value) r2 = fmax(r2, Real(1e-6));  // compute_looped_field's fmaxf
        const Real w = weight_f64<KIND>(ch, r2);
        if constexpr (KIND == kField) {
          part[0][k] += w * dx;
          part[1][k] += w * dy;
          part[2][k] += w * dz;
        } else {
          part[0][k] += w;
        }
      };
      auto points = [&](auto clamped) {
        for (int j = 0; j < cnt; ++j) {
          const ChargeT ch = tl[j];
#pragma unroll
          for (int k = 0; k < PPT; ++k) {
            const Real dy = py[k] - ch.y, dz = pz[k] - ch.z;
            term(ch, k, dy, dz, __fma_rn(dy, dy, __dmul_rn(dz, dz)), clamped);
          }
        }
      };
      // the clamp in a loop of its own: as a condition in the others its comparison
      // is evaluated for every pair (one FP64-pipe instruction more; 9,261 points x
      // 5,000 charges 1,115 us against 1,011 when a pair took 10 of them)
      if (CLAMP && clamp_tile) {
        points(std::true_type{});
      } else if (column) {
        for (int j = 0; j < cnt; ++j) {
          const ChargeT ch = tl[j];
          const Real dy = py[0] - ch.y, dz = pz[0] - ch.z;
          const Real t = __fma_rn(dy, dy, __dmul_rn(dz, dz));
#pragma unroll
          for (int k = 0; k < PPT; ++k) term(ch, k, dy, dz, t, std::false_type{});
        }
      } else {
        points(std::false_type{});
      }
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < PPT; ++k) acc[c][k] += part[c][k];
    }
  }
  if (!ok) return;

  constexpr int kTilePts = kGridThreads * PPT;
  const int slot = fr.slot_base < 0 ? -1 : fr.slot_base + (item - fr.item_base);
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    if (!((valid >> k) & 1u)) continue;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      double v;
      if constexpr (PREC == kFP32C) {
        float sl, sh, cl, ch;
        upk2(acc2[c][k / 2], sl, sh);
        upk2(cmp2[c][k / 2], cl, ch);
        const float sv = (k & 1) ? sh : sl, cv = (k & 1) ? ch : cl;
        v = __dmul_rn(__dsub_rn(widen(sv), widen(cv)), kCoulomb);
      } else {
        v = static_cast<double>(acc[c][k]) * kCoulomb;
      }
      if (slot < 0)
        out[NC * (point_off + map.point<PPT>(u, k)) + c] = v;
      else
        partial[(static_cast<int64_t>(slot) * NC + c) * kTilePts + k * kGridThreads + tid] = v;
    }
  }
}

// Sum over a frame's splits, in one order everywhere: eight partial sums (splits
// l, l + 8, ...), then ((v0 + v4) + (v2 + v6)) + ((v1 + v5) + (v3 + v7)).  By one
// thread, or by eight neighbouring lanes (l = lane & 7): an FP64 addition holds a
// scheduler's pipe for 64 cycles, so a few points with hundreds of splits would
// otherwise wait for one long chain.
constexpr int kSumLanes = 8;
__device__ __forceinline__ double sum_lanes(double v) {
#pragma unroll
  for (int o = kSumLanes / 2; o >= 1; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double sum_thread(const double (&v)[kSumLanes]) {
  return __dadd_rn(__dadd_rn(__dadd_rn(v[0], v[4]), __dadd_rn(v[2], v[6])),
                   __dadd_rn(__dadd_rn(v[1], v[5]), __dadd_rn(v[3], v[7])));
}

// Frames of few points (point fields): a CTA takes one chunk of a frame's
// charges against all of its points.  Its threads take units of one point and
// one run of kFewRun charges (the tile kernel's Kahan runs in FP32C: 32 charges
// within stages of 256, so the sums are the same bits), and then add the runs of
// each point and component in order.  With a thread per point instead, a
// 1-point launch took 20 us (739 us in FP64) for the padding of its tile.
template <int PREC, int KIND, bool CLAMP, int PPT>
__global__ void __launch_bounds__(kGridThreads)
    grid_few_kernel(const GridFrame* __restrict__ frames, int n_frames, const GridFrame one, const void* __restrict__ packed,
                    const double* __restrict__ points, double* __restrict__ out,
                    double* __restrict__ partial) {
  using ChargeT = typename GridCfg<PREC>::ChargeT;
  using Real = typename GridCfg<PREC>::Real;
  constexpr int NC = (KIND == kField) ? 3 : 1;
  constexpr int kFewRun = PREC == kFP32C ? kKahanRun : 8;
  constexpr int kStage = GridCfg<PREC>::kTile;
  constexpr int kUnits = 1024;  // (point, run) sums held at a time
  __shared__ Real sums[NC][kUnits];
  __shared__ Real acc_s[NC * kGridFewPoints], cmp_s[NC * kGridFewPoints];
  const int tid = threadIdx.x;
  const int item = static_cast<int>(blockIdx.x);
  int f;
  const GridFrame fr = load_frame<offsetof(GridFrame, item_base)>(frames, n_frames, one, item, &f);
  const int P = fr.n_points;
  const int split = item - fr.item_base;  // one tile
  const int n_begin = split * fr.chunk;
  const int n = min(fr.chunk, fr.n_charges - n_begin);
  const ChargeT* src = reinterpret_cast<const ChargeT*>(packed) + fr.charge_off + n_begin;
  const double* pts = points + 3 * fr.point_off;
  for (int i = tid; i < NC * P; i += kGridThreads) acc_s[i] = cmp_s[i] = Real(0);
  // runs: kStage / kFewRun per full stage, the last stage's last one shorter
  const int runs = (n / kStage) * (kStage / kFewRun) + (n % kStage + kFewRun - 1) / kFewRun;
  const int rb = kUnits / P;  // runs per pass
  for (int r0 = 0; r0 < runs; r0 += rb) {
    const int nr = min(rb, runs - r0);
    __syncthreads();
    for (int i = tid; i < nr * P; i += kGridThreads) {
      const int r = i / P, p = i - r * P;
      const Real x = to_real<Real>(pts[3 * p]), y = to_real<Real>(pts[3 * p + 1]),
                 z = to_real<Real>(pts[3 * p + 2]);
      const int j0 = (r0 + r) * kFewRun, cnt = min(kFewRun, n - j0);
      Real part[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) part[c] = Real(0);
#pragma unroll 8
      for (int j = 0; j < cnt; ++j) {
        const ChargeT ch = src[j0 + j];
        if constexpr (PREC == kFP32C) {
          const float dx = __fsub_rn(x, __uint_as_float(static_cast<uint32_t>(ch.xy.x)));
          const float dy = __fsub_rn(y, __uint_as_float(static_cast<uint32_t>(ch.xy.y)));
          const float dz = __fsub_rn(z, __uint_as_float(static_cast<uint32_t>(ch.zq.x)));
          const float q = __uint_as_float(static_cast<uint32_t>(ch.zq.y));
          float r2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
          if (CLAMP && r2 < 1e-6f) r2 = 1e-6f;
          const float ri = rsqrt_mufu(r2);
          if constexpr (KIND == kField) {
            const float w = __fmul_rn(__fmul_rn(q, ri), __fmul_rn(ri, ri));
            part[0] = __fmaf_rn(w, dx, part[0]);
            part[1] = __fmaf_rn(w, dy, part[1]);
            part[2] = __fmaf_rn(w, dz, part[2]);
          } else {
            part[0] = __fmaf_rn(q, ri, part[0]);
          }
        } else {
          const double dx = x - ch.x, dy = y - ch.y, dz = z - ch.z;
          double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
          if (CLAMP && r2 < 1e-6) r2 = 1e-6;
          const double w = weight_f64<KIND>(ch, r2);
          if constexpr (KIND == kField) {
            part[0] = __fma_rn(w, dx, part[0]);
            part[1] = __fma_rn(w, dy, part[1]);
            part[2] = __fma_rn(w, dz, part[2]);
          } else {
            part[0] = __dadd_rn(part[0], w);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) sums[c][i] = part[c];
    }
    __syncthreads();
    for (int i = tid; i < NC * P; i += kGridThreads) {
      const int c = i / P, p = i - c * P;
      Real acc = acc_s[i];
      [[maybe_unused]] Real cmp = cmp_s[i];
#pragma unroll 4
      for (int r = 0; r < nr; ++r) {
        if constexpr (PREC == kFP32C)
          kahan_add(acc, cmp, sums[c][r * P + p]);
        else
          acc = __dadd_rn(acc, sums[c][r * P + p]);
      }
      acc_s[i] = acc;
      if constexpr (PREC == kFP32C) cmp_s[i] = cmp;
    }
  }
  __syncthreads();
  constexpr int kTilePts = kGridThreads * PPT;
  for (int i = tid; i < NC * P; i += kGridThreads) {
    const int c = i / P, p = i - c * P;
    double v;
    if constexpr (PREC == kFP32C)
      v = __dmul_rn(__dsub_rn(widen(acc_s[i]), widen(cmp_s[i])), kCoulomb);
    else
      v = acc_s[i] * kCoulomb;
    if (fr.slot_base < 0)
      out[NC * (fr.point_off + p) + c] = v;
    else
      partial[(static_cast<int64_t>(fr.slot_base + split) * NC + c) * kTilePts + p] = v;
  }
}

// Integer-only reads of doubles.  GB300's FP64 pipe is 1/64 of its FP32 pipe
// and conversions from double run on it, so the refinement's helpers take a
// double apart with integer operations.
//   dbl_hi_float: sign, exponent and the leading 24 significand bits (the rest
//                 truncated); beyond the float range +-inf, below its normal
//                 range +-0; NaN stays NaN.
//   dbl_lo_float: the remaining 29 significand bits, v - dbl_hi_float(v),
//                 rounded to a float (|error| <= 2^-48 |v|); 0 where the high
//                 part is not a normal float, and flushed to 0 where it would
//                 be subnormal (|v| below about 1e-30: an absolute error
//                 under 1e-37).
__device__ __forceinline__ float dbl_hi_float(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  const uint32_t sign = static_cast<uint32_t>(b >> 32) & 0x80000000u;
  const int ex = static_cast<int>((b >> 52) & 0x7ff);
  const uint32_t mant = static_cast<uint32_t>((b >> 29) & 0x7fffffu);
  if (ex == 0x7ff) return __uint_as_float(sign | 0x7f800000u | (mant ? 0x400000u : 0u));
  const int e = ex - 1023 + 127;
  if (e >= 255) return __uint_as_float(sign | 0x7f800000u);
  if (e <= 0) return __uint_as_float(sign);
  return __uint_as_float(sign | (static_cast<uint32_t>(e) << 23) | mant);
}
__device__ __forceinline__ float dbl_lo_float(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  const uint32_t sign = static_cast<uint32_t>(b >> 32) & 0x80000000u;
  const int ex = static_cast<int>((b >> 52) & 0x7ff);
  const uint32_t r = static_cast<uint32_t>(b & 0x1fffffffull);  // 29 bits, weight 2^(ex - 1075)
  const int e_hi = ex - 1023 + 127;
  if (r == 0 || e_hi <= 0 || e_hi >= 255) return 0.f;
  const int t = 31 - __clz(static_cast<int>(r));  // top set bit, 0..28
  uint32_t m;
  int fe = ex - 1075 + t + 127;                   // float exponent of r's top bit
  if (t > 23) {                                   // round the low t - 23 bits, half up
    const int sh = t - 23;
    m = (r >> sh) + ((r >> (sh - 1)) & 1u);
    if (m == (1u << 24)) {
      m >>= 1;
      ++fe;
    }
  } else {
    m = r << (23 - t);
  }
  if (fe <= 0) return __uint_as_float(sign);
  return __uint_as_float(sign | (static_cast<uint32_t>(fe) << 23) | (m & 0x7fffffu));
}

// |E|^2 of one output row in FP32 from the truncated components (integer
// conversion, three FP32 operations): the key of the magnitude histogram.
__device__ __forceinline__ float field_norm2(const double* e) {
  const float x = dbl_hi_float(e[0]), y = dbl_hi_float(e[1]), z = dbl_hi_float(e[2]);
  return __fmaf_rn(x, x, __fmaf_rn(y, y, __fmul_rn(z, z)));
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// One frame of few points, FP32C, in one launch: as grid_few_kernel and the sum
// over the splits, by one cluster of CTAs that read the caller's arrays.  CTA r
// takes the splits r, r + kPointCtas, ...; the splits' results go to CTA 0's shared
// memory, which adds them in split order.  The smallest calls are a chain of
// launches (27 us of GPU time for packing, sums and the sum over the splits of one
// point and 8,000 charges); one CTA alone took 37 us for reading the charges.
constexpr int kPointCtas = 8;
constexpr int kPointThreads = 256;
constexpr int kPointUnits = 2048;       // (point, run) units per CTA at most
constexpr int kPointResults = 2048;     // results of all splits at most
constexpr int kPointCharges = 4096;     // charges per CTA at most

template <int KIND, bool CLAMP>
__global__ void __cluster_dims__(kPointCtas, 1, 1) __launch_bounds__(kPointThreads)
    grid_point_kernel(const GridFrame fr, const double* __restrict__ points, const double* __restrict__ x,
                      const double* __restrict__ q, double* __restrict__ out) {
  constexpr int NC = (KIND == kField) ? 3 : 1;
  extern __shared__ __align__(16) unsigned char point_smem[];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  // CTA 0's shared memory may be written once all CTAs of the cluster run: arrived
  // at here, waited for before the first of those stores, behind the charges' loads
  cluster_arrive();
  const int rank = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x;
  const int P = fr.n_points, ns = fr.n_split, chunk = fr.chunk, n_all = fr.n_charges;
  const int rps = (chunk + kKahanRun - 1) / kKahanRun;  // runs per split
  const int mine = (ns - rank + kPointCtas - 1) / kPointCtas;
  const int most = (ns + kPointCtas - 1) / kPointCtas;
  const int units = P * most * rps;
  float4* ch_s = reinterpret_cast<float4*>(point_smem);                  // [most][chunk]
  double* v_s = reinterpret_cast<double*>(ch_s + most * chunk);          // [ns][NC * P], CTA 0's used
  float* sums = reinterpret_cast<float*>(v_s + ns * NC * P);             // [NC][units]
  const double* pts = points + 3 * fr.point_off;
  const double* xs = x + 3 * fr.charge_off;
  const double* qs = q + fr.charge_off;
#pragma unroll 4
  for (int i = tid; i < mine * chunk; i += kPointThreads) {
    const int k = i / chunk, j = (rank + k * kPointCtas) * chunk + (i - k * chunk);
    if (j < n_all) {
      const double* xj = xs + 3 * static_cast<int64_t>(j);
      ch_s[i] = make_float4(narrow(xj[0]), narrow(xj[1]), narrow(xj[2]), narrow(qs[j]));
    }
  }
  __syncthreads();
  for (int i = tid; i < mine * rps * P; i += kPointThreads) {
    const int p = i % P, kr = i / P, k = kr / rps, r = kr - k * rps;
    const float px = narrow(pts[3 * p]), py = narrow(pts[3 * p + 1]), pz = narrow(pts[3 * p + 2]);
    const int n = min(chunk, n_all - (rank + k * kPointCtas) * chunk);
    const int cnt = max(0, min(kKahanRun, n - r * kKahanRun));
    const float4* src = ch_s + k * chunk + r * kKahanRun;
    float part[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) part[c] = 0.f;
#pragma unroll 8
    for (int j = 0; j < cnt; ++j) {
      const float4 ch = src[j];
      const float dx = __fsub_rn(px, ch.x);
      const float dy = __fsub_rn(py, ch.y);
      const float dz = __fsub_rn(pz, ch.z);
      float r2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
      if (CLAMP && r2 < 1e-6f) r2 = 1e-6f;
      const float ri = rsqrt_mufu(r2);
      if constexpr (KIND == kField) {
        const float w = __fmul_rn(__fmul_rn(ch.w, ri), __fmul_rn(ri, ri));
        part[0] = __fmaf_rn(w, dx, part[0]);
        part[1] = __fmaf_rn(w, dy, part[1]);
        part[2] = __fmaf_rn(w, dz, part[2]);
      } else {
        part[0] = __fmaf_rn(ch.w, ri, part[0]);
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) sums[c * units + i] = part[c];
  }
  __syncthreads();
  cluster_wait();
  double* v_0 = cluster.map_shared_rank(v_s, 0);
  for (int i = tid; i < mine * NC * P; i += kPointThreads) {
    const int k = i / (NC * P), cp = i - k * (NC * P), c = cp / P, p = cp - c * P;
    const int split = rank + k * kPointCtas;
    const int n = min(chunk, n_all - split * chunk);
    const int nr = (n + kKahanRun - 1) / kKahanRun;
    const float* in = sums + c * units + (k * rps) * P + p;
    float acc = 0.f, cmp = 0.f;
#pragma unroll 4
    for (int r = 0; r < nr; ++r) kahan_add(acc, cmp, in[r * P]);
    v_0[split * NC * P + cp] = __dmul_rn(__dsub_rn(widen(acc), widen(cmp)), kCoulomb);
  }
  cluster.sync();
  if (rank != 0) return;
  const int l = tid % kSumLanes;
  for (int i0 = 0; i0 < NC * P; i0 += kPointThreads / kSumLanes) {
    const int i = min(i0 + tid / kSumLanes, NC * P - 1);
    double v = l < ns ? v_s[l * NC * P + i] : 0.0;
#pragma unroll 4
    for (int split = l + kSumLanes; split < ns; split += kSumLanes) v = __dadd_rn(v, v_s[split * NC * P + i]);
    if (ns > 1) v = sum_lanes(v);
    const int c = i / P, p = i - c * P;
    if (l == 0) out[NC * (fr.point_off + p) + c] = v;
  }
}

constexpr int kMagBins = 4096;  // bits 30..19 of the float |E|^2: exponent + 4 mantissa bits

// A frame's scale from its histogram, by a whole block: the lower edge of the bin that
// holds the lower median.
__device__ __forceinline__ void frame_scale(const int* row, float* scale) {
  const int tid = threadIdx.x, lane = tid & 31;
  // 32 consecutive bins per thread
  constexpr int kPer = kMagBins / kGridThreads;
  __shared__ int warp_sum[kGridThreads / 32];
  int own[kPer], mine = 0;
#pragma unroll
  for (int b = 0; b < kPer; b += 4) {
    const int4 h = __ldcg(reinterpret_cast<const int4*>(row + tid * kPer + b));
    own[b] = h.x;
    own[b + 1] = h.y;
    own[b + 2] = h.z;
    own[b + 3] = h.w;
    mine += h.x + h.y + h.z + h.w;
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int w = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += w;
  }
  if (lane == 31) warp_sum[tid >> 5] = incl;
  __syncthreads();
  int total = 0;
#pragma unroll
  for (int w = 0; w < kGridThreads / 32; ++w) {
    if (w < (tid >> 5)) incl += warp_sum[w];
    total += warp_sum[w];
  }
  const int rank = (total - 1) / 2;
  if (total > 0 && incl > rank && incl - mine <= rank) {
    int cum = incl - mine, bin_of_rank = tid * kPer;
#pragma unroll
    for (int b = 0; b < kPer; ++b) {
      if (cum <= rank && cum + own[b] > rank) bin_of_rank = tid * kPer + b;
      cum += own[b];
    }
    *scale = __uint_as_float(static_cast<uint32_t>(bin_of_rank) << 19);
  }  // no finite value: the scale stays 0 and nothing is refined
}

// A row's bin; -1: not finite (NaN compares false).
__device__ __forceinline__ int mag_bin(const double (&v)[3]) {
  const float m2 = field_norm2(v);
  return m2 <= 3.0e38f ? static_cast<int>(__float_as_uint(m2) >> 19) : -1;
}

// A point's sum over its frame's splits, by one thread (th: thread of the tile t).
template <int NC, int PPT>
__device__ __forceinline__ void thread_sums(const GridFrame& fr, const double* __restrict__ partial, int t, int k,
                                            int th, int ns, double (&v)[NC]) {
  constexpr int kTilePts = kGridThreads * PPT;
  const double* in = partial + (static_cast<int64_t>(fr.slot_base + t) * NC) * kTilePts + k * kGridThreads + th;
  const int64_t step = static_cast<int64_t>(fr.n_tiles) * NC * kTilePts;
  double w[NC][kSumLanes];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int s = 0; s < kSumLanes; ++s) w[c][s] = s < ns ? in[s * step + c * kTilePts] : 0.0;
  for (int s0 = kSumLanes; s0 < ns; s0 += kSumLanes) {
#pragma unroll
    for (int s = 0; s < kSumLanes; ++s)
      if (s0 + s < ns) {
#pragma unroll
        for (int c = 0; c < NC; ++c) w[c][s] = __dadd_rn(w[c][s], in[(s0 + s) * step + c * kTilePts]);
      }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) v[c] = sum_thread(w[c]);
}

// The k-th point of thread th of a frame's tile t; -1 for none.
template <int PPT>
__device__ __forceinline__ int tile_point(const GridFrame& fr, const PointMap& map, int t, int th, int k) {
  if (fr.few) return k * kGridThreads + th < fr.n_points ? k * kGridThreads + th : -1;
  return map.point<PPT>(t * kGridThreads + th, k);
}

// Sums of the splits.  LANES = 1: block (tile, k), a thread takes the k-th point of
// a tile's thread; LANES = 8: eight lanes per point and eight blocks.  HIST
// (FP32C field refinement): also counts |E|^2 in 1/16-octave bins (of |E|^2; 1/32
// octave of |E|) per frame, exact integers, and a frame's last block takes the
// scale from them: the lower edge of the bin that holds the lower median.
template <int PREC, int KIND, int PPT, bool HIST, int LANES>
__global__ void __launch_bounds__(kGridThreads)
    grid_final_kernel(const GridFrame* __restrict__ frames, int n_frames, const GridFrame one,
                      const int* __restrict__ stride, const int* __restrict__ broken,
                      const double* __restrict__ partial, double* __restrict__ out, int* __restrict__ hist,
                      int* __restrict__ done, float* __restrict__ scale) {
  constexpr int NC = (KIND == kField) ? 3 : 1;
  constexpr int kTilePts = kGridThreads * PPT;
  constexpr int kBlocks = PPT * LANES;  // per tile
  const int tid = threadIdx.x, lane = tid & 31;
  const int tile = static_cast<int>(blockIdx.x) / kBlocks, part = static_cast<int>(blockIdx.x) % kBlocks;
  const int k = part / LANES;
  const int th = ((part % LANES) * kGridThreads + tid) / LANES;  // thread of the tile
  const int l = tid % LANES;
  int f;
  const GridFrame fr = load_frame<offsetof(GridFrame, tile_base)>(frames, n_frames, one, tile, &f);
  const int t = tile - fr.tile_base;
  PointMap map;
  map.set<PPT>(stride && !broken[f] ? stride[f] : 0, fr.n_points);
  const int pl = tile_point<PPT>(fr, map, t, th, k);
  double v[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) v[c] = 0.0;
  double* o = out + NC * (fr.point_off + max(pl, 0));
  if (fr.slot_base >= 0) {
    const int ns = pl >= 0 ? fr.n_split : 0;
    if constexpr (LANES == 1) {
      thread_sums<NC, PPT>(fr, partial, t, k, th, ns, v);
    } else {
      const double* in = partial + (static_cast<int64_t>(fr.slot_base + t) * NC) * kTilePts + k * kGridThreads + th;
      const int64_t step = static_cast<int64_t>(fr.n_tiles) * NC * kTilePts;
#pragma unroll
      for (int c = 0; c < NC; ++c) v[c] = l < ns ? in[l * step + c * kTilePts] : 0.0;
#pragma unroll 4
      for (int s = l + LANES; s < ns; s += LANES)
#pragma unroll
        for (int c = 0; c < NC; ++c) v[c] = __dadd_rn(v[c], in[s * step + c * kTilePts]);
#pragma unroll
      for (int c = 0; c < NC; ++c) v[c] = sum_lanes(v[c]);
    }
    if (pl >= 0 && l == 0)
#pragma unroll
      for (int c = 0; c < NC; ++c) o[c] = v[c];
  } else if (HIST && pl >= 0) {
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = o[c];
  }
  if constexpr (HIST) {
    int* row = hist + static_cast<int64_t>(f) * kMagBins;
    const int bin = pl >= 0 && l == 0 ? mag_bin(v) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, bin);
    if (bin >= 0 && lane == __ffs(same) - 1) atomicAdd(&row[bin], __popc(same));
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&done[f], 1) == fr.n_tiles * kBlocks - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    frame_scale(row, scale + f);
  }
}

// The same with one thread per point for many points (FP32C field): a block takes
// `per` tiles and counts in shared memory, so that a frame's hot bins get one addition
// per block instead of one per warp, and a frame one last-block check per block.  A
// call of 101^3 points in no order x 20 charges 84 us (158 with the kernel above, 4e6
// points 219 and 271); below about 300 tiles the blocks' 4,096 bins cost more than they
// save (51^3 x 5,000, 260 tiles, 331 and 326; 24 frames of 20,000 points 670 and 674).
// Eight blocks per SM: 219 us, 223 with six, 241 with the four of 128 registers.
constexpr int kManyTiles = 300;
template <int PPT>
__global__ void __launch_bounds__(kGridThreads, 8)
    grid_final_many_kernel(const GridFrame* __restrict__ frames, int n_frames, const GridFrame one, int n_tiles,
                           int per, const int* __restrict__ stride, const int* __restrict__ broken,
                           const double* __restrict__ partial, double* __restrict__ out, int* __restrict__ hist,
                           int* __restrict__ done, float* __restrict__ scale) {
  __shared__ int h[kMagBins];
  __shared__ int s_last;
  const int tid = threadIdx.x;
  for (int b = tid; b < kMagBins; b += kGridThreads) h[b] = 0;
  __syncthreads();
  const int t1 = min(n_tiles, (static_cast<int>(blockIdx.x) + 1) * per);
  int tile = static_cast<int>(blockIdx.x) * per;
  while (tile < t1) {
    int f;
    const GridFrame fr = load_frame<offsetof(GridFrame, tile_base)>(frames, n_frames, one, tile, &f);
    PointMap map;
    map.set<PPT>(stride && !broken[f] ? stride[f] : 0, fr.n_points);
    const int first = tile, end = min(t1, fr.tile_base + fr.n_tiles);
    for (; tile < end; ++tile) {
#pragma unroll
      for (int k = 0; k < PPT; ++k) {
        const int pl = tile_point<PPT>(fr, map, tile - fr.tile_base, tid, k);
        if (pl < 0) continue;
        double* o = out + 3 * (fr.point_off + pl);
        double v[3];
        if (fr.slot_base >= 0) {
          thread_sums<3, PPT>(fr, partial, tile - fr.tile_base, k, tid, fr.n_split, v);
#pragma unroll
          for (int c = 0; c < 3; ++c) o[c] = v[c];
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) v[c] = o[c];
        }
        const int bin = mag_bin(v);
        if (bin >= 0) atomicAdd(&h[bin], 1);
      }
    }
    // this block's part of the frame, and the frame's scale by its last block
    int* row = hist + static_cast<int64_t>(f) * kMagBins;
    __syncthreads();
    for (int b = tid; b < kMagBins; b += kGridThreads)
      if (h[b]) {
        atomicAdd(&row[b], h[b]);
        h[b] = 0;
      }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&done[f], end - first) + (end - first) == fr.n_tiles;
    __syncthreads();
    if (s_last) {
      __threadfence();
      frame_scale(row, scale + f);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// FP32C field refinement (see the header comment).
// ---------------------------------------------------------------------------
constexpr int kFlagThreads = 256;
constexpr int kFlagChunk = kFlagThreads * 4;  // points of a frame per flagging CTA
// 512 threads of at most 64 registers: the refinement CTAs must fit beside a
// serving engine launch that holds half of every SM's registers (engine.cu), as
// the grid CTAs do.
constexpr int kRefineThreads = 512;

// Grid (frame, chunk of kFlagChunk points): appends each point of the chunk with
// |E|^2 below tau^2 times the frame's scale to list[] as {output row, frame}.
// The counts behind the scale are exact integers, so the threshold and the set
// of points are deterministic.
__global__ void __launch_bounds__(kFlagThreads)
    grid_flag_kernel(const GridFrame* __restrict__ frames, const GridFrame one, const double* __restrict__ out,
                     const float* __restrict__ scale, float tau2, int64_t* __restrict__ list,
                     int* __restrict__ count) {
  __shared__ int part[kFlagThreads / 32 + 1];
  const int64_t po = gridDim.x == 1 ? one.point_off : frames[blockIdx.x].point_off;
  const int64_t P = gridDim.x == 1 ? one.n_points : frames[blockIdx.x].n_points;
  const float thr = __fmul_rn(tau2, scale[blockIdx.x]);
  constexpr int kPer = kFlagChunk / kFlagThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.y) * kFlagChunk; i0 < P;
       i0 += static_cast<int64_t>(gridDim.y) * kFlagChunk) {
    const int64_t i1 = min(P, i0 + kFlagChunk);
    // the chunk's points below the threshold, in thread order (point i0 + t +
    // kFlagThreads * k belongs to thread t), appended as one contiguous block
    unsigned mask = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int64_t i = i0 + threadIdx.x + int64_t(k) * kFlagThreads;
      if (i < i1 && field_norm2(out + 3 * (po + i)) < thr) mask |= 1u << k;
    }
    if (!__syncthreads_or(mask != 0)) continue;
    const int mine = __popc(mask);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      int run = 0;
      for (int w = 0; w < kFlagThreads / 32; ++w) {
        const int c = part[w];
        part[w] = run;
        run += c;
      }
      part[kFlagThreads / 32] = atomicAdd(count, run);
    }
    __syncthreads();
    int k_out = part[kFlagThreads / 32] + part[warp] + incl - mine;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (mask & (1u << k)) {
        list[2 * static_cast<int64_t>(k_out)] = po + i0 + threadIdx.x + int64_t(k) * kFlagThreads;
        list[2 * static_cast<int64_t>(k_out) + 1] = blockIdx.x;
        ++k_out;
      }
    }
  }
}

// Double-float ("float-float") arithmetic: a value is an unevaluated sum
// h + l of two floats with |l| <= ulp(h)/2, about 48 significant bits, built
// from the error-free transformations TwoSum (Knuth) and TwoProduct by FMA
// (Dekker / Kahan; see Muller et al., Handbook of Floating-Point Arithmetic,
// ch. 4 and 14).  Every operation below is written with explicit roundings
// (__fadd_rn, __fmul_rn, __fmaf_rn) so the compiler cannot contract or
// reorder the error terms.
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
  p = __fmul_rn(a, b);
  e = __fmaf_rn(a, b, -p);
}

// 1e-6 as a double-float pair: the float nearest to it and the float nearest
// to the rest (1e-6 - 9.99999997e-7 = 2.5e-15).
constexpr float kClampH = 1e-6f;
constexpr float kClampL = static_cast<float>(1e-6 - static_cast<double>(1e-6f));

// The field term of one charge at one point in double-float, added to
// (sh[k], sl[k]).  Point (ph, pl), charge coordinates (ch, cl) and charge
// (qh, ql) as float pairs.  Relative error of the term about 1e-13.
template <bool CLAMP>
__device__ __forceinline__ void df_field_term(const float (&ph)[3], const float (&pl)[3],
                                              const float4& chq, const float4& clq,
                                              float (&sh)[3], float (&sl)[3]) {
  const float ch[3] = {chq.x, chq.y, chq.z}, cl[3] = {clq.x, clq.y, clq.z};
  float dh[3], dl[3], sq[3], sqe[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float e;
    two_sum(ph[k], -ch[k], dh[k], e);                      // dh + e = ph - ch exactly
    dl[k] = __fadd_rn(e, __fsub_rn(pl[k], cl[k]));
    {  // renormalise: ph - ch may be exact (e = 0) while pl - cl is not small against it
      const float h = __fadd_rn(dh[k], dl[k]);
      dl[k] = __fsub_rn(dl[k], __fsub_rn(h, dh[k]));
      dh[k] = h;
    }
    two_prod(dh[k], dh[k], sq[k], sqe[k]);                 // dh^2 exactly
    sqe[k] = __fmaf_rn(__fadd_rn(dh[k], dh[k]), dl[k], sqe[k]);  // + 2 dh dl
  }
  float t1, e1, r2h, e2;
  two_sum(sq[0], sq[1], t1, e1);
  two_sum(t1, sq[2], r2h, e2);
  float r2l = __fadd_rn(__fadd_rn(e1, e2), __fadd_rn(__fadd_rn(sqe[0], sqe[1]), sqe[2]));
  {  // renormalise (|r2h| >= |r2l|)
    const float h = __fadd_rn(r2h, r2l);
    r2l = __fsub_rn(r2l, __fsub_rn(h, r2h));
    r2h = h;
  }
  // compute_looped_field's r^2 >= 1e-6, compared as double-float values
  // (lexicographically: both pairs are normalised), FP32 operations only.
  if (CLAMP && (r2h < kClampH || (r2h == kClampH && r2l < kClampL))) {
    r2h = kClampH;
    r2l = kClampL;
  }
  // r^-1: MUFU seed refined by one Newton step with the residual in double-float
  const float y0 = rsqrt_mufu(r2h);
  float a, ae, b, be;
  two_prod(y0, y0, a, ae);                                  // a + ae = y0^2
  two_prod(r2h, a, b, be);                                  // b + be = r2h a
  const float t = __fadd_rn(__fsub_rn(b, 1.0f), __fmaf_rn(r2h, ae, __fmaf_rn(r2l, a, be)));
  const float yl = __fmul_rn(__fmul_rn(-0.5f, y0), t);     // y = y0 + yl
  // y^3 = (a + (ae + 2 y0 yl)) (y0 + yl)
  const float y2l = __fmaf_rn(__fadd_rn(y0, y0), yl, ae);
  float y3h, e3;
  two_prod(a, y0, y3h, e3);
  const float y3l = __fmaf_rn(a, yl, __fmaf_rn(y2l, y0, e3));
  // w = q y^3
  float wh, e4;
  two_prod(chq.w, y3h, wh, e4);
  const float wl = __fmaf_rn(chq.w, y3l, __fmaf_rn(clq.w, y3h, e4));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float p, pe, s, se;
    two_prod(wh, dh[k], p, pe);
    const float plo = __fmaf_rn(wh, dl[k], __fmaf_rn(wl, dh[k], pe));
    two_sum(sh[k], p, s, se);
    sh[k] = s;
    sl[k] = __fadd_rn(sl[k], __fadd_rn(se, plo));
  }
}

// Sum of two double-float values (h, l), renormalised.
__device__ __forceinline__ void df_add(float& h, float& l, float bh, float bl) {
  float s, e;
  two_sum(h, bh, s, e);
  e = __fadd_rn(e, __fadd_rn(l, bl));
  h = __fadd_rn(s, e);
  l = __fsub_rn(e, __fsub_rn(h, s));
}

// Recomputes the listed points in double-float arithmetic: one CTA per point
// at a time, the frame's charges (double-float records of prep_kernel) split
// over the threads.  A launch has few points, so what counts is one point's
// latency: a thread loads the next two charges while it evaluates two, into
// independent sums, which are added at the end; the threads' sums are combined
// by a fixed tree.
template <bool CLAMP>
__global__ void __launch_bounds__(kRefineThreads, 2)
    grid_refine_kernel(const GridFrame* __restrict__ frames, const GridFrame one, const int64_t* __restrict__ list,
                       const int* __restrict__ count, const double* __restrict__ points,
                       const float4* __restrict__ dfq, double* __restrict__ out) {
  __shared__ float red[kRefineThreads / 32][6];
  const int n_list = *count;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = blockIdx.x; e < n_list; e += gridDim.x) {
    const int64_t row = list[2 * e];
    const int64_t f = list[2 * e + 1];
    const int64_t co = frames ? frames[f].charge_off : one.charge_off;
    const int n = frames ? frames[f].n_charges : one.n_charges;
    const float4* src = dfq + 2 * co;
    float ph[3], pl[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      ph[k] = dbl_hi_float(points[3 * row + k]);
      pl[k] = dbl_lo_float(points[3 * row + k]);
    }
    float sh[3] = {0.f, 0.f, 0.f}, sl[3] = {0.f, 0.f, 0.f};
    float th[3] = {0.f, 0.f, 0.f}, tl[3] = {0.f, 0.f, 0.f};
    // a charge past the end: zero charge 1 A from the point (its term is exactly 0)
    auto load = [&](int j, float4& hi, float4& lo) {
      if (j < n) {
        hi = src[2 * static_cast<int64_t>(j)];
        lo = src[2 * static_cast<int64_t>(j) + 1];
      } else {
        hi = make_float4(__fadd_rn(ph[0], 1.f), ph[1], ph[2], 0.f);
        lo = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    int j = threadIdx.x;
    float4 h0, l0, h1, l1;
    load(j, h0, l0);
    load(j + kRefineThreads, h1, l1);
    while (j < n) {
      const float4 a0 = h0, b0 = l0, a1 = h1, b1 = l1;
      j += 2 * kRefineThreads;
      load(j, h0, l0);
      load(j + kRefineThreads, h1, l1);
      df_field_term<CLAMP>(ph, pl, a0, b0, sh, sl);
      df_field_term<CLAMP>(ph, pl, a1, b1, th, tl);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) df_add(sh[k], sl[k], th[k], tl[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float bh = __shfl_xor_sync(0xffffffffu, sh[k], o);
        const float bl = __shfl_xor_sync(0xffffffffu, sl[k], o);
        df_add(sh[k], sl[k], bh, bl);
      }
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        red[warp][2 * k] = sh[k];
        red[warp][2 * k + 1] = sl[k];
      }
    __syncthreads();
    if (threadIdx.x < 3) {
      const int k = threadIdx.x;
      float h = red[0][2 * k], l = red[0][2 * k + 1];
#pragma unroll
      for (int w = 1; w < kRefineThreads / 32; ++w) df_add(h, l, red[w][2 * k], red[w][2 * k + 1]);
      out[3 * row + k] = (static_cast<double>(h) + static_cast<double>(l)) * kCoulomb;
    }
    __syncthreads();
  }
}

constexpr int kPrepThreads = 256;
// Charges per preparation block: one per thread, as the loads' latency is what a small
// launch waits for (2,000 charges 3.3 us, 5.3 with four per thread).
constexpr int kPrepCharges = 256;

__device__ __forceinline__ bool same_yz(const double* a, const double* b, bool f32) {
  if (f32)  // the FP32C kernels see the FP32 images
    return __float_as_uint(narrow(a[1])) == __float_as_uint(narrow(b[1])) &&
           __float_as_uint(narrow(a[2])) == __float_as_uint(narrow(b[2]));
  return __double_as_longlong(a[1]) == __double_as_longlong(b[1]) &&
         __double_as_longlong(a[2]) == __double_as_longlong(b[2]);
}

__device__ __forceinline__ bool same_x(const double* a, const double* b, bool f32) {
  return f32 ? __float_as_uint(narrow(a[0])) == __float_as_uint(narrow(b[0]))
             : __double_as_longlong(a[0]) == __double_as_longlong(b[0]);
}

// Preparation, one launch: blocks [0, n_charge_blocks) pack the charges (FP32C:
// every component duplicated; FP64: Charge64) and, for the refinement, their
// double-float records {xh, yh, zh, qh} {xl, yl, zl, ql}; the others look for the
// frames' lattice strides, kGridPrepPoints points each.  A frame's stride is where x
// first changes; it holds if every point's (y, z) equal those one stride earlier.  stride[f] is written by the frame's
// first block, broken[f] (zeroed by the caller) by any block that finds a
// difference.
template <int PREC, bool DF>
__global__ void __launch_bounds__(kPrepThreads)
    prep_kernel(int64_t n, const double* __restrict__ x, const double* __restrict__ q,
                void* __restrict__ packed, float4* __restrict__ dfq, int n_charge_blocks,
                const GridFrame* __restrict__ frames, int n_frames, const GridFrame one,
                const double* __restrict__ points, int min_rows, int* __restrict__ stride, int* __restrict__ broken) {
  if (static_cast<int>(blockIdx.x) < n_charge_blocks) {
    const int64_t i0 = static_cast<int64_t>(blockIdx.x) * kPrepCharges;
    const int64_t i1 = min(n, i0 + kPrepCharges);
    for (int64_t i = i0 + threadIdx.x; i < i1; i += kPrepThreads) {
      const double v[4] = {x[3 * i], x[3 * i + 1], x[3 * i + 2], q[i]};
      if constexpr (PREC == kFP32C) {
        ChargeDup c;
        c.xy = make_ulonglong2(dup2(narrow(v[0])), dup2(narrow(v[1])));
        c.zq = make_ulonglong2(dup2(narrow(v[2])), dup2(narrow(v[3])));
        static_cast<ChargeDup*>(packed)[i] = c;
        if constexpr (DF) {
          dfq[2 * i] = make_float4(dbl_hi_float(v[0]), dbl_hi_float(v[1]), dbl_hi_float(v[2]),
                                   dbl_hi_float(v[3]));
          dfq[2 * i + 1] = make_float4(dbl_lo_float(v[0]), dbl_lo_float(v[1]), dbl_lo_float(v[2]),
                                       dbl_lo_float(v[3]));
        }
      } else {
        static_cast<Charge64*>(packed)[i] = Charge64{v[0], v[1], v[2], v[3]};
      }
    }
    return;
  }
  const int b = static_cast<int>(blockIdx.x) - n_charge_blocks;
  int f;
  const GridFrame fr = load_frame<offsetof(GridFrame, prep_base)>(frames, n_frames, one, b, &f);
  const int part = b - fr.prep_base;
  const int P = fr.n_points;
  const double* pts = points + 3 * fr.point_off;
  constexpr bool kF32 = PREC == kFP32C;
  __shared__ int s_first[kPrepThreads / 32];
  // x is constant over a mesh's first S points and another after them: S by search over
  // the block's threads, 257 intervals at a time (two looks for up to 66,000 points).
  // Points that are no mesh may give any S; the comparison below decides.
  const int limit = P / min_rows;  // at least min_rows rows
  int lo = 0, span = limit + 1;    // x[lo] is point 0's, x[lo + span] another's, or lies past the limit
  while (span > 1) {
    const int part = (span + kPrepThreads) / (kPrepThreads + 1);
    const int i = lo + (static_cast<int>(threadIdx.x) + 1) * part;
    const bool other = i >= lo + span || !same_x(pts, pts + 3 * static_cast<int64_t>(i), kF32);
    // the first thread that sees another x, from each warp's first
    const unsigned seen = __ballot_sync(0xffffffffu, other);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
      s_first[threadIdx.x >> 5] = seen ? static_cast<int>(threadIdx.x) + __ffs(seen) - 1 : kPrepThreads;
    __syncthreads();
    int first = kPrepThreads;
#pragma unroll
    for (int w = 0; w < kPrepThreads / 32; ++w) first = min(first, s_first[w]);
    lo += first * part;
    span = min(part, span - first * part);
  }
  const int S = lo + 1;
  const bool mesh = S <= limit && P % S == 0 && same_yz(pts, pts + 3 * static_cast<int64_t>(S), kF32);
  if (part == 0 && threadIdx.x == 0) stride[f] = mesh ? S : 0;
  if (!mesh) return;
  const int64_t j0 = max(static_cast<int64_t>(part) * kGridPrepPoints, static_cast<int64_t>(S));
  const int64_t j1 = min(static_cast<int64_t>(P), static_cast<int64_t>(part + 1) * kGridPrepPoints);
  bool bad = false;
#pragma unroll 4
  for (int64_t j = j0 + threadIdx.x; j < j1; j += kPrepThreads)
    bad |= !same_yz(pts + 3 * j, pts + 3 * (j - S), kF32);
  if (__syncthreads_or(bad) && threadIdx.x == 0) broken[f] = 1;
}

__global__ void pack_f64_kernel(int64_t n, int64_t n_pad, const double* __restrict__ x,
                                const double* __restrict__ q, Charge64* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_pad;
       i += (int64_t)gridDim.x * blockDim.x) {
    Charge64 c;
    if (i < n) {
      c.x = x[3 * i];
      c.y = x[3 * i + 1];
      c.z = x[3 * i + 2];
      c.q = q[i];
    } else {
      c.x = c.y = c.z = 1.0e4;
      c.q = 0.0;
    }
    out[i] = c;
  }
}

// Layout of GridLaunch::zeroed.
struct Zeroed {
  int *stride, *broken, *done, *count, *hist;
  float* scale;
  Zeroed(int* base, int n_frames)
      : stride(base), broken(base + n_frames), done(base + 2 * n_frames), count(base + 4 * n_frames),
        hist(base + ((4 * n_frames + 1 + 3) & ~3)), scale(reinterpret_cast<float*>(base + 3 * n_frames)) {}
};

template <int PREC, int KIND, bool CLAMP, int PPT>
cudaError_t launch_grid_c(const GridLaunch& g, cudaStream_t s) {
  const Zeroed z(g.zeroed, g.n_frames);
  const bool refine = g.tau > 0.0;
  const int charge_blocks = static_cast<int>((g.n_charges + kPrepCharges - 1) / kPrepCharges);
  float4* dfq = static_cast<float4*>(g.dfq);
  const int* stride = g.n_prep > 0 ? z.stride : nullptr;  // null: no frame is looked at for a mesh
  if (charge_blocks + g.n_prep > 0) {
    if (refine && PREC == kFP32C)
      prep_kernel<PREC, PREC == kFP32C><<<charge_blocks + g.n_prep, kPrepThreads, 0, s>>>(
          g.n_charges, g.x, g.q, g.packed, dfq, charge_blocks, g.frames, g.n_frames, g.one, g.points, PPT, z.stride,
          z.broken);
    else
      prep_kernel<PREC, false><<<charge_blocks + g.n_prep, kPrepThreads, 0, s>>>(
          g.n_charges, g.x, g.q, g.packed, dfq, charge_blocks, g.frames, g.n_frames, g.one, g.points, PPT, z.stride,
          z.broken);
  }
  if (g.few_items > 0)
    grid_few_kernel<PREC, KIND, CLAMP, PPT>
        <<<g.few_items, kGridThreads, 0, s>>>(g.frames, g.n_frames, g.one, g.packed, g.points, g.out, g.partial);
  if (g.n_items > g.few_items) {
    // same carveout as the streamline engine, so both fit on one SM
    cudaFuncSetAttribute(grid_kernel<PREC, KIND, CLAMP, PPT>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    grid_kernel<PREC, KIND, CLAMP, PPT><<<g.n_items - g.few_items, kGridThreads, 0, s>>>(
        g.frames, g.n_frames, g.one, g.few_items, stride, z.broken, g.packed, g.points, g.out, g.partial, g.status);
  }
  // Eight lanes per point where that is shorter: FP64 additions per scheduler with
  // one thread per point against eight.
  const double splits = double(g.n_items) / std::max(g.n_tiles, 1);
  const double warps = double(g.n_tiles) * PPT * (kGridThreads / 32) / (4.0 * std::max(g.num_sms, 1));
  const bool lanes = std::max(1.0, 8.0 * warps) * (splits / 8.0 + 3.0) < std::max(1.0, warps) * splits;
  auto final = [&](auto hist, auto ln) {
    constexpr int L = decltype(ln)::value;
    grid_final_kernel<PREC, KIND, PPT, decltype(hist)::value, L><<<g.n_tiles * PPT * L, kGridThreads, 0, s>>>(
        g.frames, g.n_frames, g.one, stride, z.broken, g.partial, g.out, z.hist, z.done, z.scale);
  };
  auto final_lanes = [&](auto hist) {
    if (lanes)
      final(hist, std::integral_constant<int, kSumLanes>{});
    else
      final(hist, std::integral_constant<int, 1>{});
  };
  if (refine) {
    if constexpr (KIND == kField && PREC == kFP32C) {
      if (!lanes && g.n_tiles >= kManyTiles) {
        const int per = std::max(1, g.n_tiles / (8 * std::max(g.num_sms, 1)));
        grid_final_many_kernel<PPT><<<(g.n_tiles + per - 1) / per, kGridThreads, 0, s>>>(
            g.frames, g.n_frames, g.one, g.n_tiles, per, stride, z.broken, g.partial, g.out, z.hist, z.done, z.scale);
      } else {
        final_lanes(std::true_type{});
      }
      const dim3 fgrid(g.n_frames, std::min((g.max_points - 1) / kFlagChunk + 1, 65535));
      grid_flag_kernel<<<fgrid, kFlagThreads, 0, s>>>(g.frames, g.one, g.out, z.scale,
                                                      static_cast<float>(g.tau * g.tau), g.list, z.count);
      grid_refine_kernel<CLAMP><<<std::max(g.num_sms, 1) * 4, kRefineThreads, 0, s>>>(
          g.n_frames == 1 ? nullptr : g.frames, g.one, g.list, z.count, g.points, dfq, g.out);
    }
  } else if (g.partial) {
    final_lanes(std::false_type{});
  }
  return cudaGetLastError();
}

template <int PREC, int KIND, int PPT>
cudaError_t launch_grid_k(const GridLaunch& g, cudaStream_t s) {
  if constexpr (KIND == kField)
    if (g.clamp) return launch_grid_c<PREC, KIND, true, PPT>(g, s);
  return launch_grid_c<PREC, KIND, false, PPT>(g, s);
}

template <int PREC, int KIND, bool CLAMP, int PPT>
cudaError_t preload_c() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, grid_kernel<PREC, KIND, CLAMP, PPT>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_few_kernel<PREC, KIND, CLAMP, PPT>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, prep_kernel<PREC, false>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_final_kernel<PREC, KIND, PPT, false, 1>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_final_kernel<PREC, KIND, PPT, false, kSumLanes>);
  if constexpr (PREC == kFP32C)
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_point_kernel<KIND, CLAMP>);
  if constexpr (KIND == kField && PREC == kFP32C) {
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, prep_kernel<PREC, true>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_final_kernel<PREC, KIND, PPT, true, 1>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_final_kernel<PREC, KIND, PPT, true, kSumLanes>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_final_many_kernel<PPT>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_flag_kernel);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, grid_refine_kernel<CLAMP>);
  }
  return e;
}

// Calls f with the launch's (precision, kind, points per thread) as constants.
template <typename F>
cudaError_t with_form(int prec, int kind, int ppt, F f) {
  auto by_ppt = [&](auto p, auto k) {
    return ppt == 8 ? f(p, k, std::integral_constant<int, 8>{}) : f(p, k, std::integral_constant<int, 4>{});
  };
  auto by_kind = [&](auto p) {
    return kind == kField ? by_ppt(p, std::integral_constant<int, kField>{})
                          : by_ppt(p, std::integral_constant<int, kEsp>{});
  };
  return prec == kFP32C ? by_kind(std::integral_constant<int, kFP32C>{})
                        : by_kind(std::integral_constant<int, kFP64>{});
}

}  // namespace

namespace {
struct PointSizes {
  int64_t charges, units, results;
  explicit PointSizes(const GridLaunch& g) {
    const int64_t most = (g.one.n_split + kPointCtas - 1) / kPointCtas;
    charges = most * g.one.chunk;
    units = most * g.one.n_points * ((int64_t(g.one.chunk) + kKahanRun - 1) / kKahanRun);
    results = int64_t(g.one.n_split) * g.one.n_points * (g.kind == kField ? 3 : 1);
  }
};
}  // namespace

bool grid_point_fits(const GridLaunch& g) {
  if (g.n_frames != 1 || g.prec != kFP32C || !g.one.few || g.tau > 0.0) return false;
  const PointSizes n(g);
  return n.charges <= kPointCharges && n.units <= kPointUnits && n.results <= kPointResults;
}

cudaError_t launch_grid_point(const GridLaunch& g, cudaStream_t s) {
  const PointSizes n(g);
  const size_t smem = size_t(n.charges) * sizeof(float4) + size_t(n.results) * sizeof(double) +
                      size_t(n.units) * (g.kind == kField ? 3 : 1) * sizeof(float);
  // the limit belongs to the kernel, not to the calling thread: always the largest size,
  // so that a thread cannot lower it between another's setting and its launch
  constexpr int kMost = kPointCharges * sizeof(float4) + kPointResults * sizeof(double) +
                        kPointUnits * 3 * sizeof(float);
  auto run = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
    if (e != cudaSuccess) return e;
    kernel<<<kPointCtas, kPointThreads, smem, s>>>(g.one, g.points, g.x, g.q, g.out);
    return cudaGetLastError();
  };
  if (g.kind != kField) return run(grid_point_kernel<kEsp, false>);
  return g.clamp ? run(grid_point_kernel<kField, true>) : run(grid_point_kernel<kField, false>);
}

size_t grid_slot_doubles(int kind, int ppt) { return size_t(kGridThreads) * ppt * (kind == kField ? 3 : 1); }

size_t grid_zero_ints(int n_frames, bool refine) {
  return size_t((4 * n_frames + 1 + 3) & ~3) + (refine ? size_t(n_frames) * kMagBins : 0);
}

cudaError_t launch_grid(const GridLaunch& g, cudaStream_t s, bool cleared) {
  if (g.n_items <= 0) return cudaSuccess;
  if (!cleared && (g.n_prep > 0 || g.tau > 0.0)) {
    const cudaError_t e =
        cudaMemsetAsync(g.zeroed, 0, grid_zero_ints(g.n_frames, g.tau > 0.0) * sizeof(int), s);
    if (e != cudaSuccess) return e;
  }
  return with_form(g.prec, g.kind, g.ppt, [&](auto p, auto k, auto t) {
    return launch_grid_k<decltype(p)::value, decltype(k)::value, decltype(t)::value>(g, s);
  });
}

cudaError_t preload_grid_kernels(int prec, int kind, int clamp, int ppt) {
  return with_form(prec, kind, ppt, [&](auto p, auto k, auto t) {
    constexpr int P = decltype(p)::value, K = decltype(k)::value, T = decltype(t)::value;
    if constexpr (K == kField)
      if (clamp) return preload_c<P, K, true, T>();
    return preload_c<P, K, false, T>();
  });
}

cudaError_t preload_grid_kernels() {
  cudaError_t e = cudaSuccess;
  for (int prec : {int(kFP64), int(kFP32C)})
    for (int ppt : {4, 8})
      for (int form = 0; form < 3 && e == cudaSuccess; ++form)
        e = preload_grid_kernels(prec, form < 2 ? kField : kEsp, form == 1, ppt);
  return e;
}

cudaError_t launch_pack_f64(int64_t n, int64_t n_pad, const double* x, const double* q, void* packed,
                            cudaStream_t s) {
  if (n_pad <= 0) return cudaSuccess;
  const int blocks = static_cast<int>(std::min<int64_t>((n_pad + 255) / 256, 4096));
  pack_f64_kernel<<<blocks, 256, 0, s>>>(n, n_pad, x, q, static_cast<Charge64*>(packed));
  return cudaGetLastError();
}

}  // namespace cpetgb
