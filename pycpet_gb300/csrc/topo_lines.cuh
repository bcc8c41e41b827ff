// topo_lines.cuh -- device code shared by the streamline kernels (topo.cu: the
// persistent kernel and the serving engine; topo_team.cu: few lines per SM).
// One definition of the pair terms, the Kahan runs, the lane reduction and the
// per-line phase machine, so a line's result is the same bits whichever kernel
// steps it.
#pragma once
#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace cpetgb {
namespace {

constexpr int kLanePairs = 32;                  // charge pairs per lane between Kahan steps
constexpr int kChargePad32 = 64;                // FP32C frames: one charge pair per lane
constexpr int kChargePad64 = 256;               // FP64 frames
constexpr int kLaneRun64 = 16;                  // FP64: sources per lane and run

enum Phase : int { kMain = 0, kStart1 = 1, kStart2 = 2, kEnd1 = 3, kEnd2 = 4 };

struct SlotRec {      // per-slot record in shared memory (owner lane only)
  double x0[3], xip[3], xipp[3], xend[3], xe1[3];
};

__device__ __forceinline__ bool outside(const double p[3], const double h[3]) {
  return p[0] < -h[0] || p[0] > h[0] || p[1] < -h[1] || p[1] > h[1] || p[2] < -h[2] ||
         p[2] > h[2];
}

// Exact strict box test from the FP32 image pf = RN(p) of an FP64 position:
// RN is monotonic, so |pf| > RN(h) implies |p| > h and |pf| < RN(h) implies
// |p| < h; only a tie needs the FP64 comparison.
__device__ __forceinline__ bool outside_fast(const double p[3], const float pf[3],
                                             const double h[3], const float hf[3]) {
  bool out = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float a = fabsf(pf[k]);
    if (a > hf[k] || (a == hf[k] && fabs(p[k]) > h[k])) out = true;
  }
  return out;
}

__device__ __forceinline__ double curve_f64(const double a[3], const double b[3]) {
  const double c0 = a[1] * b[2] - a[2] * b[1];
  const double c1 = a[2] * b[0] - a[0] * b[2];
  const double c2 = a[0] * b[1] - a[1] * b[0];
  const double nc = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
  const double na = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
  return nc / (na * na * na);
}

// The frame a CTA is working on (uniform across the CTA).
struct FrameCtx {
  int64_t line_off;
  int n_lines;
  double step;
  double half[3];
  float hf[3];  // RN(half): the FP32 side of the exact box test
};

// Per-lane slot state (meaningful in lanes 0..S-1 only).
struct Slot {
  int line;     // -1 = idle
  int phase;
  int steps;
  int cap;
  double pos[3];  // where the next field evaluation happens
  float posf[3];  // its FP32 image (FP32C pair terms)
};

__device__ __forceinline__ void set_pos(Slot& sl, const double v[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    sl.pos[k] = v[k];
    sl.posf[k] = static_cast<float>(v[k]);
  }
}

__device__ void slot_load(Slot& sl, SlotRec& rec, int line, const TopoParams& p) {
  sl.line = line;
  if (line < 0) return;
  const double* s = p.starts + 3 * static_cast<int64_t>(line);
  double st[3];
  for (int k = 0; k < 3; ++k) rec.x0[k] = st[k] = s[k];
  set_pos(sl, st);
  sl.cap = max(p.n_iter[line], 0);
  if (sl.cap > kMaxLineCap) {  // refuse rather than run for hours
    atomicCAS(p.status, kDevOk, kDevBadCap);
    sl.cap = 0;
  }
  sl.steps = 0;
  if (sl.cap > 0) {
    sl.phase = kMain;
  } else {  // no loop step: the end point is the start point
    sl.phase = kStart1;
    for (int k = 0; k < 3; ++k) rec.xend[k] = s[k];
  }
}

// Results of a finished line: start-to-end distance and the mean of the
// curvatures at the start (x0, xip, xipp) and at the end (xend, xe1, xe2).
__device__ __forceinline__ void finish_line(const double x0[3], const double xip[3], const double xipp[3],
                                            const double xend[3], const double xe1[3], const double xe2[3],
                                            int line, int steps, const TopoParams& p) {
  double v1[3], v2[3], w1[3], w2[3], dd = 0.0;
  for (int k = 0; k < 3; ++k) {
    v1[k] = xip[k] - x0[k];
    v2[k] = xipp[k] - 2.0 * xip[k] + x0[k];
    w1[k] = xe1[k] - xend[k];
    w2[k] = xe2[k] - 2.0 * xe1[k] + xend[k];
    const double d = x0[k] - xend[k];
    dd += d * d;
  }
  const int64_t li = line;
  p.result[2 * li + 0] = sqrt(dd);
  p.result[2 * li + 1] = 0.5 * (curve_f64(v1, v2) + curve_f64(w1, w2));
  if (p.ends)
    for (int k = 0; k < 3; ++k) p.ends[3 * li + k] = xend[k];
  if (p.steps) p.steps[li] = steps;
}

// Advance one slot given the new position `nx` (= pos + step vector).
// Returns true when the line has finished (result written).
template <bool FAST_BOX>
__device__ bool slot_advance(Slot& sl, SlotRec& rec, const double nx[3], const TopoParams& p,
                             const FrameCtx& fc) {
  switch (sl.phase) {
    case kMain: {
      sl.steps += 1;
      if (sl.steps == 1)
        for (int k = 0; k < 3; ++k) rec.xip[k] = nx[k];
      if (sl.steps == 2)
        for (int k = 0; k < 3; ++k) rec.xipp[k] = nx[k];
      set_pos(sl, nx);
      const bool out =
          FAST_BOX ? outside_fast(sl.pos, sl.posf, fc.half, fc.hf) : outside(nx, fc.half);
      if (out || sl.steps >= sl.cap) {
        for (int k = 0; k < 3; ++k) rec.xend[k] = nx[k];
        if (sl.steps >= 2) {
          sl.phase = kEnd1;  // next evaluation at the end point (= nx)
        } else {
          sl.phase = kStart2;  // steps == 1: the end point is also x_init_plus
        }
      }
      return false;
    }
    case kStart1:
      for (int k = 0; k < 3; ++k) rec.xip[k] = nx[k];
      set_pos(sl, nx);
      sl.phase = kStart2;
      return false;
    case kStart2:
      for (int k = 0; k < 3; ++k) rec.xipp[k] = nx[k];
      set_pos(sl, rec.xend);
      sl.phase = kEnd1;
      return false;
    case kEnd1:
      for (int k = 0; k < 3; ++k) rec.xe1[k] = nx[k];
      set_pos(sl, nx);
      sl.phase = kEnd2;
      return false;
    default:  // kEnd2: nx is the second step after the end point
      finish_line(rec.x0, rec.xip, rec.xipp, rec.xend, rec.xe1, nx, sl.line, sl.steps, p);
      return true;
  }
}

// ---------------------------------------------------------------------------
// Field sweep over the charges for NA active slots.
// ---------------------------------------------------------------------------

// FP32C.  Charges in "pair" layout: A[p] = {x_2p, x_2p+1, y_2p, y_2p+1},
// B[p] = {z_2p, z_2p+1, q_2p, q_2p+1}, so each 64-bit half of a 16-byte load is
// a ready operand of the packed f32x2 instructions: one instruction evaluates
// a pair term for two charges.  Lanes take pairs lane-strided; every
// kLanePairs pairs (fewer in a frame's last run: frames are padded to one pair
// per lane only) the two packed streams are added and Kahan-accumulated.
//
// One charge pair against NA positions, up to the reciprocal square roots for
// all positions first (the MUFU results are then used as late as possible): 415
// ms per 100,000 lines over 8,000 charges, 421 with one position after the other.
template <int NA>
__device__ __forceinline__ void pair_terms(const ulonglong2& a, const ulonglong2& b,
                                           const uint64_t (&ex2)[NA][3], uint64_t (&part)[NA][3]) {
  uint64_t dx[NA], dy[NA], dz[NA], r[NA];
#pragma unroll
  for (int e = 0; e < NA; ++e) {
    dz[e] = sub2(ex2[e][2], b.x);
    dy[e] = sub2(ex2[e][1], a.y);
    dx[e] = sub2(ex2[e][0], a.x);
  }
#pragma unroll
  for (int e = 0; e < NA; ++e) r[e] = mul2(dz[e], dz[e]);
#pragma unroll
  for (int e = 0; e < NA; ++e) r[e] = fma2(dy[e], dy[e], r[e]);
#pragma unroll
  for (int e = 0; e < NA; ++e) r[e] = fma2(dx[e], dx[e], r[e]);
#pragma unroll
  for (int e = 0; e < NA; ++e) r[e] = rsqrt2(r[e]);
#pragma unroll
  for (int e = 0; e < NA; ++e) {
    const uint64_t w = mul2(mul2(b.y, r[e]), mul2(r[e], r[e]));
    part[e][0] = fma2(w, dx[e], part[e][0]);
    part[e][1] = fma2(w, dy[e], part[e][1]);
    part[e][2] = fma2(w, dz[e], part[e][2]);
  }
}

// Dipole pairs: A[p] = {x pair, y pair}, B[p] = {z pair, 3 mu_x pair},
// C[p] = {mu_y pair, mu_z pair}.  Per dipole the term of
// calc_field_base_dipole (CPET/utils/math_module.c:335-371) without the
// constant factor (the step only uses the field's direction):
//   r^-5 ((3 mu_x R_x + mu_y R_y + mu_z R_z) R_c - mu_c r^2)
//   = w R_c - r^-3 mu_c,  w = (3 mu_x R_x + mu_y R_y + mu_z R_z) r^-5,
// the x component taking mu_x as (3 mu_x) * (-1/3) r^-3.
template <int NA>
__device__ __forceinline__ void dipole_terms(const ulonglong2& a, const ulonglong2& b, const ulonglong2& c,
                                             const uint64_t (&ex2)[NA][3], uint64_t (&part)[NA][3]) {
  const uint64_t m_third = pk2(-1.f / 3.f, -1.f / 3.f), m_one = pk2(-1.f, -1.f);
#pragma unroll
  for (int e = 0; e < NA; ++e) {
    const uint64_t dx = sub2(ex2[e][0], a.x);
    const uint64_t dy = sub2(ex2[e][1], a.y);
    const uint64_t dz = sub2(ex2[e][2], b.x);
    const uint64_t r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    const uint64_t ri = rsqrt2(r2);
    const uint64_t ri2 = mul2(ri, ri);
    const uint64_t ri3 = mul2(ri2, ri);
    const uint64_t w = mul2(fma2(b.y, dx, fma2(c.x, dy, mul2(c.y, dz))), mul2(ri3, ri2));
    const uint64_t t3 = mul2(ri3, m_third), tn = mul2(ri3, m_one);
    part[e][0] = fma2(t3, b.y, fma2(w, dx, part[e][0]));
    part[e][1] = fma2(tn, c.x, fma2(w, dy, part[e][1]));
    part[e][2] = fma2(tn, c.y, fma2(w, dz, part[e][2]));
  }
}

// One Kahan run of one lane: cnt pairs from index `at` on, 32 apart, added to
// part[].  A, B, C: the frame's blocks in one address space (C: dipoles only).
template <int NA, bool DIP, int kFull, int kRest>
__device__ __forceinline__ void lane_run(const ulonglong2* A, const ulonglong2* B, const ulonglong2* C,
                                         int at, int cnt, const uint64_t (&ex2)[NA][3],
                                         uint64_t (&part)[NA][3]) {
  if (cnt == kLanePairs) {
#pragma unroll kFull
    for (int i = 0; i < kLanePairs; ++i) {
      const int k = at + 32 * i;
      if constexpr (DIP)
        dipole_terms<NA>(A[k], B[k], C[k], ex2, part);
      else
        pair_terms<NA>(A[k], B[k], ex2, part);
    }
  } else {
#pragma unroll kRest
    for (int i = 0; i < cnt; ++i) {
      const int k = at + 32 * i;
      if constexpr (DIP)
        dipole_terms<NA>(A[k], B[k], C[k], ex2, part);
      else
        pair_terms<NA>(A[k], B[k], ex2, part);
    }
  }
}

// lane_run for few lines per warp, where a run's latency counts: blocks of kBlk
// pairs, evaluated stage by stage over the whole block (a pair's eight dependent
// stages take about 100 cycles, one pair after the other 3,200 per run; the
// blocks 1,260 at NA = 1 and 2,300 at NA = 2, one warp alone).  The last block
// is filled up with zero charges (they add exactly 0) at the run's last pair.
template <int NA, bool DIP>
__device__ __forceinline__ void lane_run_blocks(const ulonglong2* A, const ulonglong2* B,
                                                const ulonglong2* C, int at, int cnt,
                                                const uint64_t (&ex2)[NA][3], uint64_t (&part)[NA][3]) {
  constexpr int kBlk = DIP ? (NA == 1 ? 8 : 4) : 16 / NA;
  auto block = [&](int i, auto full) {
    ulonglong2 a[kBlk], b[kBlk];
    [[maybe_unused]] ulonglong2 c[kBlk];
#pragma unroll
    for (int u = 0; u < kBlk; ++u) {
      const bool in = decltype(full)::value || i + u < cnt;
      const int k = at + 32 * (in ? i + u : cnt - 1);
      a[u] = A[k];
      b[u] = B[k];
      if (!in) b[u].y = 0ull;
      if constexpr (DIP) {
        c[u] = C[k];
        if (!in) c[u] = make_ulonglong2(0ull, 0ull);
      }
    }
    if constexpr (DIP) {
#pragma unroll
      for (int u = 0; u < kBlk; ++u) dipole_terms<NA>(a[u], b[u], c[u], ex2, part);
    } else {
      constexpr int M = kBlk * NA;
      uint64_t dx[M], dy[M], dz[M], r[M];
#pragma unroll
      for (int m = 0; m < M; ++m) {
        dz[m] = sub2(ex2[m % NA][2], b[m / NA].x);
        dy[m] = sub2(ex2[m % NA][1], a[m / NA].y);
        dx[m] = sub2(ex2[m % NA][0], a[m / NA].x);
      }
#pragma unroll
      for (int m = 0; m < M; ++m) r[m] = fma2(dx[m], dx[m], fma2(dy[m], dy[m], mul2(dz[m], dz[m])));
#pragma unroll
      for (int m = 0; m < M; ++m) r[m] = rsqrt2(r[m]);
#pragma unroll
      for (int m = 0; m < M; ++m) r[m] = mul2(mul2(b[m / NA].y, r[m]), mul2(r[m], r[m]));
#pragma unroll
      for (int m = 0; m < M; ++m) {
        part[m % NA][0] = fma2(r[m], dx[m], part[m % NA][0]);
        part[m % NA][1] = fma2(r[m], dy[m], part[m % NA][1]);
        part[m % NA][2] = fma2(r[m], dz[m], part[m % NA][2]);
      }
    }
  };
  int i = 0;
#pragma unroll 1
  for (; i + kBlk <= cnt; i += kBlk) block(i, std::true_type{});
  if (i < cnt) block(i, std::false_type{});
}

// Lane partials (acc - cmp, unevaluated pairs) as NV = 4S values v = 3e + c,
// reduced across the warp by a reduce-scatter of error-free pair additions:
// each of the LV levels halves the values a lane keeps, a butterfly finishes;
// afterwards the lanes with (lane >> (5 - LV)) == v hold the total of value v.
// Every value goes through the same tree (lanes 16, 8, 4, 2, 1 apart) and the
// pair addition is symmetric, so a total does not depend on S or on the other
// values.
template <int NA, int S>
__device__ __forceinline__ void reduce_lanes(const float (&acc)[NA][3], const float (&cmp)[NA][3],
                                             int lane, float& total) {
  constexpr int NV = 4 * S;
  constexpr int LV = (S == 4) ? 4 : (S == 2 ? 3 : 2);
  float h[NV], l[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int e = v / 3, c = v % 3;
    h[v] = (e < NA) ? acc[e < NA ? e : 0][c] : 0.f;
    l[v] = (e < NA) ? -cmp[e < NA ? e : 0][c] : 0.f;
  }
#pragma unroll
  for (int lvl = 0, half = NV / 2; lvl < LV; ++lvl, half >>= 1) {
    const int off = 16 >> lvl;
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const float sh = upper ? h[j] : h[j + half];
      const float sl = upper ? l[j] : l[j + half];
      const float kh = upper ? h[j + half] : h[j];
      const float kl = upper ? l[j + half] : l[j];
      const float rh = __shfl_xor_sync(0xffffffffu, sh, off);
      const float rl = __shfl_xor_sync(0xffffffffu, sl, off);
      h[j] = kh;
      l[j] = kl;
      pair_add(h[j], l[j], rh, rl);
    }
  }
#pragma unroll
  for (int off = 16 >> LV; off >= 1; off >>= 1) {
    const float rh = __shfl_xor_sync(0xffffffffu, h[0], off);
    const float rl = __shfl_xor_sync(0xffffffffu, l[0], off);
    pair_add(h[0], l[0], rh, rl);
  }
  total = h[0];
}

// Positions of NA slots (the FP32 images), passed by value.
template <int NA>
struct Points {
  float v[NA][3];
};

// Where a sweep's pairs lie: kSrcShared -- all in the CTA's dynamic shared
// memory; kSrcGlobal -- all in global memory (L2); kSrcSplit -- pairs [0,
// res_pairs) in shared memory, the rest in global memory; res_pairs is a multiple of the 32 x kLanePairs pairs of one Kahan run,
// so every run reads one source and the sums do not depend on the split.
constexpr int kSrcShared = 0;
constexpr int kSrcSplit = 1;
constexpr int kSrcGlobal = 2;

// Field of a whole frame at NA positions, over the 32 lanes of a warp; returns
// reduce_lanes' total for S = 1, 2, 4, 4 slots.  sm_off: byte offset of the
// shared copy (its blocks of res_pairs pairs, one after the other); g: the
// frame in global memory (blocks of n_pairs pairs).
template <int NA, bool DIP, int SRC, int kFull, int kRest>
__device__ __forceinline__ float sweep_frame(const Points<NA>& at, uint32_t sm_off, int res_pairs,
                                             const ulonglong2* __restrict__ g, int n_pairs) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const ulonglong2* s = reinterpret_cast<const ulonglong2*>(smem_raw + sm_off);
  const int lane = threadIdx.x & 31;
  uint64_t ex2[NA][3];
  float acc[NA][3], cmp[NA][3];
#pragma unroll
  for (int e = 0; e < NA; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ex2[e][c] = pk2(at.v[e][c], at.v[e][c]);
      acc[e][c] = cmp[e][c] = 0.f;
    }
  // n_pairs is a multiple of 32: every lane runs the same number of pairs
  for (int base = 0; base < n_pairs; base += 32 * kLanePairs) {
    uint64_t part[NA][3];
#pragma unroll
    for (int e = 0; e < NA; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) part[e][c] = 0ull;
    const int cnt = min(kLanePairs, (n_pairs - base) >> 5);
    if (SRC == kSrcShared || (SRC == kSrcSplit && base < res_pairs))
      lane_run<NA, DIP, kFull, kRest>(s, s + res_pairs, s + 2 * res_pairs, base + lane, cnt, ex2, part);
    else
      lane_run<NA, DIP, kFull, kRest>(g, g + n_pairs, g + 2 * n_pairs, base + lane, cnt, ex2, part);
#pragma unroll
    for (int e = 0; e < NA; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float lo, hi;
        upk2(part[e][c], lo, hi);
        kahan_add(acc[e][c], cmp[e][c], __fadd_rn(lo, hi));
      }
  }
  float total;
  reduce_lanes<NA, (NA == 3 ? 4 : NA)>(acc, cmp, lane, total);
  return total;
}

// The sweep of a frame held in shared memory, a function of its own, not inlined:
// its schedule then does not change with the step loop around it (inlined
// there, the same loop ran 415 to 453 ms per 100,000 lines over 8,000 charges
// depending on code outside it), and the call costs a few of a sweep's 20,000 to
// 50,000 cycles.  Unroll of the full runs: 2 pairs 441 ms, 4 418, 8 415, 16 428.
// Sweeps that read global memory are inlined: the function's loads are issued
// too late to hide the L2's latency (serving engine 50% slower).
template <int NA, bool DIP>
__device__ __noinline__ float sweep_shared(Points<NA> at, uint32_t sm_off, const ulonglong2* __restrict__ g,
                                           int n_pairs) {
  constexpr int kFull = DIP ? (NA >= 3 ? 2 : (NA == 2 ? 4 : 8)) : (NA == 1 ? 16 : 8);
  constexpr int kRest = DIP ? (NA >= 2 ? 1 : 4) : (NA == 1 ? 8 : 2);
  return sweep_frame<NA, DIP, kSrcShared, kFull, kRest>(at, sm_off, n_pairs, g, n_pairs);
}

// The sweep for the `na` active slots among S (lanes 0 .. S-1 hold their FP32
// positions posf, src_of their owner lanes); the calling slot's field (rank rk)
// in E.
template <int S, bool DIP, int SRC>
__device__ __forceinline__ void sweep_slots(int na, const float (&posf)[3], const int (&src_of)[S], int rk,
                                            uint32_t sm_off, int res_pairs, const ulonglong2* g,
                                            int n_pairs, float (&E)[3]) {
  Points<S> at;
#pragma unroll
  for (int e = 0; e < S; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) at.v[e][c] = __shfl_sync(0xffffffffu, posf[c], src_of[e]);
  float total = 0.f;
  auto sweep = [&](auto n) {
    constexpr int NA = decltype(n)::value;
    Points<NA> pt;
#pragma unroll
    for (int e = 0; e < NA; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) pt.v[e][c] = at.v[e][c];
    if constexpr (SRC == kSrcShared) {
      total = sweep_shared<NA, DIP>(pt, sm_off, g, n_pairs);
    } else {
      // about eight independent pair chains in flight per lane: unroll 8 / NA; twice
      // that for four lines on global memory alone (the serving engine, 48,000
      // lines of 8,000 and 20,000 charges: 0.750 s against 0.785, two CTAs per SM
      // 0.54 against 0.58; from shared and global memory both run alike)
      constexpr int kFull = NA == 4 && SRC == kSrcGlobal ? 4 : (NA >= 3 ? 2 : (NA == 2 ? 4 : 8));
      total = sweep_frame<NA, DIP, SRC, kFull, 1>(pt, sm_off, res_pairs, g, n_pairs);
    }
  };
  switch (na) {
    case 1: sweep(std::integral_constant<int, 1>{}); break;
    case 2: sweep(std::integral_constant<int, 2>{}); break;
    case 3: sweep(std::integral_constant<int, (S > 2 ? 3 : 2)>{}); break;
    default: sweep(std::integral_constant<int, S>{}); break;
  }
  // component c of slot rank e sits in lanes (3e + c) << (5 - LV) and up
  const int shift = na == 1 ? 3 : (na == 2 ? 2 : 1);
#pragma unroll
  for (int c = 0; c < 3; ++c) E[c] = __shfl_sync(0xffffffffu, total, (3 * rk + c) << shift);
}

// FP64.  Bound: the FP64 pipe (64 cycles per warp instruction); a charge pair
// takes 12 of its instructions (3 differences, 3 for r^2, 3 for q r^-3 with
// common.cuh's seed, 3 sums) where rsqrt() and three products took 19.  A run
// is kLaneRun64 charges per lane, summed plainly; the runs are added in order.
template <int NA, int S>
__device__ __forceinline__ void run_f64(const Charge64* __restrict__ g, int base, int cnt,
                                        const double (&ex)[S][3], double (&part)[NA][3]) {
#pragma unroll 2
  for (int i = 0; i < cnt; ++i) {
    const Charge64 ch = g[base + 32 * i];
#pragma unroll
    for (int e = 0; e < NA; ++e) {
      const double dx = __dsub_rn(ex[e][0], ch.x);
      const double dy = __dsub_rn(ex[e][1], ch.y);
      const double dz = __dsub_rn(ex[e][2], ch.z);
      const double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
      const double w = weight_r3_f64(ch.q, r2);
      part[e][0] = __fma_rn(w, dx, part[e][0]);
      part[e][1] = __fma_rn(w, dy, part[e][1]);
      part[e][2] = __fma_rn(w, dz, part[e][2]);
    }
  }
}

// FP64 dipoles: the term of dipole_terms, r^-5 dot R - r^-3 mu (21 FP64-pipe
// instructions, 29 with rsqrt()).
template <int NA, int S>
__device__ __forceinline__ void run_f64(const Dipole64* __restrict__ g, int base, int cnt,
                                        const double (&ex)[S][3], double (&part)[NA][3]) {
#pragma unroll 2
  for (int i = 0; i < cnt; ++i) {
    const Dipole64 d = g[base + 32 * i];
#pragma unroll
    for (int e = 0; e < NA; ++e) {
      const double dx = __dsub_rn(ex[e][0], d.x);
      const double dy = __dsub_rn(ex[e][1], d.y);
      const double dz = __dsub_rn(ex[e][2], d.z);
      const double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
      double r3, r5;
      inv_r3_r5_f64(r2, r3, r5);
      const double dot = __fma_rn(3.0 * d.mx, dx, __fma_rn(d.my, dy, __dmul_rn(d.mz, dz)));
      const double w = __dmul_rn(r5, dot);
      part[e][0] = __fma_rn(w, dx, __fma_rn(-r3, d.mx, part[e][0]));
      part[e][1] = __fma_rn(w, dy, __fma_rn(-r3, d.my, part[e][1]));
      part[e][2] = __fma_rn(w, dz, __fma_rn(-r3, d.mz, part[e][2]));
    }
  }
}

// Lane sums of one component added across the warp (lanes 16, 8, 4, 2, 1 apart).
__device__ __forceinline__ double reduce_lanes_f64(double v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// A whole frame: sources from global memory (padded with zero charges or
// moments far away), run by run.
template <int NA, int S, typename Src>
__device__ __forceinline__ void sweep_f64(const Src* __restrict__ g, int n_pad, int lane,
                                          const double (&ex)[S][3], double (&E)[S][3]) {
  double acc[NA][3];
#pragma unroll
  for (int e = 0; e < NA; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[e][c] = 0.0;
  for (int j = 0; j < n_pad; j += 32 * kLaneRun64) {
    double part[NA][3];
#pragma unroll
    for (int e = 0; e < NA; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) part[e][c] = 0.0;
    run_f64<NA, S>(g, j + lane, min(kLaneRun64, (n_pad - j) >> 5), ex, part);
#pragma unroll
    for (int e = 0; e < NA; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[e][c] = __dadd_rn(acc[e][c], part[e][c]);
  }
#pragma unroll
  for (int e = 0; e < NA; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) E[e][c] = reduce_lanes_f64(acc[e][c]);
}

// One component (Ec) of the Euler step vector h E / |E|.  FP32C: formed in FP32
// (the factor k does not change the direction), then added to the FP64 position.
__device__ __forceinline__ double euler_vec(const float (&E)[3], float Ec, double step) {
  const float n2 = __fmaf_rn(E[0], E[0], __fmaf_rn(E[1], E[1], __fmul_rn(E[2], E[2])));
  return static_cast<double>(__fmul_rn(Ec, __fdiv_rn(static_cast<float>(step), __fsqrt_rn(n2))));
}
__device__ __forceinline__ double euler_vec(const double (&E)[3], double Ec, double step) {
  return __ddiv_rn(__dmul_rn(step, Ec),
                   __dsqrt_rn(__fma_rn(E[2], E[2], __fma_rn(E[1], E[1], __dmul_rn(E[0], E[0])))));
}
template <typename Real>
__device__ __forceinline__ void euler_step(const Real (&E)[3], const double (&pos)[3], double step,
                                           double (&nx)[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) nx[c] = __dadd_rn(pos[c], euler_vec(E, E[c], step));
}

}  // namespace
}  // namespace cpetgb
