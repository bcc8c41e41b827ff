// topo_team.cu -- streamlines stepped by teams of warps: launches of few lines,
// and the last lines of larger ones.
//
// The persistent kernel (topo.cu) gives a line to one warp, which sweeps all of
// the frame's charges for every step.  That fills the GPU as long as there are
// several lines per warp; with fewer, a step lasts as long as one warp needs
// for the whole frame while other warps idle.  Here a team of kTeamWarps warps
// steps up to kTeamLines lines together:
//   A  the Kahan runs of all its lines are dealt out to its warps: a unit is one
//      run of one or two lines, its lane sums go to shared memory;
//   B  warp k owns line k: it adds the line's runs in order (the same Kahan
//      sequence per lane as one warp sweeping the whole frame), reduces them
//      across the lanes and makes the step, one component per lane (an FP64
//      instruction costs a warp the same whether one lane is active or three,
//      and GB300's FP64 pipe is slow).
// The sums, their order and the lane tree are those of the persistent kernel
// and the engine, so a line's result is the same bits.  Two teams per CTA share
// the frame's charges in shared memory; one computes while the other is in its
// serial phase.
//
// The kernel runs in rounds of a limited number of steps (topo_team_rounds): at
// the end of a round the running lines go to a list, from which the next
// round's launch deals them evenly over the SMs again.  Lines end at very
// different times; without this the SMs whose lines are short idle while
// others still step several.
//
// Bound: FP32 pipe while lines x runs fill the warps, then the latency of one
// run (32 dependent pair steps per lane) plus phase B and its two barriers.
#include <algorithm>
#include <climits>
#include <cmath>

#include "topo_lines.cuh"

namespace cpetgb {
namespace {

constexpr int kTeams = 2;                          // per CTA
constexpr int kTeamWarps = 8;                      // warps per team
constexpr int kTeamThreads = kTeamWarps * 32;
constexpr int kTeamLines = kTeamLinesPerSm / kTeams;  // lines per team: one per warp in phase B
constexpr int kTeamUnits = 32;                     // (line, run) sums a team exchanges at a time
// Rounds: at most kTeamRounds launches, each stepping a kTeamRounds-th of the box
// diagonal (a line is 0.28 diagonals long on average, the longest of some thousand
// 0.75), but at least kTeamMinSteps steps: a round costs about 10 us (launch, charges to
// shared memory; 3 us once no line is left), a step 1 to 3 us, in FP64 10 and more.
// 12 rounds against 20 (ms): FP64 1,000 lines x 4,000 charges 82.9 and 77.0, 5,000 lines x
// 8,000 dipoles 48.7 and 47.7, 1,000 lines x 8,000 charges 9.95 and 10.0.
constexpr int kTeamRounds = 20;
constexpr int kTeamMinSteps = 128;
static_assert(kTeamLines <= kTeamWarps, "phase B gives each line a warp");

template <int PREC>
struct TeamReal {
  using T = float;
};
template <>
struct TeamReal<kFP64> {
  using T = double;
};

template <int PREC>
struct TeamShared {
  typename TeamReal<PREC>::T at[kTeamLines][3];  // where each line is evaluated next
  unsigned alive;                                // lines still running
};

// Slot of the k-th line still running, and (*next) of the one after it.
__device__ __forceinline__ int team_slot(unsigned alive, int k, int* next) {
  for (; k > 0; --k) alive &= alive - 1;
  *next = __ffs(alive & (alive - 1)) - 1;
  return __ffs(alive) - 1;
}

// u / d for u < 40, 1 <= d <= 8 (a division would cost a step 100 cycles).
__device__ __forceinline__ int small_div(int u, int d) {
  constexpr unsigned long long kInv = 0x20252b3440568000ull;  // byte d - 1: ceil(256 / d), d >= 2
  return d == 1 ? u : static_cast<int>((u * static_cast<unsigned>((kInv >> (8 * (d - 1))) & 255u)) >> 8);
}

template <int PREC>
constexpr size_t team_unit_bytes() {
  return 3 * 32 * sizeof(typename TeamReal<PREC>::T);
}
template <int PREC>
constexpr size_t team_fixed_bytes() {  // everything but the sources
  return ((kTeams * sizeof(TeamShared<PREC>) + 127) / 128) * 128 + 128 +
         kTeams * kTeamUnits * team_unit_bytes<PREC>();
}

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeamThreads) : "memory");
}

// One run of NA lines, FP32C: lane sums of line e to out[e][c][lane].  A, B, C:
// the blocks in global memory, or (SMEM) at byte offset sm_off of the dynamic
// shared memory, res_pairs pairs each.
template <int NA, bool DIP, bool SMEM>
__device__ __forceinline__ void team_run(Points<NA> at, const ulonglong2* __restrict__ g, int pairs,
                                      uint32_t sm_off, int base, int cnt, float* out0, float* out1) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  uint64_t ex2[NA][3], part[NA][3];
#pragma unroll
  for (int e = 0; e < NA; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ex2[e][c] = pk2(at.v[e][c], at.v[e][c]);
      part[e][c] = 0ull;
    }
  if constexpr (SMEM) {
    const ulonglong2* s = reinterpret_cast<const ulonglong2*>(smem_raw + sm_off);
    lane_run_blocks<NA, DIP>(s, s + pairs, s + 2 * pairs, base + lane, cnt, ex2, part);
  } else {
    lane_run_blocks<NA, DIP>(g, g + pairs, g + 2 * pairs, base + lane, cnt, ex2, part);
  }
#pragma unroll
  for (int e = 0; e < NA; ++e)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float lo, hi;
      upk2(part[e][c], lo, hi);
      (e == 0 ? out0 : out1)[32 * c + lane] = __fadd_rn(lo, hi);
    }
}

// The frame a CTA works on, in global and (a prefix of whole runs) shared memory.
struct TeamSource {
  const ulonglong2* g;
  uint32_t sm_off;  // byte offset of the shared copy
  int n_pairs;      // FP32C pairs, or FP64 sources
  int res_pairs;    // FP32C pairs in shared memory
};

// Phase A: the units of runs [r0, r0 + rb) of the K running lines.
template <bool DIP>
__device__ __forceinline__ void team_phase_a(const TeamSource& src, const TeamShared<kFP32C>& sh,
                                             unsigned alive, float* sums, int K, int r0, int rb,
                                             int per_line, int wid, int lane) {
  constexpr int kRun = 32 * kLanePairs;
  // Two lines per unit while that leaves at least a unit per warp: one line
  // alone reads 32 bytes of shared memory per lane and pair, more than the
  // SM's 128 bytes per clock serve at the FP32 pipe's rate.
  const int na = ((K + 1) / 2) * rb >= kTeamWarps ? 2 : 1;
  const int groups = na == 2 ? (K + 1) / 2 : K;
  for (int u = wid; u < rb * groups; u += kTeamWarps) {
    const int rr = small_div(u, groups);
    int g = u - rr * groups;
    // warps w and w + 4 share a scheduler: 2, 4 or 8 groups are rotated from run to
    // run, so that the short last group of an odd K moves over all four schedulers
    if ((groups & (groups - 1)) == 0) g = (g + ((rr * groups) >> 2)) & (groups - 1);
    const int k0 = g * na;
    const int base = (r0 + rr) * kRun;
    const int cnt = min(kLanePairs, (src.n_pairs - base) >> 5);
    const bool in_smem = base < src.res_pairs;
    float* out = sums + (k0 * per_line + rr) * 96;
    int s1;
    const int s0 = team_slot(alive, k0, &s1);
    if (na == 2 && k0 + 1 < K) {
      Points<2> at;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        at.v[0][c] = sh.at[s0][c];
        at.v[1][c] = sh.at[s1][c];
      }
      if (in_smem)
        team_run<2, DIP, true>(at, src.g, src.res_pairs, src.sm_off, base, cnt, out, out + per_line * 96);
      else
        team_run<2, DIP, false>(at, src.g, src.n_pairs, src.sm_off, base, cnt, out, out + per_line * 96);
    } else {
      Points<1> at;
#pragma unroll
      for (int c = 0; c < 3; ++c) at.v[0][c] = sh.at[s0][c];
      if (in_smem)
        team_run<1, DIP, true>(at, src.g, src.res_pairs, src.sm_off, base, cnt, out, out);
      else
        team_run<1, DIP, false>(at, src.g, src.n_pairs, src.sm_off, base, cnt, out, out);
    }
  }
}

template <bool DIP>
__device__ __forceinline__ void team_phase_a(const TeamSource& src, const TeamShared<kFP64>& sh,
                                             unsigned alive, double* sums, int K, int r0, int rb,
                                             int per_line, int wid, int lane) {
  constexpr int kRun = 32 * kLaneRun64;
  for (int u = wid; u < rb * K; u += kTeamWarps) {
    const int rr = small_div(u, K), k = u - rr * K;
    const int base = (r0 + rr) * kRun;
    int unused;
    const int s = team_slot(alive, k, &unused);
    const double ex[1][3] = {{sh.at[s][0], sh.at[s][1], sh.at[s][2]}};
    double part[1][3] = {{0.0, 0.0, 0.0}};
    const int cnt = min(kLaneRun64, (src.n_pairs - base) >> 5);
    if constexpr (DIP)
      run_f64<1, 1>(reinterpret_cast<const Dipole64*>(src.g), base + lane, cnt, ex, part);
    else
      run_f64<1, 1>(reinterpret_cast<const Charge64*>(src.g), base + lane, cnt, ex, part);
    double* out = sums + (k * per_line + rr) * 96;
#pragma unroll
    for (int c = 0; c < 3; ++c) out[32 * c + lane] = part[0][c];
  }
}

// A line owned by one warp: component c of its points in lane c (lanes 3 and
// up hold copies of component 0), the rest uniform across the warp.
struct TeamLine {
  double x0, xip, xipp, xend, xe1, pos;
  int line, phase, steps, cap;

  // As slot_load.
  __device__ __forceinline__ void load(int ln, int c, int lane, const TopoParams& p) {
    line = ln;
    x0 = p.starts[3 * static_cast<int64_t>(ln) + c];
    pos = x0;
    cap = max(p.n_iter[ln], 0);
    if (cap > kMaxLineCap) {
      if (lane == 0) atomicCAS(p.status, kDevOk, kDevBadCap);
      cap = 0;
    }
    steps = 0;
    phase = cap > 0 ? kMain : kStart1;
    xip = xipp = xe1 = 0.0;
    xend = x0;
  }
  __device__ __forceinline__ void load(const TopoState& t, int c) {
    x0 = t.x0[c];
    xip = t.xip[c];
    xipp = t.xipp[c];
    xend = t.xend[c];
    xe1 = t.xe1[c];
    pos = t.pos[c];
    line = t.line;
    phase = t.phase;
    steps = t.steps;
    cap = t.cap;
  }
  __device__ __forceinline__ void store(TopoState& t, int lane) const {
    if (lane < 3) {
      t.x0[lane] = x0;
      t.xip[lane] = xip;
      t.xipp[lane] = xipp;
      t.xend[lane] = xend;
      t.xe1[lane] = xe1;
      t.pos[lane] = pos;
    }
    if (lane == 0) {
      t.line = line;
      t.phase = phase;
      t.steps = steps;
      t.cap = cap;
    }
  }
  // Where the line is evaluated after a step to nx, whatever the box test says.
  __device__ __forceinline__ double next(double nx) const { return phase == kStart2 ? xend : nx; }
  __device__ __forceinline__ bool last() const { return phase == kEnd2; }
  // As slot_advance; nx is this lane's component of the new position, pos the
  // next one (already moved on), posf its FP32 image.
  template <bool FAST_BOX>
  __device__ __forceinline__ void advance(double nx, float posf, double half, float hf, int lane,
                                          const TopoParams& p) {
    if (phase == kMain) {
      steps += 1;
      if (steps == 1) xip = nx;
      if (steps == 2) xipp = nx;
      bool beyond;
      if (FAST_BOX) {
        const float a = fabsf(posf);
        beyond = a > hf || (a == hf && fabs(pos) > half);
      } else {
        beyond = nx < -half || nx > half;
      }
      const bool out = (__ballot_sync(0xffffffffu, beyond) & 7u) != 0;
      if (out || steps >= cap) {
        xend = nx;
        phase = steps >= 2 ? kEnd1 : kStart2;
      }
      return;
    }
    if (phase == kStart1) {
      xip = nx;
      phase = kStart2;
      return;
    }
    if (phase == kStart2) {
      xipp = nx;
      phase = kEnd1;
      return;
    }
    if (phase == kEnd1) {
      xe1 = nx;
      phase = kEnd2;
      return;
    }
    double a[6][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      a[0][c] = __shfl_sync(0xffffffffu, x0, c);
      a[1][c] = __shfl_sync(0xffffffffu, xip, c);
      a[2][c] = __shfl_sync(0xffffffffu, xipp, c);
      a[3][c] = __shfl_sync(0xffffffffu, xend, c);
      a[4][c] = __shfl_sync(0xffffffffu, xe1, c);
      a[5][c] = __shfl_sync(0xffffffffu, nx, c);
    }
    if (lane == 0) finish_line(a[0], a[1], a[2], a[3], a[4], a[5], line, steps, p);
  }
};

// Lines first, first + 1, ... (count of them, alternating between the teams) of
// a frame, run to their ends.
template <int PREC, bool DIP>
__device__ __forceinline__ void team_lines(const TopoParams& p, const TopoFrame& fr, const TeamSource& src,
                                           TeamShared<PREC>& sh, typename TeamReal<PREC>::T* sums,
                                           int first, int count, const TopoState* in_list, TopoState* out_list,
                                           int* left_out, int team, int wid, int lane) {
  using Real = typename TeamReal<PREC>::T;
  constexpr int kRun = PREC == kFP32C ? 32 * kLanePairs : 32 * kLaneRun64;
  const int runs = (src.n_pairs + kRun - 1) / kRun;
  const int c = lane < 3 ? lane : 0;
  const double half = fr.half[c];
  const float hf = static_cast<float>(half);
  TeamLine ln{};
  // steps of this launch: a share of the box diagonal, at least kTeamMinSteps; no
  // limit in the last round
  int budget = INT_MAX;
  if (left_out) {
    const double diag = 2.0 * sqrt(fr.half[0] * fr.half[0] + fr.half[1] * fr.half[1] + fr.half[2] * fr.half[2]);
    const double share = diag / fabs(fr.step) * (1.0 / kTeamRounds);
    budget = share < 1.0e9 ? max(static_cast<int>(share), kTeamMinSteps) : 1000000000;
  }
  {
    const int mine = (count - team + kTeams - 1) / kTeams;  // this team's lines, one per warp
    if (wid < mine) {
      const int j = first + wid * kTeams + team;
      if (in_list)
        ln.load(in_list[fr.left_off + j], c);
      else
        ln.load(static_cast<int>(fr.line_off + j), c, lane, p);
      if (lane < 3) sh.at[wid][lane] = static_cast<Real>(ln.pos);
    }
    if (wid == 0 && lane == 0) sh.alive = (1u << mine) - 1u;
  }
  team_sync(team);
  unsigned alive;
  for (;; --budget) {
    alive = sh.alive;
    if (alive == 0 || budget == 0) break;
    const int K = __popc(alive);
    const bool own = (alive >> wid) & 1u;
    const int rank = __popc(alive & ((1u << wid) - 1u));
    // units go to the warps without a line first: the owners are still at the
    // box test of the previous step
    const int turn = own ? kTeamWarps - K + rank : wid - rank;
    const int per_line = min(runs, kTeamUnits >> (32 - __clz(K - 1)));  // runs per exchange
    Real acc[1][3] = {{Real(0), Real(0), Real(0)}};
    [[maybe_unused]] float cmp[1][3] = {{0.f, 0.f, 0.f}};
    for (int r0 = 0; r0 < runs; r0 += per_line) {
      const int rb = min(per_line, runs - r0);
      team_phase_a<DIP>(src, sh, alive, sums, K, r0, rb, per_line, turn, lane);
      team_sync(team);
      if (own) {
        const Real* in = sums + rank * per_line * 96 + lane;
#pragma unroll 4
        for (int r = 0; r < rb; ++r) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const Real v = in[96 * r + 32 * k];
            if constexpr (PREC == kFP32C)
              kahan_add(acc[0][k], cmp[0][k], v);
            else
              acc[0][k] = __dadd_rn(acc[0][k], v);
          }
        }
      }
      if (r0 + per_line < runs) team_sync(team);  // the exchange is written again
    }
    double nx = 0.0;
    Real at = Real(0);
    if (own) {
      Real E[3];
      if constexpr (PREC == kFP32C) {
        float total;
        reduce_lanes<1, 1>(acc, cmp, lane, total);  // component k in lanes 8k .. 8k + 7
#pragma unroll
        for (int k = 0; k < 3; ++k) E[k] = __shfl_sync(0xffffffffu, total, 8 * k);
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) E[k] = reduce_lanes_f64(acc[0][k]);
      }
      const Real Ec = lane == 1 ? E[1] : (lane == 2 ? E[2] : E[0]);
      nx = __dadd_rn(ln.pos, euler_vec(E, Ec, fr.step));
      ln.pos = ln.next(nx);
      at = static_cast<Real>(ln.pos);
      if (lane < 3) sh.at[wid][lane] = at;
      if (ln.last() && lane == 0) atomicAnd(&sh.alive, ~(1u << wid));
    }
    team_sync(team);
    if (own) ln.template advance<PREC == kFP32C>(nx, static_cast<float>(at), half, hf, lane, p);
  }
  if (alive && ((alive >> wid) & 1u)) {  // the round is over: to the next round's list
    int k = 0;
    if (lane == 0) k = atomicAdd(left_out, 1);
    k = __shfl_sync(0xffffffffu, k, 0);
    ln.store(out_list[fr.left_off + k], lane);
  }
}

// Items are (frame, up to `chunk` lines); CTA b takes items b, b + gridDim.x, ...
// chunk is the smallest line count per item for which all items fit the waves of
// CTAs that kTeamLinesPerSm lines each would need, so the lines are spread evenly
// over the SMs.
template <int PREC, bool DIP>
__global__ void __launch_bounds__(kTeams* kTeamThreads, 1)
    team_kernel(TopoParams p, TopoFrame frame0, int fresh, int round) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_chunk, s_frame, s_first, s_count;
  using Real = typename TeamReal<PREC>::T;
  TeamShared<PREC>* teams = reinterpret_cast<TeamShared<PREC>*>(smem_raw);
  constexpr size_t kBarOff = ((kTeams * sizeof(TeamShared<PREC>) + 127) / 128) * 128;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + kBarOff);
  Real* sums = reinterpret_cast<Real*>(smem_raw + kBarOff + 128);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / kTeamWarps, wid = warp % kTeamWarps;
  const int n_frames = p.frames ? p.n_frames : 1;
  const int G = static_cast<int>(gridDim.x);
  // this launch's lines: the frames' tables, or the list of the launch before
  const bool from_list = !fresh || round > 0;
  const int n_round = fresh ? round - 1 : round;  // lists written before this launch, less one
  const TopoState* in_list = from_list ? p.left + (n_round & 1) * p.left_records : nullptr;
  const int* in_count = from_list ? p.left_count + n_round * n_frames : nullptr;
  const bool more = round + 1 < p.rounds;
  TopoState* out_list = more ? p.left + ((n_round + 1) & 1) * p.left_records : nullptr;
  int* out_count = more ? p.left_count + (n_round + 1) * n_frames : nullptr;
  auto count_of = [&](int f) {
    return from_list ? in_count[f] : (p.frames ? p.frames[f].n_lines : frame0.n_lines);
  };
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    long long total = 0;
    for (int f = lane; f < n_frames; f += 32) total += count_of(f);
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const long long wave = static_cast<long long>(G) * kTeamLinesPerSm;
    const long long slots = G * ((total + wave - 1) / wave);
    int chunk = total > 0 ? static_cast<int>((total + slots - 1) / slots) : 0;
    while (chunk > 0 && chunk < kTeamLinesPerSm) {
      long long items = 0;
      for (int f = lane; f < n_frames; f += 32) items += (count_of(f) + chunk - 1) / chunk;
      for (int o = 16; o > 0; o >>= 1) items += __shfl_xor_sync(0xffffffffu, items, o);
      if (items <= slots) break;
      ++chunk;
    }
    if (lane == 0) s_chunk = chunk;
  }
  __syncthreads();
  const int chunk = s_chunk;
  if (chunk == 0) return;
  int loaded = -1;
  uint32_t load_parity = 0;
  TopoFrame fr = frame0;
  TeamSource src{};
  for (long long item = blockIdx.x;; item += G) {
    if (warp == 0) {  // the item's frame and lines
      long long base = 0;
      int found = 0;
      for (int f0 = 0; f0 < n_frames && !found; f0 += 32) {
        const int n = f0 + lane < n_frames ? count_of(f0 + lane) : 0;
        const long long mine = (n + chunk - 1) / chunk;
        long long incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
          const long long v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, base + incl > item);
        if (hit) {
          if (lane == __ffs(hit) - 1) {
            const int first = static_cast<int>(item - (base + incl - mine)) * chunk;
            s_frame = f0 + lane;
            s_first = first;
            s_count = min(chunk, n - first);
          }
          found = 1;
        }
        base += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (!found && lane == 0) s_frame = -1;
    }
    __syncthreads();
    const int f = s_frame;
    if (f < 0) break;
    const int first = s_first, count = s_count;
    if (f != loaded) {  // (every team is done with the previous frame)
      if (p.frames) fr = p.frames[f];
      loaded = f;
      const size_t elem = PREC == kFP32C ? 16 : 32;
      src.g = reinterpret_cast<const ulonglong2*>(static_cast<const char*>(p.packed) + fr.packed_off * elem);
      src.n_pairs = fr.n_pad;
      if constexpr (PREC == kFP32C) {
        const int res = fr.team_resident;
        src.n_pairs = fr.n_pad / 2;
        src.res_pairs = res / 2;
        src.sm_off = static_cast<uint32_t>(team_fixed_bytes<PREC>());
        if (threadIdx.x == 0) {
          const uint32_t blk = static_cast<uint32_t>(res / 2) * 16u;  // bytes of one block's prefix
          constexpr int n_blk = DIP ? 3 : 2;
          mbar_arrive_expect_tx(bar, blk * n_blk);
          constexpr uint32_t kCopy = 32768;
          for (int b = 0; b < n_blk; ++b) {
            const char* bs = reinterpret_cast<const char*>(src.g) + static_cast<size_t>(b) * (fr.n_pad / 2) * 16;
            char* bd = reinterpret_cast<char*>(smem_raw) + src.sm_off + static_cast<size_t>(b) * blk;
            for (uint32_t off = 0; off < blk; off += kCopy)
              bulk_g2s(bd + off, bs + off, min(kCopy, blk - off), bar);
          }
        }
        const bool mine = mbar_wait(bar, load_parity, p.status);
        load_parity ^= 1u;
        if (!__syncthreads_and(mine)) return;
      }
    }
    team_lines<PREC, DIP>(p, fr, src, teams[team], sums + team * kTeamUnits * 96, first, count, in_list, out_list,
                          out_count ? out_count + f : nullptr, team, wid, lane);
    __syncthreads();  // both teams are done with the item and the frame's charges
  }
}

// Sources a CTA can hold in shared memory beside the exchanged sums (0: FP64).
int team_resident_limit(int prec, int source) {
  if (prec != kFP32C) return 0;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const int64_t room = int64_t(optin) - static_cast<int64_t>(team_fixed_bytes<kFP32C>()) - 256;
  if (room <= 0) return 0;
  return static_cast<int>(room / (source == kDipoles ? 24 : 16)) / kChargePad32 * kChargePad32;
}

template <int PREC, bool DIP>
cudaError_t launch_team_t(const TopoParams& p, const TopoFrame& f0, int fresh, int num_sms,
                          cudaStream_t s) {
  const auto bytes = [](int resident) { return team_fixed_bytes<PREC>() + static_cast<size_t>(resident) * (DIP ? 24 : 16); };
  const size_t smem = bytes(PREC == kFP32C ? p.max_team_resident : 0);
  // (always the largest size: see launch_topo_t)
  const cudaError_t err = cudaFuncSetAttribute(
      team_kernel<PREC, DIP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      static_cast<int>(bytes(team_resident_limit(PREC, DIP ? kDipoles : kCharges))));
  if (err != cudaSuccess) return err;
  const int64_t lines = p.frames ? p.sum_lines : p.n_lines;
  const int grid = fresh ? static_cast<int>(std::min<int64_t>(num_sms, lines)) : num_sms;
  for (int round = 0; round < p.rounds; ++round) {
    team_kernel<PREC, DIP><<<grid, kTeams * kTeamThreads, smem, s>>>(p, f0, fresh, round);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

// As topo_resident_count, less the space of the exchanged sums.
int topo_team_resident(int prec, int source, int n_pad) {
  const int limit = team_resident_limit(prec, source);
  if (limit <= 0) return 0;
  if (n_pad <= limit) return n_pad;
  constexpr int kRun = 2 * 32 * kLanePairs;
  return limit / kRun * kRun;
}

double topo_diag_steps(const double* half, double step) {
  return 2.0 * std::sqrt(half[0] * half[0] + half[1] * half[1] + half[2] * half[2]) / std::fabs(step);
}

int topo_team_rounds(int num_sms, int64_t sum_lines, double diag_steps) {
  if (sum_lines <= num_sms) return 1;  // a line per SM at most: nothing to even out
  const double r = std::ceil(diag_steps / kTeamMinSteps);  // infinite for a zero step
  return r < kTeamRounds ? std::max(1, static_cast<int>(r)) : kTeamRounds;
}

cudaError_t launch_topo_team(int prec, const TopoParams& p, const TopoFrame& f0, int fresh, int num_sms,
                             cudaStream_t s) {
  if (p.source == kDipoles)
    return prec == kFP32C ? launch_team_t<kFP32C, true>(p, f0, fresh, num_sms, s)
                          : launch_team_t<kFP64, true>(p, f0, fresh, num_sms, s);
  return prec == kFP32C ? launch_team_t<kFP32C, false>(p, f0, fresh, num_sms, s)
                        : launch_team_t<kFP64, false>(p, f0, fresh, num_sms, s);
}

}  // namespace cpetgb
