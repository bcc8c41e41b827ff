// topo.cu -- persistent streamline kernel (K3).
//
// Replaces thread_operation (CPET/utils/math_module.c:523-591), run by the
// reference once per streamline in a multiprocessing.Pool
// (CPET/source/calculator.py:675-712), and the windowed PyTorch pipeline of
// compute_topo_GPU_batch_filter (CPET/source/calculator.py:793-978,
// CPET/utils/gpu.py:24-399).  Semantics kept from thread_operation:
//   * Euler step x <- x + h * E/|E| with the unsoftened Coulomb field
//     (propagate_topo, math_module.c:489-503; calc_field_base 296-333);
//   * at most n_iter steps; the loop stops at the first position strictly
//     outside the box (math_module.c:539-554) and keeps that position;
//   * two extra steps from the start point and two from the end point, the
//     curvature |v' x v''| / |v'|^3 at both ends (curve, math_module.c:108-121)
//     with v' = x1 - x0, v'' = x2 - 2 x1 + x0, averaged; distance |x_end - x0|
//     (euclidean_dist, math_module.c:99-105).
// Results are written at the line's start-order index.
//
// Organisation (one persistent grid, all SMs):
//   * a warp owns S line slots; slot s lives in lane s (FP64 position, step
//     count, cap, phase) plus a small record in shared memory (start point and
//     the points needed for the curvature);
//   * every step the 32 lanes split the frame's charges (lane-strided) and
//     evaluate the field at all active slots' positions; the per-lane partial
//     sums are reduced across the warp;
//   * a slot whose line is finished writes its result and takes the next line
//     index from a global atomic counter: lines are retired and refilled
//     without any block-wide synchronisation, so short and long lines mix.
//
// Precision forms:
//   FP32C  charges in pairs of float4 records held in shared memory (bulk
//          async copies per CTA; a frame larger than shared memory keeps a
//          prefix there and streams the rest from L2); pair terms in FP32 with
//          the MUFU rsqrt,
//          per-lane Kahan accumulation across charge tiles and an error-free
//          (TwoSum) warp reduction; the step vector is formed in FP32 and added
//          to an FP64 position; box test, curvature and distance in FP64.
//   FP64   every operation in IEEE double; charges read from global memory
//          (L2-resident) as (x,y,z,q) doubles.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "topo_lines.cuh"

namespace cpetgb {
namespace {

constexpr int kTopoThreads = 512;
constexpr int kTopoWarps = kTopoThreads / 32;
// Line slots per warp S (template parameter): 4 (default) or 2.

// ---------------------------------------------------------------------------
// Persistent kernel.
// ---------------------------------------------------------------------------

// Hand-over of a frame's last lines.  Once the queue is empty and a CTA holds at
// most kTeamLinesPerSm lines, most of its warps have nothing to do and the rest
// sweep a line alone; its warps then write their lines' states to the frame's
// records and leave, and the team kernel finishes them, spread over all SMs.  A CTA
// hands over at most kTeamLinesPerSm lines of a frame (it has that many left when its
// first warp does, and gets no more), so a frame with records for that many from
// every CTA, or for all of its lines, never runs out of them; one with fewer has none.
struct HandOver {
  TopoState* rec;  // the frame's records; null: no hand-over
  int* count;      // records written
};

__device__ __forceinline__ HandOver hand_over_of(const TopoParams& p, const TopoFrame& fr, int f) {
  const bool room = fr.left_cap > 0 && fr.left_cap >= min(fr.n_lines, static_cast<int>(gridDim.x) * kTeamLinesPerSm);
  return HandOver{p.left && room ? p.left + fr.left_off : nullptr, p.left_count + f};
}

__device__ __forceinline__ void hand_over(const HandOver& h, const Slot& sl, const SlotRec& rec,
                                          unsigned active, int lane) {
  const int na = __popc(active);
  const int leader = __ffs(active) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(h.count, na);
  base = __shfl_sync(0xffffffffu, base, leader);
  if ((active >> lane) & 1u) {
    TopoState* t = h.rec + base + __popc(active & ((1u << lane) - 1u));
    for (int k = 0; k < 3; ++k) {
      t->x0[k] = rec.x0[k];
      t->xip[k] = rec.xip[k];
      t->xipp[k] = rec.xipp[k];
      t->xend[k] = rec.xend[k];
      t->xe1[k] = rec.xe1[k];
      t->pos[k] = sl.pos[k];
    }
    t->line = sl.line;
    t->phase = sl.phase;
    t->steps = sl.steps;
    t->cap = sl.cap;
  }
}

// One line slot set per warp; processes the lines of frame `fc` (g: its sources
// in global memory, FP32C in the pair layout; res_pairs of its pairs also in
// shared memory at sm_off) until the frame's queue is exhausted and the warp's
// slots are drained.
template <int PREC, int S, bool DIP, int SRC>
__device__ __forceinline__ void run_frame(const TopoParams& p, const FrameCtx& fc, int* queue,
                                          const ulonglong2* g, uint32_t sm_off, int res_pairs, int n_pad,
                                          SlotRec* my_rec, int lane, const HandOver& hand, int* s_idle) {
  Slot sl;
  sl.line = -1;
  sl.phase = kMain;
  sl.steps = sl.cap = 0;
  sl.pos[0] = sl.pos[1] = sl.pos[2] = 0.0;
  sl.posf[0] = sl.posf[1] = sl.posf[2] = 0.f;
  // One frame: the first lines are dealt out evenly over the CTAs, the queue
  // hands out the rest.  A table of frames: all from the queue (a CTA may reach
  // a frame late, or not at all).
  const int dealt = p.frames ? 0 : static_cast<int>(gridDim.x) * kTopoWarps * S;
  if (lane < S) {
    const int li = p.frames ? atomicAdd(queue, 1)
                            : (lane * kTopoWarps + (threadIdx.x >> 5)) * static_cast<int>(gridDim.x) +
                                  static_cast<int>(blockIdx.x);
    if (li >= fc.n_lines) atomicAdd(s_idle, 1);
    slot_load(sl, *my_rec, li < fc.n_lines ? static_cast<int>(fc.line_off + li) : -1, p);
  }
  for (;;) {
    const unsigned active = __ballot_sync(0xffffffffu, lane < S && sl.line >= 0);
    const int na = __popc(active);
    if (na == 0) break;
    // (other warps count s_idle up meanwhile: a vote, so that the warp's lanes, whatever
    // each of them read, take the same branch to the shuffles of hand_over)
    if (hand.rec &&
        __any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(s_idle) >= kTopoWarps * S - kTeamLinesPerSm)) {
      hand_over(hand, sl, *my_rec, active, lane);
      break;
    }
    // owner lane of each active slot, in order; this lane's rank among them
    int src_of[S];
    int my_rank = -1;
    {
      unsigned m = active;
#pragma unroll
      for (int e = 0; e < S; ++e) {
        src_of[e] = m ? (__ffs(m) - 1) : 0;
        if (m) m &= m - 1;
        if (src_of[e] == lane && e < na) my_rank = e;
      }
    }

    double nx[3];
    if constexpr (PREC == kFP32C) {
      float Ef[3];
      sweep_slots<S, DIP, SRC>(na, sl.posf, src_of, max(my_rank, 0), sm_off, res_pairs, g, n_pad / 2, Ef);
      if (my_rank >= 0) euler_step(Ef, sl.pos, fc.step, nx);
    } else {
      double ex[S][3];
#pragma unroll
      for (int e = 0; e < S; ++e)
#pragma unroll
        for (int c = 0; c < 3; ++c) ex[e][c] = __shfl_sync(0xffffffffu, sl.pos[c], src_of[e]);
      double Es[S][3];
      if constexpr (DIP) {
        const Dipole64* src = reinterpret_cast<const Dipole64*>(g);
        switch (na) {
          case 1: sweep_f64<1, S>(src, n_pad, lane, ex, Es); break;
          case 2: sweep_f64<2, S>(src, n_pad, lane, ex, Es); break;
          case 3: sweep_f64<(S > 2 ? 3 : 2), S>(src, n_pad, lane, ex, Es); break;
          default: sweep_f64<S, S>(src, n_pad, lane, ex, Es); break;
        }
      } else {
        const Charge64* src = reinterpret_cast<const Charge64*>(g);
        switch (na) {
          case 1: sweep_f64<1, S>(src, n_pad, lane, ex, Es); break;
          case 2: sweep_f64<2, S>(src, n_pad, lane, ex, Es); break;
          case 3: sweep_f64<(S > 2 ? 3 : 2), S>(src, n_pad, lane, ex, Es); break;
          default: sweep_f64<S, S>(src, n_pad, lane, ex, Es); break;
        }
      }
      if (my_rank >= 0) {
        double E[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int e = 0; e < S; ++e)
          if (e == my_rank)
#pragma unroll
            for (int c = 0; c < 3; ++c) E[c] = Es[e][c];
        euler_step(E, sl.pos, fc.step, nx);
      }
    }

    if (my_rank >= 0) {
      if (slot_advance<PREC == kFP32C>(sl, *my_rec, nx, p, fc)) {
        const int li = dealt + atomicAdd(queue, 1);
        if (li >= fc.n_lines) atomicAdd(s_idle, 1);
        slot_load(sl, *my_rec, li < fc.n_lines ? static_cast<int>(fc.line_off + li) : -1, p);
      }
    }
    __syncwarp();
  }
}

// One frame's share of a launch's work.
__device__ __forceinline__ double frame_work(const TopoFrame& fr) {
  return static_cast<double>(fr.n_lines) * fr.n_pad;
}

// The CTAs start spread over the frames by their work and visit them in table
// order from there.  With all CTAs starting at the first frame, a frame of 3,000
// lines fills the slots of 94 CTAs at once and leaves them nothing to refill
// with, and half of the launch's lines are handed over (6 frames x 3,000 lines of
// 5,000 to 20,000 charges: 93 ms here and 72 ms of rounds; spread, 123 and 38).
// A CTA stays on a frame while its line queue lasts, then moves on (after its
// own warps are done or have handed their lines over, so the shared copy of the
// charges can be replaced).
// DIP: the sources are point dipoles (FP32C: three 16-byte pair blocks per
// frame; FP64: Dipole64 records) instead of point charges.  SRC: kSrcShared when
// every frame of the launch fits shared memory, kSrcSplit otherwise (FP64:
// always, its sources are read from global memory).
template <int PREC, int S, bool DIP, int SRC>
__global__ void __launch_bounds__(kTopoThreads, 1) topo_kernel(TopoParams p, TopoFrame frame0) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_skip, s_first;
  __shared__ int s_idle;  // line slots of this CTA that found the frame's queue empty
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  SlotRec* recs = reinterpret_cast<SlotRec*>(smem_raw);  // [kTopoWarps][S]
  constexpr uint32_t rec_bytes = sizeof(SlotRec) * kTopoWarps * S;
  constexpr uint32_t sm_off = rec_bytes + 128;  // the resident sources
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + rec_bytes);
  SlotRec* my_rec = recs + warp * S + (lane < S ? lane : 0);
  const int n_frames = p.frames ? p.n_frames : 1;
  uint32_t load_parity = 0;
  if (PREC == kFP32C && threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }

  if (p.frames && warp == 0) {
    // work (lines x sources) before this CTA's share, and the frame it lies in
    double total = 0.0;
    for (int f = lane; f < n_frames; f += 32) total += frame_work(p.frames[f]);
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const double mine = total * (blockIdx.x + 0.5) / gridDim.x;
    double base = 0.0;
    int first = 0;
    for (int f0 = 0; f0 < n_frames; f0 += 32) {
      double incl = f0 + lane < n_frames ? frame_work(p.frames[f0 + lane]) : 0.0;
      for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const unsigned past = __ballot_sync(0xffffffffu, f0 + lane < n_frames && base + incl > mine);
      if (past) {
        first = f0 + __ffs(past) - 1;
        break;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_first = first;
  }
  __syncthreads();
  const int first_frame = p.frames ? s_first : 0;

  for (int i = 0; i < n_frames; ++i) {
    const int f = first_frame + i < n_frames ? first_frame + i : first_frame + i - n_frames;
    const TopoFrame fr = p.frames ? p.frames[f] : frame0;
    int* queue = p.queue + f;
    __syncthreads();  // the CTA's warps are done with the previous frame
    if (threadIdx.x == 0) {
      // a table's frame may be used up before this CTA reaches it; a single
      // frame's first lines are dealt to this CTA whatever the queue says
      s_skip = p.frames && *reinterpret_cast<volatile int*>(queue) >= fr.n_lines;
      s_idle = 0;
    }
    __syncthreads();
    if (s_skip) continue;
    const size_t elem = (PREC == kFP32C) ? 16 : 32;
    const char* src = static_cast<const char*>(p.packed) + fr.packed_off * elem;
    if constexpr (PREC == kFP32C) {
      // the frame's first fr.resident sources -- all of them, or a prefix of
      // whole Kahan runs when the frame exceeds shared memory -- block by block
      if (threadIdx.x == 0) {
        const uint32_t blk = static_cast<uint32_t>(fr.resident / 2) * 16u;  // bytes of one block's prefix
        constexpr int n_blk = DIP ? 3 : 2;
        mbar_arrive_expect_tx(bar, blk * n_blk);
        constexpr uint32_t kChunk = 32768;
        for (int b = 0; b < n_blk; ++b) {  // block b of the frame starts at b * n_pad/2 pairs
          const char* bs = src + static_cast<size_t>(b) * (fr.n_pad / 2) * 16;
          unsigned char* bd = smem_raw + sm_off + static_cast<size_t>(b) * blk;
          for (uint32_t off = 0; off < blk; off += kChunk)
            bulk_g2s(bd + off, bs + off, min(kChunk, blk - off), bar);
        }
      }
      const bool mine = mbar_wait(bar, load_parity, p.status);
      load_parity ^= 1u;
      if (!__syncthreads_and(mine)) return;
    }
    FrameCtx fc;
    fc.line_off = fr.line_off;
    fc.n_lines = fr.n_lines;
    fc.step = fr.step;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      fc.half[k] = fr.half[k];
      fc.hf[k] = static_cast<float>(fr.half[k]);
    }
    const HandOver hand = hand_over_of(p, fr, f);
    run_frame<PREC, S, DIP, SRC>(p, fc, queue, reinterpret_cast<const ulonglong2*>(src), sm_off, fr.resident / 2,
                            fr.n_pad, my_rec, lane, hand, &s_idle);
  }
}

// ---------------------------------------------------------------------------
// Serving engine: continuous batching of streamline requests.
// ---------------------------------------------------------------------------
// Warps claim chunks of lines from a ring the host appends to while the
// kernel runs; a slot that finishes a line takes the next line of the warp's
// chunk (or of a newly claimed chunk, possibly of another frame), so requests
// arriving while others are in flight are admitted as slots free up.  Each
// step the warp sweeps the charges once per distinct frame among its active
// slots.  Charges are read from global memory (L2).
//
// Lifetime of a launch: a warp without lines polls for chunks, and stays while
// any warp of the launch has lines or claims happen, so work published later
// finds every warp of the launch (a launch whose idle warps had left would
// serve it with the few warps still busy, while the next launch waits behind
// it).  Once no warp has had lines and nothing was claimed for kEngineIdleNs,
// the first warp to see it closes the launch: no warp claims again, and each
// ends when its lines are done.  Work published after that goes to the next
// launch, which the host keeps queued.
constexpr int kEngineThreads = 256;
constexpr int kEngineWarps = kEngineThreads / 32;
constexpr unsigned long long kEngineIdleNs = 50000000ull;      // launch idle 50 ms: it closes
constexpr unsigned long long kEngineMaxWaitNs = 60000000000ull;  // bound on one idle wait (60 s)

__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Claims the next published chunk; -1 when none is published.  The claim
// counter lives in device memory (L2 atomics); every failed CAS means another
// warp advanced it, so the loop ends within the number of published chunks.
// The host sees claims through a monotonic mirror in host-mapped memory.
__device__ int engine_claim(const EngineParams& E) {
  for (int tries = 0; tries < (1 << 20); ++tries) {
    const int t = ld_acquire_sys(E.tail);
    const int h = *reinterpret_cast<volatile int*>(E.head);
    if (h >= t) return -1;
    if (atomicCAS(E.head, h, h + 1) == h) {
      atomicMax_system(E.head_mirror, h + 1);
      return h;
    }
  }
  return -1;
}

__device__ __forceinline__ int ld_volatile(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

// Idle wait of a warp with no line (lane 0 only): polls for a chunk with a
// sleep growing from 20 to 320 us.  Returns the claimed chunk, or -1 once the
// launch is closed -- by this warp when neither a busy warp nor a claim was
// seen for kEngineIdleNs, or after kEngineMaxWaitNs in any case.
__device__ int engine_idle_wait(const EngineParams& E) {
  const unsigned long long t0 = globaltimer_ns();
  unsigned long long quiet_since = t0;
  int last_head = ld_volatile(E.head);
  unsigned sleep_ns = 20000;
  for (;;) {
    if (ld_volatile(E.closing)) return -1;
    const int got = engine_claim(E);
    if (got >= 0) return got;
    const unsigned long long now = globaltimer_ns();
    const int h = ld_volatile(E.head);
    if (ld_volatile(E.busy) > 0 || h != last_head) {
      quiet_since = now;
      last_head = h;
    } else if (now - quiet_since > kEngineIdleNs) {
      atomicExch(E.closing, 1);
      return -1;
    }
    if (now - t0 > kEngineMaxWaitNs) {
      atomicExch(E.closing, 1);
      return -1;
    }
    __nanosleep(sleep_ns);
    if (sleep_ns < 320000) sleep_ns *= 2;
  }
}

__device__ __forceinline__ EngineChunk engine_read_chunk(const EngineParams& E, int idx) {
  const volatile EngineChunk* c = E.chunks + (idx % E.chunk_capacity);
  EngineChunk r;
  r.frame = c->frame;
  r.request = c->request;
  r.line_begin = c->line_begin;
  r.line_end = c->line_end;
  r.step = c->step;
  r.half[0] = c->half[0];
  r.half[1] = c->half[1];
  r.half[2] = c->half[2];
  return r;
}

// slot_load for lines the host wrote while the kernel may run: read past L1.
__device__ void engine_slot_load(Slot& sl, SlotRec& rec, int line, const TopoParams& p) {
  sl.line = line;
  const double* s = p.starts + 3 * static_cast<int64_t>(line);
  double st[3];
  for (int k = 0; k < 3; ++k) rec.x0[k] = st[k] = __ldcg(s + k);
  set_pos(sl, st);
  sl.cap = max(__ldcg(p.n_iter + line), 0);
  if (sl.cap > kMaxLineCap) {
    atomicCAS(p.status, kDevOk, kDevBadCap);
    sl.cap = 0;
  }
  sl.steps = 0;
  if (sl.cap > 0) {
    sl.phase = kMain;
  } else {
    sl.phase = kStart1;
    for (int k = 0; k < 3; ++k) rec.xend[k] = st[k];
  }
}

// Per-slot request context, kept in shared memory (read once per step).
struct EngineSlotCtx {
  long long off;  // the frame's first packed element
  int frame;
  int req;
  int n_pad;
  int pad_;
  double step;
  double half[3];
};

template <int PREC, int S>
__global__ void __launch_bounds__(kEngineThreads, 2) engine_kernel(EngineParams E) {
  __shared__ SlotRec recs[kEngineWarps][S];
  __shared__ EngineSlotCtx sctx[kEngineWarps][S];
  __shared__ EngineChunk wchunk[kEngineWarps];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  SlotRec& rec = recs[warp][lane < S ? lane : 0];
  EngineSlotCtx& my = sctx[warp][lane < S ? lane : 0];
  const size_t elem = (PREC == kFP32C) ? 16 : 32;
  if (lane < S) my.frame = -1;

  Slot sl;
  sl.line = -1;
  sl.phase = kMain;
  sl.steps = sl.cap = 0;
  sl.pos[0] = sl.pos[1] = sl.pos[2] = 0.0;
  sl.posf[0] = sl.posf[1] = sl.posf[2] = 0.f;
  int c_next = 0, c_end = 0;  // the warp's chunk cursor (uniform across the warp)
  int backoff = 0;            // steps to wait before claiming again after an empty queue
  bool counted = false;       // this warp is counted in E.busy (uniform)
  __syncwarp();

  for (;;) {
    // refill idle slots, claiming chunks as needed
    unsigned need = __ballot_sync(0xffffffffu, lane < S && sl.line < 0);
    const bool all_idle = __popc(need) == S;
    if (all_idle && counted && c_next >= c_end) {  // no line held or left in the chunk
      if (lane == 0) atomicSub(E.busy, 1);
      counted = false;
    }
    if (backoff > 0 && !all_idle) {
      --backoff;
      need = (c_next < c_end) ? need : 0u;  // only lines of the current chunk
    }
    bool took = false;  // a line was given to a slot in this pass
    while (need) {
      if (c_next >= c_end) {
        int got = -1;
        if (lane == 0) {
          if (!ld_volatile(E.closing)) got = engine_claim(E);
          if (got < 0 && all_idle && !took) got = engine_idle_wait(E);
          if (got >= 0 && !counted) atomicAdd(E.busy, 1);
          if (got >= 0) wchunk[warp] = engine_read_chunk(E, got);
        }
        got = __shfl_sync(0xffffffffu, got, 0);
        __syncwarp();
        if (got < 0) {
          backoff = 8;
          break;
        }
        counted = true;
        c_next = wchunk[warp].line_begin;
        c_end = wchunk[warp].line_end;
        continue;
      }
      const int target = __ffs(need) - 1;
      const int line = c_next++;
      if (lane == target) {
        const EngineChunk& ch = wchunk[warp];
        // frame slots are reused while the kernel runs: read the table past L1
        my.off = __ldcg(&E.frames[ch.frame].packed_off);
        my.frame = ch.frame;
        my.req = ch.request;
        my.n_pad = __ldcg(&E.frames[ch.frame].n_pad);
        my.step = ch.step;
        for (int k = 0; k < 3; ++k) my.half[k] = ch.half[k];
        engine_slot_load(sl, rec, line, E.p);
      }
      took = true;
      need &= ~(1u << target);
      __syncwarp();
    }
    const unsigned active = __ballot_sync(0xffffffffu, lane < S && sl.line >= 0);
    if (active == 0) break;

    double nx[3] = {0.0, 0.0, 0.0};
    unsigned remaining = active;
    while (remaining) {
      const int leader = __ffs(remaining) - 1;
      const EngineSlotCtx& L = sctx[warp][leader];
      const int f = L.frame;
      const unsigned group =
          __ballot_sync(0xffffffffu, lane < S && sl.line >= 0 && my.frame == f) & remaining;
      remaining &= ~group;
      const int na = __popc(group);
      const int n_pad = L.n_pad;
      const ulonglong2* gA = reinterpret_cast<const ulonglong2*>(
          static_cast<const char*>(E.p.packed) + L.off * static_cast<long long>(elem));
      int src_of[S];
      int my_rank = -1;
      {
        unsigned m = group;
#pragma unroll
        for (int e = 0; e < S; ++e) {
          src_of[e] = m ? (__ffs(m) - 1) : 0;
          if (m) m &= m - 1;
          if (src_of[e] == lane && e < na) my_rank = e;
        }
      }
      if constexpr (PREC == kFP32C) {
        float Ef[3];
        sweep_slots<S, false, kSrcGlobal>(na, sl.posf, src_of, max(my_rank, 0), 0, 0, gA, n_pad / 2, Ef);
        if (my_rank >= 0) euler_step(Ef, sl.pos, my.step, nx);
      } else {
        double ex[S][3];
#pragma unroll
        for (int e = 0; e < S; ++e)
#pragma unroll
          for (int c = 0; c < 3; ++c) ex[e][c] = __shfl_sync(0xffffffffu, sl.pos[c], src_of[e]);
        double Es[S][3];
        const Charge64* g = reinterpret_cast<const Charge64*>(gA);
        switch (na) {
          case 1: sweep_f64<1, S>(g, n_pad, lane, ex, Es); break;
          case 2: sweep_f64<2, S>(g, n_pad, lane, ex, Es); break;
          case 3: sweep_f64<(S > 2 ? 3 : 2), S>(g, n_pad, lane, ex, Es); break;
          default: sweep_f64<S, S>(g, n_pad, lane, ex, Es); break;
        }
        if (my_rank >= 0) {
          double Ev[3] = {0.0, 0.0, 0.0};
#pragma unroll
          for (int e = 0; e < S; ++e)
            if (e == my_rank)
#pragma unroll
              for (int c = 0; c < 3; ++c) Ev[c] = Es[e][c];
          euler_step(Ev, sl.pos, my.step, nx);
        }
      }
    }

    if (lane < S && sl.line >= 0) {
      FrameCtx fc;
      fc.line_off = 0;
      fc.n_lines = 0;
      fc.step = my.step;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        fc.half[k] = my.half[k];
        fc.hf[k] = static_cast<float>(my.half[k]);
      }
      if (slot_advance<PREC == kFP32C>(sl, rec, nx, E.p, fc)) {
        __threadfence_system();  // the line's results before its completion count
        atomicAdd_system(E.done + my.req, 1);
        sl.line = -1;
      }
    }
    __syncwarp();
  }
}

__global__ void pack_pairs_kernel(int64_t n, int64_t n_pad, const double* __restrict__ x,
                                  const double* __restrict__ q, float4* __restrict__ out) {
  const int64_t n_pairs = n_pad / 2;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n_pairs;
       p += (int64_t)gridDim.x * blockDim.x) {
    float c[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t i = 2 * p + h;
      if (i < n) {
        c[h][0] = static_cast<float>(x[3 * i]);
        c[h][1] = static_cast<float>(x[3 * i + 1]);
        c[h][2] = static_cast<float>(x[3 * i + 2]);
        c[h][3] = static_cast<float>(q[i]);
      } else {  // zero charge far outside any box
        c[h][0] = c[h][1] = c[h][2] = 1.0e4f;
        c[h][3] = 0.f;
      }
    }
    out[p] = make_float4(c[0][0], c[1][0], c[0][1], c[1][1]);            // A
    out[n_pairs + p] = make_float4(c[0][2], c[1][2], c[0][3], c[1][3]);  // B
  }
}

// Dipoles, FP32C: A[p] = {x, x', y, y'}, B[p] = {z, z', 3 mu_x, 3 mu_x'},
// C[p] = {mu_y, mu_y', mu_z, mu_z'} for the pair (2p, 2p + 1); padding =
// zero moments far outside any box (they add exactly 0).
__global__ void pack_dipole_pairs_kernel(int64_t n, int64_t n_pad, const double* __restrict__ x,
                                         const double* __restrict__ mu, float4* __restrict__ out) {
  const int64_t n_pairs = n_pad / 2;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n_pairs;
       p += (int64_t)gridDim.x * blockDim.x) {
    float c[2][6];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t i = 2 * p + h;
      const bool in = i < n;
      c[h][0] = in ? static_cast<float>(x[3 * i]) : 1.0e4f;
      c[h][1] = in ? static_cast<float>(x[3 * i + 1]) : 1.0e4f;
      c[h][2] = in ? static_cast<float>(x[3 * i + 2]) : 1.0e4f;
      c[h][3] = in ? static_cast<float>(3.0 * mu[3 * i]) : 0.f;
      c[h][4] = in ? static_cast<float>(mu[3 * i + 1]) : 0.f;
      c[h][5] = in ? static_cast<float>(mu[3 * i + 2]) : 0.f;
    }
    out[p] = make_float4(c[0][0], c[1][0], c[0][1], c[1][1]);
    out[n_pairs + p] = make_float4(c[0][2], c[1][2], c[0][3], c[1][3]);
    out[2 * n_pairs + p] = make_float4(c[0][4], c[1][4], c[0][5], c[1][5]);
  }
}

__global__ void pack_dipole64_kernel(int64_t n, int64_t n_pad, const double* __restrict__ x,
                                     const double* __restrict__ mu, Dipole64* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_pad;
       i += (int64_t)gridDim.x * blockDim.x) {
    Dipole64 d;
    if (i < n) {
      d.x = x[3 * i]; d.y = x[3 * i + 1]; d.z = x[3 * i + 2];
      d.mx = mu[3 * i]; d.my = mu[3 * i + 1]; d.mz = mu[3 * i + 2];
    } else {
      d.x = d.y = d.z = 1.0e4;
      d.mx = d.my = d.mz = 0.0;
    }
    out[i] = d;
  }
}

// Dynamic shared memory: slot records, the mbarrier, and the resident sources
// (16 bytes per FP32C charge, 24 per FP32C dipole).
size_t topo_smem_bytes(int S, int max_resident_pad, bool dip = false) {
  return sizeof(SlotRec) * kTopoWarps * S + 128 +
         static_cast<size_t>(max_resident_pad) * (dip ? 24 : 16);
}

template <int PREC, int S, bool DIP, int SRC>
cudaError_t launch_topo_t(const TopoParams& p, const TopoFrame& f0, int total_lines, int num_sms,
                          cudaStream_t s) {
  const size_t smem = topo_smem_bytes(S, PREC == kFP32C ? p.max_resident_pad : 0, DIP);
  // the limit belongs to the kernel, not to the calling thread: always the largest size,
  // so that a thread cannot lower it between another's setting and its launch
  const size_t most = topo_smem_bytes(S, static_cast<int>(topo_resident_limit(PREC, DIP ? kDipoles : kCharges)), DIP);
  const cudaError_t err = cudaFuncSetAttribute(
      topo_kernel<PREC, S, DIP, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
  if (err != cudaSuccess) return err;
  // one CTA per SM: its 512 threads take more than half of an SM's registers
  const int grid = std::max(1, std::min(num_sms, total_lines));
  topo_kernel<PREC, S, DIP, SRC><<<grid, kTopoThreads, smem, s>>>(p, f0);
  return cudaGetLastError();
}

__global__ void pack_frames_kernel(int prec, const TopoFrame* __restrict__ frames,
                                   const int64_t* __restrict__ src, const double* __restrict__ x,
                                   const double* __restrict__ q, void* __restrict__ packed) {
  const int f = blockIdx.y;
  const TopoFrame fr = frames[f];
  const int64_t off = src[2 * f], n = src[2 * f + 1];
  const double* fx = x + 3 * off;
  const double* fq = q + off;
  if (prec == kFP32C) {
    float4* out = static_cast<float4*>(packed) + fr.packed_off;
    const int64_t n_pairs = fr.n_pad / 2;
    for (int64_t pp = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pp < n_pairs;
         pp += (int64_t)gridDim.x * blockDim.x) {
      float c[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t i = 2 * pp + h;
        if (i < n) {
          c[h][0] = static_cast<float>(fx[3 * i]);
          c[h][1] = static_cast<float>(fx[3 * i + 1]);
          c[h][2] = static_cast<float>(fx[3 * i + 2]);
          c[h][3] = static_cast<float>(fq[i]);
        } else {
          c[h][0] = c[h][1] = c[h][2] = 1.0e4f;
          c[h][3] = 0.f;
        }
      }
      out[pp] = make_float4(c[0][0], c[1][0], c[0][1], c[1][1]);
      out[n_pairs + pp] = make_float4(c[0][2], c[1][2], c[0][3], c[1][3]);
    }
  } else {
    Charge64* out = static_cast<Charge64*>(packed) + fr.packed_off;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < fr.n_pad;
         i += (int64_t)gridDim.x * blockDim.x) {
      Charge64 c;
      if (i < n) {
        c.x = fx[3 * i];
        c.y = fx[3 * i + 1];
        c.z = fx[3 * i + 2];
        c.q = fq[i];
      } else {
        c.x = c.y = c.z = 1.0e4;
        c.q = 0.0;
      }
      out[i] = c;
    }
  }
}

}  // namespace

int topo_charge_pad(int prec) { return prec == kFP32C ? kChargePad32 : kChargePad64; }

int engine_threads() { return kEngineThreads; }

// ctas = SMs x CTAs per SM (1 or 2; a CTA takes half of an SM's registers).
// At one CTA per SM the engine runs beside grid launches: its SMs keep the
// largest shared-memory carveout so grid blocks (33 KB of staged charge
// tiles) fit next to it.
cudaError_t launch_engine(int prec, const EngineParams& e, int ctas, cudaStream_t s) {
  cudaError_t err;
  if (prec == kFP32C) {
    err = cudaFuncSetAttribute(engine_kernel<kFP32C, 4>,
                               cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    if (err != cudaSuccess) return err;
    engine_kernel<kFP32C, 4><<<ctas, kEngineThreads, 0, s>>>(e);
  } else {
    err = cudaFuncSetAttribute(engine_kernel<kFP64, 4>,
                               cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    if (err != cudaSuccess) return err;
    engine_kernel<kFP64, 4><<<ctas, kEngineThreads, 0, s>>>(e);
  }
  return cudaGetLastError();
}

// Charges (or dipoles) of a frame held in shared memory: all of them when the
// frame fits, else the largest prefix of whole Kahan runs (32 x kLanePairs
// pairs) that fits; 0 for FP64.
int topo_resident_count(int prec, int source, int n_pad) {
  const int limit = static_cast<int>(topo_resident_limit(prec, source));
  if (limit <= 0) return 0;
  if (n_pad <= limit) return n_pad;
  constexpr int kRun = 2 * 32 * kLanePairs;
  return (limit / kRun) * kRun;
}

size_t topo_resident_limit(int prec, int source) {
  if (prec != kFP32C) return 0;  // FP64 sources are read from global memory (L2)
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t fixed = topo_smem_bytes(4, 0) + 256;  // + static shared memory
  if (optin <= static_cast<int>(fixed)) return 0;
  size_t n = (static_cast<size_t>(optin) - fixed) / (source == kDipoles ? 24 : 16);
  return (n / kChargePad32) * kChargePad32;
}

cudaError_t launch_pack_dipoles(int prec, int64_t n, int64_t n_pad, const double* x,
                                const double* mu, void* packed, cudaStream_t s) {
  if (n_pad <= 0) return cudaSuccess;
  if (prec == kFP32C) {
    const int blocks = static_cast<int>(std::min<int64_t>((n_pad / 2 + 255) / 256, 4096));
    pack_dipole_pairs_kernel<<<blocks, 256, 0, s>>>(n, n_pad, x, mu, static_cast<float4*>(packed));
  } else {
    const int blocks = static_cast<int>(std::min<int64_t>((n_pad + 255) / 256, 4096));
    pack_dipole64_kernel<<<blocks, 256, 0, s>>>(n, n_pad, x, mu, static_cast<Dipole64*>(packed));
  }
  return cudaGetLastError();
}

size_t topo_source_bytes(int prec, int source) {
  if (source == kDipoles) return prec == kFP32C ? 24 : sizeof(Dipole64);
  return prec == kFP32C ? 16 : sizeof(Charge64);
}

cudaError_t launch_pack_topo(int prec, int64_t n, int64_t n_pad, const double* x, const double* q,
                             void* packed, cudaStream_t s) {
  if (prec != kFP32C) return launch_pack_f64(n, n_pad, x, q, packed, s);
  if (n_pad <= 0) return cudaSuccess;
  const int blocks = static_cast<int>(std::min<int64_t>((n_pad / 2 + 255) / 256, 4096));
  pack_pairs_kernel<<<blocks, 256, 0, s>>>(n, n_pad, x, q, static_cast<float4*>(packed));
  return cudaGetLastError();
}

cudaError_t launch_pack_topo_frames(int prec, int n_frames, const TopoFrame* d_frames,
                                    const int64_t* d_src, const double* x, const double* q,
                                    void* packed, int max_pairs, cudaStream_t s) {
  if (n_frames <= 0) return cudaSuccess;
  const int bx = std::max(1, std::min((max_pairs + 255) / 256, 256));
  pack_frames_kernel<<<dim3(bx, n_frames), 256, 0, s>>>(prec, d_frames, d_src, x, q, packed);
  return cudaGetLastError();
}

template <int PREC, bool DIP, int SRC>
cudaError_t launch_topo_s(const TopoParams& p, const TopoFrame& f0, int num_sms, cudaStream_t s, int slots) {
  return slots == 2 ? launch_topo_t<PREC, 2, DIP, SRC>(p, f0, p.n_lines, num_sms, s)
                    : launch_topo_t<PREC, 4, DIP, SRC>(p, f0, p.n_lines, num_sms, s);
}

// whole: every frame of the launch fits shared memory.
template <bool DIP>
cudaError_t launch_topo_prec(int prec, bool whole, const TopoParams& p, const TopoFrame& f0, int num_sms,
                             cudaStream_t s, int slots) {
  if (prec == kFP64) return launch_topo_s<kFP64, DIP, kSrcSplit>(p, f0, num_sms, s, slots);
  return whole ? launch_topo_s<kFP32C, DIP, kSrcShared>(p, f0, num_sms, s, slots)
               : launch_topo_s<kFP32C, DIP, kSrcSplit>(p, f0, num_sms, s, slots);
}

// Line slots per warp: the tuned variant of the launch's class, which knows its lines
// but not its sources; 4 for frames of at most 1,024 sources once a CTA's slots are filled
// more than once, as a step then is mostly what a warp pays once for all of its lines.
// Four slots and two, 108 / 197 / 395 lines per SM (us): 60 charges 925 and 1,207 / 1,398
// and 1,946 / 2,359 and 3,563; 1,000 charges 1,848 and 2,141 / 2,892 and 3,405 / 5,129 and
// 6,362; but 2,000 charges 2,697 and 2,447 / 4,130 and 4,007 / 7,279 and 7,522.
constexpr int kFewSources = 1024;
int topo_slots(int prec, bool whole, const TopoParams& p, int64_t lines, int num_sms) {
  if (prec == kFP32C && whole && p.max_resident_pad <= kFewSources && lines > 96 * int64_t(num_sms)) return 4;
  return tuned_topo_slots(prec, whole, p.n_lines);
}

// Single frame: p.packed holds round_up(n_charges, topo_charge_pad(prec)) charges
// packed by launch_pack_topo (the tail being zero charges far from the box).
cudaError_t launch_topo(int prec, const TopoParams& p_in, int num_sms, cudaStream_t s) {
  if (p_in.n_lines <= 0) return cudaSuccess;
  TopoParams p = p_in;
  const int pad = topo_charge_pad(prec);
  TopoFrame f0;
  f0.packed_off = 0;
  f0.line_off = 0;
  f0.n_pad = ((std::max(p.n_charges, 1) + pad - 1) / pad) * pad;
  f0.n_lines = p.n_lines;
  f0.resident = topo_resident_count(prec, p.source, f0.n_pad);
  f0.team_resident = topo_team_resident(prec, p.source, f0.n_pad);
  f0.left_off = 0;
  f0.step = p.step;
  for (int k = 0; k < 3; ++k) f0.half[k] = p.half[k];
  p.frames = nullptr;
  p.n_frames = 1;
  p.max_resident_pad = f0.resident;
  p.max_team_resident = f0.team_resident;
  const bool whole = f0.resident == f0.n_pad;
  f0.left_cap = p.left ? topo_left_capacity(num_sms, p.n_lines, p.fresh) : 0;
  if (p.fresh) return launch_topo_team(prec, p, f0, 1, num_sms, s);
  const int slots = topo_slots(prec, whole, p, p.n_lines, num_sms);
  const cudaError_t e = p.source == kDipoles
                            ? launch_topo_prec<true>(prec, whole, p, f0, num_sms, s, slots)
                            : launch_topo_prec<false>(prec, whole, p, f0, num_sms, s, slots);
  if (e != cudaSuccess || f0.left_cap == 0) return e;
  return launch_topo_team(prec, p, f0, 0, num_sms, s);
}

// FP64: a team has the FP64 pipe busy with a line per warp.  All lines in the rounds of
// teams against the persistent kernel with rounds for its last lines (GB300, lines per
// SM: ms):
//   1,000 charges  24: 21.6 against 27.7   64: 54.1 / 62.4   256: 198 / 213
//   4,000 charges, 52 steps across the box  24: 7.3 / 7.8  128: 31.7 / 34.9
// FP32C: teams / the persistent kernel with hand-over (from 20 lines per SM) / without
// (us; box of 3 A, 5,200 steps across it):
//   lines per SM       2            8            16               20                   32
//   1,000 charges   5790/ 5169   6743/ 5940   8157/ 7496    9431/10678/ 7923   12506/11601/ 9522
//   2,000 charges   5853/ 4854   6925/ 5961   8822/ 8314   10448/11783/ 9409   14273/13356/11211
//   3,000 charges   7174/ 7981   9205/ 9361  11831/12105   14058/16183/13613   18766/17371/16634
//   4,000 charges   7615/ 9372   9776/10892  12622/13777   15138/15592/14935   19858/19640/19232
//   6,000 charges   8311/12029  12804/15484  17832/21737   21625/24633/26980   30210/32381/32623
//   8,000 charges   7580/12616  11926/17704  18056/22583   22245/26988/31413   32153/36388/39136
//   2,000 dipoles   9106/ 7581  10565/ 9206  13228/13443   15715/17253/14344   20135/19568/17889
//   4,000 dipoles   9604/12086  13185/16321  18836/20941   23929/26773/26980   31800/36513/36416
// and with 520 steps (rounds are 128 steps at least, so a launch's 10 us count):
//   3,000 charges    755/  823   1006/  968   1352/ 1251    1715/ 1793/ 1408    2064/ 1911/ 1728
//   8,000 charges    800/ 1310   1439/ 1829   2062/ 2343    2716/ 3040/ 3246    3745/ 3930/ 4028
//   8,000 dipoles   1098/ 2090   2025/ 2876   3169/ 3752    3824/ 4296/ 4730    5352/ 5478/ 6082
//   30,000 charges  1865/ 8113   3948/ 9229   6880/10177    9370/10075/13370   12191/13756/16096
// (Above 20 lines per SM teams still win for 6,000 and more charges of long lines; at 24
// with short ones they lose to hand-over or to neither.)
// A frame of one Kahan run (2,048 sources) has nothing to split, so teams only add their
// barriers and rounds; with two runs they pay up to 9 to 16 lines per SM, from three on
// to 20, and to 32 where the persistent kernel reads sources from L2.  Hand-over
// pays where a line alone on a warp is slow (sources from L2, 200 pairs' work per lane), or
// with less work where lines are long.
bool topo_fresh(int prec, int source, bool resident, double n_pad, int64_t sum_lines, int num_sms, bool lists) {
  int64_t per_sm = kMaxLeft;
  if (prec != kFP64) {
    const double lane_pairs = n_pad / 64.0;
    if (lane_pairs <= kLanePairs) return false;
    per_sm = std::min<int64_t>(resident ? 20 : 32,
                               static_cast<int64_t>(std::ceil(lane_pairs / (source == kDipoles ? 3 : 4))));
  }
  if (!lists) per_sm = std::min<int64_t>(per_sm, kTeamLinesPerSm);
  return sum_lines <= std::min(per_sm * num_sms, std::max(kMaxLeft, int64_t(kTeamLinesPerSm) * num_sms));
}

bool topo_hands_over(int prec, int source, bool resident, int n_pad, double diag_steps) {
  if (prec == kFP64 || !resident) return true;
  const double work = n_pad / 64.0 * (source == kDipoles ? 1.75 : 1.0);  // charge pairs per lane
  return work >= 200.0 || (work >= 120.0 && diag_steps >= 2000.0);
}

int topo_left_capacity(int num_sms, int64_t n_lines, bool fresh) {
  // every line, or what the CTAs of one launch may hold when they hand over
  return static_cast<int>(fresh ? n_lines : std::min(n_lines, int64_t(num_sms) * kTeamLinesPerSm));
}

cudaError_t launch_topo_frames(int prec, const TopoParams& p, int num_sms, cudaStream_t s) {
  // (line offsets alone can make n_lines positive)
  if (p.n_frames <= 0 || p.n_lines <= 0 || p.sum_lines <= 0) return cudaSuccess;
  TopoFrame dummy{};
  if (p.fresh) return launch_topo_team(prec, p, dummy, 1, num_sms, s);
  const int slots = topo_slots(prec, p.all_resident != 0, p, p.sum_lines, num_sms);
  const cudaError_t e = launch_topo_prec<false>(prec, p.all_resident != 0, p, dummy, num_sms, s, slots);
  if (e != cudaSuccess || !p.left) return e;
  return launch_topo_team(prec, p, dummy, 0, num_sms, s);
}

}  // namespace cpetgb
