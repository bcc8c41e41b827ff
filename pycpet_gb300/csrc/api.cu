// api.cu -- the C ABI of libcpetgb.so (declared in include/cpetgb.h).
//
// Host-side responsibilities: argument validation, the per-device context
// (SM count, a library stream for host-memory calls, the device status word),
// stream-ordered scratch memory (cudaMallocAsync on the call's stream),
// host<->device staging for CPETGB_HOST calls, the work decomposition of the
// grid kernels (point tiles x charge splits, largest first), and the mapping
// of device-side status words to return codes.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "cpetgb.h"
#include "kernels.cuh"

using namespace cpetgb;

namespace {

constexpr int kVersion = 10000;  // 1.0.0
constexpr int kMaxDevices = 64;

thread_local std::string g_err;
std::mutex g_mu;
std::atomic<int> g_default_prec{CPETGB_FP32C};
// FP32C field: points with |E| below this fraction of their frame's median |E|
// are recomputed in double-float arithmetic (0 turns the refinement off).
std::atomic<double> g_refine_tau{0.15};

struct Ctx {
  bool ready = false;
  int sms = 0;
  cudaStream_t stream = nullptr;  // used by CPETGB_HOST calls without a stream
  int* status = nullptr;          // device status word (DevStatus)
};
Ctx g_ctx[kMaxDevices];

int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  cudaGetLastError();  // clear a sticky launch error of this thread
  const int code = (e == cudaErrorMemoryAllocation) ? CPETGB_ENOMEM : CPETGB_ECUDA;
  return fail(code, "%s: %s", what, cudaGetErrorString(e));
}

#define CK(expr, what)                          \
  do {                                          \
    cudaError_t e_ = (expr);                    \
    if (e_ != cudaSuccess) return cuda_fail(e_, what); \
  } while (0)

// Pinned staging buffers of the float32 host calls: kStagingBuffers of kStagingBytes
// for the whole process, allocated together with the first engine, or else on the first
// such call.  Page-locking memory waits for kernels in flight on the device (2.6 s behind
// a busy streamline engine), so that one call may wait for other threads' kernels; none
// after it does.  A call that is larger, or that finds
// no buffer free, copies from and to the caller's pageable arrays.  A buffer belongs
// to one call at a time (any thread, any stream) and goes back after the call has
// waited for its copies.  8 MB hold a call of 51^3 points and 100,000 charges.
constexpr int kStagingBuffers = 2;
constexpr size_t kStagingBytes = size_t(8) << 20;
struct StagingPool {
  std::mutex mu;
  void* buf[kStagingBuffers] = {};
  bool busy[kStagingBuffers] = {};
  bool made = false;
  void make() {  // (mu held)
    if (made) return;
    made = true;
    for (void*& b : buf)
      if (cudaHostAlloc(&b, kStagingBytes, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        b = nullptr;
      }
  }
};
StagingPool& staging_pool() {
  static StagingPool* pool = new StagingPool();  // never destroyed: calls may outlive static destruction
  return *pool;
}

struct Staging {
  void* p = nullptr;
  int index = -1;
  cudaStream_t stream;
  bool waited = false;  // set once no copy to or from the buffer is in flight
  Staging(size_t need, cudaStream_t s) : stream(s) {
    if (need > kStagingBytes) return;
    StagingPool& pool = staging_pool();
    std::lock_guard<std::mutex> lock(pool.mu);
    pool.make();
    for (int i = 0; i < kStagingBuffers && !p; ++i)
      if (pool.buf[i] && !pool.busy[i]) {
        pool.busy[i] = true;
        p = pool.buf[i];
        index = i;
      }
  }
  ~Staging() {
    if (!p) return;
    if (!waited) cudaStreamSynchronize(stream);
    StagingPool& pool = staging_pool();
    std::lock_guard<std::mutex> lock(pool.mu);
    pool.busy[index] = false;
  }
  Staging(const Staging&) = delete;
  Staging& operator=(const Staging&) = delete;
};

Ctx* context(int* rc) {
  int dev = -1, count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count <= 0) {
    cudaGetLastError();
    *rc = fail(CPETGB_ENODEV, "no CUDA device available");
    return nullptr;
  }
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    *rc = fail(CPETGB_ENODEV, "cannot query the current CUDA device");
    return nullptr;
  }
  Ctx& c = g_ctx[dev];
  std::lock_guard<std::mutex> lock(g_mu);
  if (!c.ready) {
    cudaError_t e = cudaDeviceGetAttribute(&c.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&c.status, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(c.status, 0, sizeof(int));
    if (e == cudaSuccess) {
      // Keep freed scratch in the device's stream-ordered pool.
      cudaMemPool_t pool;
      if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        uint64_t keep = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
      }
    }
    if (e != cudaSuccess) {
      *rc = cuda_fail(e, "device context setup");
      return nullptr;
    }
    c.ready = true;
  }
  *rc = CPETGB_OK;
  return &c;
}

// Stream-ordered scratch, released (to the pool) on the same stream.
struct Scratch {
  cudaStream_t s;
  std::vector<void*> ptrs;
  unsigned char* block = nullptr;  // what is left of the last reserve()
  size_t left = 0;
  explicit Scratch(cudaStream_t st) : s(st) {}
  ~Scratch() {
    for (void* p : ptrs) cudaFreeAsync(p, s);
  }
  static size_t bytes_of(size_t bytes) { return (std::max<size_t>(bytes, 1) + 255) / 256 * 256; }
  // One allocation for the get() calls that follow, up to `bytes` of bytes_of() sums
  // (an allocation and its release cost a call about 1.5 us).
  cudaError_t reserve(size_t bytes) {
    void* v = nullptr;
    const cudaError_t e = cudaMallocAsync(&v, bytes_of(bytes), s);
    if (e != cudaSuccess) return e;
    ptrs.push_back(v);
    block = static_cast<unsigned char*>(v);
    left = bytes_of(bytes);
    return e;
  }
  template <typename T>
  cudaError_t get(T** p, size_t count) {
    *p = nullptr;
    const size_t need = bytes_of(count * sizeof(T));
    if (need > left) {
      void* v = nullptr;
      const cudaError_t e = cudaMallocAsync(&v, need, s);
      if (e != cudaSuccess) return e;
      ptrs.push_back(v);
      *p = static_cast<T*>(v);
      return e;
    }
    *p = reinterpret_cast<T*>(block);
    block += need;
    left -= need;
    return cudaSuccess;
  }
};

template <typename T>
cudaError_t h2d(T** dst, Scratch& S, const T* src, size_t count) {
  cudaError_t e = S.get(dst, count);
  if (e == cudaSuccess && count)
    e = cudaMemcpyAsync(*dst, src, count * sizeof(T), cudaMemcpyHostToDevice, S.s);
  return e;
}

// A table of the call's own.  Where the call is recorded into a caller's CUDA graph the
// copy is a node that reads its source at every replay, long after the call has freed its
// table, so the graph gets a copy of the table to keep.
template <typename T>
cudaError_t h2d_table(T** dst, Scratch& S, const T* src, size_t count) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamGetCaptureInfo(S.s, &status, nullptr, &graph, nullptr, nullptr, nullptr);
  if (e != cudaSuccess) return e;
  if (status != cudaStreamCaptureStatusActive || count == 0) return h2d(dst, S, src, count);
  T* kept = static_cast<T*>(std::malloc(count * sizeof(T)));
  if (!kept) return cudaErrorMemoryAllocation;
  std::memcpy(kept, src, count * sizeof(T));
  cudaUserObject_t owner;
  e = cudaUserObjectCreate(&owner, kept, [](void* p) { std::free(p); }, 1, cudaUserObjectNoDestructorSync);
  if (e != cudaSuccess) {
    std::free(kept);
    return e;
  }
  e = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(owner, 1);
    return e;
  }
  return h2d(dst, S, static_cast<const T*>(kept), count);
}

// Hand-over records (cpetgb_set_hand_over_records).
thread_local bool g_hand_over = true;

// Allocates hand-over records by alloc(), without which a streamline launch runs too
// (its lines end where they started, in one round): no memory for them is no error.
template <typename Alloc>
cudaError_t left_or_none(Alloc alloc, TopoState** left, int* rounds) {
  const cudaError_t e = g_hand_over ? alloc() : cudaErrorMemoryAllocation;
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  *left = nullptr;
  *rounds = 1;
  return cudaSuccess;
}

// Converts a status word read from the device into a return code (and clears it there).
int status_code(Ctx* c, int st) {
  if (st != kDevOk) {
    cudaMemset(c->status, 0, sizeof(int));
    if (st == kDevWaitTimeout)
      return fail(CPETGB_ETIMEOUT, "a device-side wait exceeded its limit");
    if (st == kDevBadArgument)
      return fail(CPETGB_ERANGE, "histogram range is not finite or is inverted");
    if (st == kDevBadCap)
      return fail(CPETGB_EINVAL, "a streamline step cap exceeds %d", kMaxLineCap);
    return fail(CPETGB_ECUDA, "device status %d", st);
  }
  return CPETGB_OK;
}

// Waits for the stream and converts the device status word into a return code.
int finish(Ctx* c, cudaStream_t s) {
  CK(cudaStreamSynchronize(s), "stream synchronize");
  int st = 0;
  CK(cudaMemcpy(&st, c->status, sizeof(int), cudaMemcpyDeviceToHost), "status read");
  return status_code(c, st);
}

bool valid_prec(int p) { return p == CPETGB_FP64 || p == CPETGB_FP32C; }
bool valid_mem(int m) { return m == CPETGB_HOST || m == CPETGB_DEVICE; }
size_t packed_size(int prec) { return prec == CPETGB_FP32C ? 16 : 32; }  // streamline layouts
constexpr size_t kGridRecord = 32;  // grid layouts: Charge64 or the duplicated FP32C record

// ---------------------------------------------------------------------------
// Autotuner table: (operation, precision, class, size bucket) -> variant.
// Filled by pycpet_gb300.autotune (timed candidates), read at every launch.
// ---------------------------------------------------------------------------
std::mutex g_tune_mu;
std::map<int, int> g_tune;

constexpr int kOpGrid = 0, kOpTopo = 1;
// points per thread {4, 8} x work items per SM: variants 0-9 {4, 8, 16, 32, 64},
// 10-13 {128, 256} (numbered after the first ten so saved tables keep their meaning)
constexpr int kGridVariants = 14;
constexpr int kTopoVariants = 2;  // line slots per warp {4, 2}

int size_bucket(double v, double base) {
  if (!(v > base)) return 0;
  const int b = static_cast<int>(std::floor(std::log(v / base) / std::log(4.0)));
  return std::min(std::max(b, 0), 15);
}

int tune_key(int op, int prec, int cls, double size) {
  const int b = op == kOpGrid ? size_bucket(size, 1e6) : size_bucket(size, 1e3);
  return (op << 12) | (prec << 8) | ((cls & 15) << 4) | b;
}

int tune_lookup(int key) {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  auto it = g_tune.find(key);
  return it == g_tune.end() ? -1 : it->second;
}

// The variant for a launch: the entry of its own size bucket, else that of the
// nearest tuned bucket of the same (operation, precision, class), the smaller
// one on a tie; -1 when nothing of that class is tuned.
int tune_choose(int key) {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  auto it = g_tune.find(key);
  if (it != g_tune.end()) return it->second;
  const int b = key & 15;
  for (int d = 1; d < 16; ++d) {
    for (int nb : {b - d, b + d}) {
      if (nb < 0 || nb > 15) continue;
      auto jt = g_tune.find((key & ~15) | nb);
      if (jt != g_tune.end()) return jt->second;
    }
  }
  return -1;
}

double grid_pair_evals(int n_frames, const int64_t* desc) {
  double total = 0.0;
  for (int f = 0; f < n_frames; ++f) total += double(desc[4 * f + 1]) * double(desc[4 * f + 3]);
  return total;
}

// ---------------------------------------------------------------------------
// Grid work decomposition: the frame table of a launch (kernels.cuh).
// ---------------------------------------------------------------------------
struct GridTable {
  std::vector<GridFrame> frames;
  int64_t n_items = 0, n_tiles = 0, n_prep = 0, few_items = 0, n_slots = 0;
};

int plan_grid(int prec, int n_frames, const int64_t* desc, int sms, int ppt, int items_per_sm, GridTable& t) {
  const int64_t tile = int64_t(kGridThreads) * ppt;
  // A CTA's time is proportional to its charge count: each frame's charges are
  // split so that about items_per_sm items of equal cost fall on each SM.  The
  // chunks decide how the sums are grouped, so they depend on the frame sizes
  // alone.
  auto full_tiles = [&](int64_t P) { return (P + tile - 1) / tile; };
  double total = 0.0;
  for (int f = 0; f < n_frames; ++f)
    total += double(full_tiles(desc[4 * f + 3])) * double(tile) * double(desc[4 * f + 1]);
  const double target = std::max(1.0, total / (double(std::max(sms, 1)) * items_per_sm));
  const bool mesh =
      grid_pair_evals(n_frames, desc) >= (prec == CPETGB_FP64 ? kGridMeshPairsFp64 : kGridMeshPairsFp32);
  // Is a frame looked at for a mesh?  Not when columns may need a tile more and such
  // spare tiles are a sixth of the launch's tiles or above: mesh or not, their CTAs fall
  // on the same SMs again and again (tiles side by side, an even number of SMs) and cost
  // the launch more than columns save.  Potential, without a look and with one: 100 frames
  // of 512 points x 1,000 charges 28 and 44 us, of 11^3 x 1,000 52 and 60, one of 11^3 x
  // 40,000 43 and 50; 64 of 16^3 x 4,000, eight tiles and one, 269 and 255.  (Splits side
  // by side instead spread them, but 24 frames' fields took 2.19 ms instead of 2.13.)
  const int64_t few = prec == CPETGB_FP64 ? kGridFewPoints : kGridFewPointsFp32;
  auto worth = [&](int64_t n, int64_t P) {
    return mesh && P > few && n >= (prec == CPETGB_FP64 ? kGridMeshChargesFp64 : kGridMeshChargesFp32);
  };
  auto column_tiles = [&](int64_t P) { return ((P + ppt - 1) / ppt + 64 + kGridThreads - 1) / kGridThreads; };
  int64_t tiles = 0, spare = 0;
  for (int f = 0; f < n_frames; ++f) {
    const int64_t n = desc[4 * f + 1], P = desc[4 * f + 3];
    if (P > few) tiles += full_tiles(P);
    if (worth(n, P)) spare += column_tiles(P) - full_tiles(P);
  }
  auto looks = [&](int64_t n, int64_t P) {
    return worth(n, P) && (6 * spare < tiles || column_tiles(P) == full_tiles(P));
  };
  t.frames.resize(size_t(n_frames));
  for (int f = 0; f < n_frames; ++f) {
    const int64_t n = desc[4 * f + 1], P = desc[4 * f + 3];
    GridFrame& fr = t.frames[f];
    fr = GridFrame{};
    fr.charge_off = desc[4 * f];
    fr.point_off = desc[4 * f + 2];
    fr.n_charges = static_cast<int32_t>(n);
    fr.n_points = static_cast<int32_t>(P);
    fr.few = P > 0 && P <= few;
    int64_t split = 1;
    if (n > 0) {
      split = static_cast<int64_t>(std::ceil(double(tile) * double(n) / target));
      // FP32C: at least 256 charges each.  FP64 is so much slower that an uneven
      // number of items per SM costs more than short chunks: 9,261 points x 5,000
      // charges, 361 items of 264 charges 1,390 us, 1,216 of 79 1,160.
      const int64_t least = prec == CPETGB_FP64 && !fr.few ? 32 : 256;
      split = std::max<int64_t>(1, std::min<int64_t>(split, std::max<int64_t>(1, n / least)));
    }
    const int64_t chunk = n > 0 ? (n + split - 1) / split : 0;
    if (n > 0) split = (n + chunk - 1) / chunk;
    fr.chunk = static_cast<int32_t>(chunk);
    fr.n_split = static_cast<int32_t>(split);
    // (a mesh's columns and its other points are rounded up to warps separately)
    fr.n_tiles = P == 0 ? 0 : (fr.few ? 1 : static_cast<int32_t>(looks(n, P) ? column_tiles(P) : full_tiles(P)));
  }
  // few-points frames first; the others longest chunk first, so the last wave
  // holds the shortest items
  std::stable_sort(t.frames.begin(), t.frames.end(), [](const GridFrame& a, const GridFrame& b) {
    return a.few != b.few ? a.few > b.few : a.chunk > b.chunk;
  });
  for (GridFrame& fr : t.frames) {
    const int64_t items = int64_t(fr.n_tiles) * fr.n_split;
    fr.item_base = static_cast<int32_t>(t.n_items);
    fr.tile_base = static_cast<int32_t>(t.n_tiles);
    fr.prep_base = static_cast<int32_t>(t.n_prep);
    fr.slot_base = fr.n_split > 1 ? static_cast<int32_t>(t.n_slots) : -1;
    t.n_items += items;
    t.n_tiles += fr.n_tiles;
    if (fr.n_split > 1) t.n_slots += items;
    if (fr.few) {
      t.few_items += items;
    } else if (looks(fr.n_charges, fr.n_points)) {
      t.n_prep += (int64_t(fr.n_points) + kGridPrepPoints - 1) / kGridPrepPoints;
    }
    if (t.n_items > INT_MAX || t.n_tiles * ppt > INT_MAX)
      return fail(CPETGB_EINVAL, "launch too large (%lld work items)", (long long)t.n_items);
  }
  return CPETGB_OK;
}

// Entries the refinement list may need: every point of every frame (frames
// may share point ranges, so this is the sum, not the extent).
int64_t refine_list_len(int n_frames, const int64_t* desc) {
  int64_t n = 0;
  for (int f = 0; f < n_frames; ++f) n += desc[4 * f + 3];
  return std::max<int64_t>(n, 1);
}

int64_t max_frame_points(int n_frames, const int64_t* desc) {
  int64_t m = 0;
  for (int f = 0; f < n_frames; ++f) m = std::max(m, desc[4 * f + 3]);
  return m;
}

// Everything of a launch that does not depend on its buffers.
GridLaunch grid_launch(int kind, int prec, int clamp, int ppt, int n_frames, const int64_t* desc,
                       const GridTable& t, int64_t tot_ch, const Ctx* c) {
  GridLaunch g{};
  g.kind = kind;
  g.prec = prec;
  g.clamp = clamp ? 1 : 0;
  g.ppt = ppt;
  g.n_frames = n_frames;
  if (n_frames == 1) g.one = t.frames[0];
  g.n_items = static_cast<int>(t.n_items);
  g.n_tiles = static_cast<int>(t.n_tiles);
  g.n_prep = static_cast<int>(t.n_prep);
  g.few_items = static_cast<int>(t.few_items);
  g.n_charges = tot_ch;
  g.max_points = static_cast<int>(max_frame_points(n_frames, desc));
  g.status = c->status;
  g.num_sms = c->sms;
  // A frame of one or two points never has a point below tau x its lower
  // median, so launches of such frames only (point fields) skip the pass.
  const double tau = g_refine_tau.load();
  const bool refine =
      kind == CPETGB_FIELD && prec == CPETGB_FP32C && tau > 0.0 && tot_ch > 0 && g.max_points >= 3;
  g.tau = refine ? tau : 0.0;
  return g;
}

// A grid launch's plan, and its scratch (from S, released after it on the stream).
struct GridWork {
  GridTable plan;
  GridLaunch g{};
  int ppt = 4;
  bool point = false;  // one kernel, no scratch
  size_t n_list = 0;
  size_t zero_ints() const { return grid_zero_ints(g.n_frames, g.tau > 0.0); }
  size_t packed_bytes() const { return size_t(std::max<int64_t>(g.n_charges, 1)) * kGridRecord; }
  size_t partial_doubles() const { return size_t(plan.n_slots) * grid_slot_doubles(g.kind, ppt); }
  size_t scratch_bytes() const {
    if (point) return 0;
    size_t b = Scratch::bytes_of(packed_bytes()) + Scratch::bytes_of(zero_ints() * sizeof(int));
    if (g.n_frames != 1) b += Scratch::bytes_of(plan.frames.size() * sizeof(GridFrame));
    if (plan.n_slots) b += Scratch::bytes_of(partial_doubles() * sizeof(double));
    if (g.tau > 0.0)
      b += Scratch::bytes_of(n_list * sizeof(int64_t)) + Scratch::bytes_of(size_t(g.n_charges) * 32);
    return b;
  }
  int prepare(int kind, int prec, int clamp, int n_frames, const int64_t* desc, int64_t tot_ch, const Ctx* c) {
    int ips = 8;
    tuned_grid_shape(prec, kind, grid_pair_evals(n_frames, desc), &ppt, &ips);
    const int rc = plan_grid(prec, n_frames, desc, c->sms, ppt, ips, plan);
    if (rc != CPETGB_OK) return rc;
    g = grid_launch(kind, prec, clamp, ppt, n_frames, desc, plan, tot_ch, c);
    point = grid_point_fits(g);
    n_list = g.tau > 0.0 ? size_t(refine_list_len(n_frames, desc)) * 2 : 0;
    return CPETGB_OK;
  }
  int allocate(Scratch& S) {
    if (point) return CPETGB_OK;
    unsigned char* packed = nullptr;
    CK(S.get(&packed, packed_bytes()), "alloc packed charges");
    if (reinterpret_cast<uintptr_t>(packed) % 16 != 0)  // bulk async copies need 16-byte sources
      return fail(CPETGB_ECUDA, "scratch allocation is not 16-byte aligned");
    g.packed = packed;
    if (g.n_frames != 1) {
      GridFrame* d_frames = nullptr;
      CK(h2d_table(&d_frames, S, static_cast<const GridFrame*>(plan.frames.data()), plan.frames.size()),
         "copy frame table");
      g.frames = d_frames;
    }
    CK(S.get(&g.zeroed, zero_ints()), "alloc counters");
    if (plan.n_slots) CK(S.get(&g.partial, partial_doubles()), "alloc partial sums");
    if (g.tau > 0.0) {
      unsigned char* dfq = nullptr;
      CK(S.get(&g.list, n_list), "alloc refinement list");
      CK(S.get(&dfq, size_t(g.n_charges) * 32), "alloc double-float charges");
      g.dfq = dfq;
    }
    return CPETGB_OK;
  }
  int launch(const double* pts, const double* x, const double* q, double* out, cudaStream_t s, bool cleared) {
    g.points = pts;
    g.x = x;
    g.q = q;
    g.out = out;
    if (point)
      CK(launch_grid_point(g, s), "point kernel launch");
    else
      CK(launch_grid(g, s, cleared), "grid launch");
    return CPETGB_OK;
  }
};

int grid_batch_impl(int kind, int prec, int mem, int clamp, int n_frames, const int64_t* desc,
                    const double* pts, const double* x, const double* q, double* out,
                    void* stream) {
  if (kind != CPETGB_FIELD && kind != CPETGB_ESP) return fail(CPETGB_EINVAL, "bad grid kind %d", kind);
  if (!valid_prec(prec)) return fail(CPETGB_EINVAL, "bad precision %d", prec);
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (n_frames < 0 || (n_frames > 0 && !desc)) return fail(CPETGB_EINVAL, "bad frame table");
  int64_t tot_pts = 0, tot_ch = 0;
  for (int f = 0; f < n_frames; ++f) {
    const int64_t co = desc[4 * f], n = desc[4 * f + 1], po = desc[4 * f + 2], P = desc[4 * f + 3];
    if (co < 0 || n < 0 || po < 0 || P < 0 || n > INT_MAX || P > INT_MAX)
      return fail(CPETGB_EINVAL, "frame %d: negative or oversized offset/count", f);
    tot_pts = std::max(tot_pts, po + P);
    tot_ch = std::max(tot_ch, co + n);
  }
  if (tot_pts == 0) return CPETGB_OK;
  if (!pts || !out) return fail(CPETGB_EINVAL, "points/output pointer is NULL");
  if (tot_ch > 0 && (!x || !q)) return fail(CPETGB_EINVAL, "charge pointer is NULL");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mem == CPETGB_HOST && !s) s = c->stream;
  const int NC = kind == CPETGB_FIELD ? 3 : 1;

  GridWork w;
  rc = w.prepare(kind, prec, clamp, n_frames, desc, tot_ch, c);
  if (rc != CPETGB_OK) return rc;
  Scratch S(s);
  if (!w.point) CK(S.reserve(w.scratch_bytes()), "alloc scratch");
  rc = w.allocate(S);
  if (rc != CPETGB_OK) return rc;
  const double *dp = pts, *dx = x, *dq = q;
  double* dout = out;
  if (mem == CPETGB_HOST) {
    CK(h2d(const_cast<double**>(&dp), S, pts, size_t(tot_pts) * 3), "copy points");
    if (tot_ch) {
      CK(h2d(const_cast<double**>(&dx), S, x, size_t(tot_ch) * 3), "copy charge positions");
      CK(h2d(const_cast<double**>(&dq), S, q, size_t(tot_ch)), "copy charges");
    }
    CK(S.get(&dout, size_t(tot_pts) * NC), "alloc output");
  }
  rc = w.launch(dp, dx, dq, dout, s, false);
  if (rc != CPETGB_OK) return rc;
  if (mem == CPETGB_HOST) {
    CK(cudaMemcpyAsync(out, dout, size_t(tot_pts) * NC * sizeof(double), cudaMemcpyDeviceToHost, s),
       "copy output");
    return finish(c, s);
  }
  return CPETGB_OK;
}

// Field or potential from float32 host arrays to float32 / float16 host rows
// (RowFormat): one copy in, one out, the conversions on the device.
int grid_f32_impl(int kind, int prec, int clamp, int P, int N, const float* pts, const float* x,
                  const float* q, int fmt, void* rows) {
  if (P < 0 || N < 0) return fail(CPETGB_EINVAL, "negative size");
  if (P == 0) return CPETGB_OK;
  if (!valid_prec(prec)) return fail(CPETGB_EINVAL, "bad precision %d", prec);
  if (!pts || !rows || (N && (!x || !q))) return fail(CPETGB_EINVAL, "NULL pointer");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = c->stream;
  const size_t np = size_t(P) * 3, nx = size_t(N) * 3, nq = size_t(N), n_in = np + nx + nq;
  const size_t n_val = size_t(P) * (kind == CPETGB_FIELD ? 3 : 1);
  const size_t row_bytes =
      fmt == kRowsField ? size_t(P) * 24 : (fmt == kRowsEspHalf ? size_t(P) * 8 : n_val * sizeof(float));
  const size_t out_bytes = ((row_bytes + 15) & ~size_t(15)) + 16;  // the status word behind the rows
  const size_t in_bytes = (n_in * sizeof(float) + 255) & ~size_t(255);
  const int64_t desc[4] = {0, N, 0, P};
  GridWork w;
  rc = w.prepare(kind, prec, clamp, 1, desc, N, c);
  if (rc != CPETGB_OK) return rc;
  Staging host(in_bytes + out_bytes, s);
  Scratch S(s);
  CK(S.reserve(w.scratch_bytes() + Scratch::bytes_of(n_in * sizeof(float)) + Scratch::bytes_of(n_in * sizeof(double)) +
               Scratch::bytes_of(n_val * sizeof(double)) + Scratch::bytes_of(out_bytes)),
     "alloc scratch");
  float* d_in = nullptr;
  double *d64 = nullptr, *d_val = nullptr;
  unsigned char* d_rows = nullptr;
  CK(S.get(&d_in, n_in), "alloc inputs");
  CK(S.get(&d64, n_in), "alloc inputs");
  CK(S.get(&d_val, n_val), "alloc output");
  CK(S.get(&d_rows, out_bytes), "alloc rows");
  rc = w.allocate(S);
  if (rc != CPETGB_OK) return rc;
  if (host.p) {
    float* h = static_cast<float*>(host.p);
    std::memcpy(h, pts, np * sizeof(float));
    if (N) {
      std::memcpy(h + np, x, nx * sizeof(float));
      std::memcpy(h + np + nx, q, nq * sizeof(float));
    }
    CK(cudaMemcpyAsync(d_in, h, n_in * sizeof(float), cudaMemcpyHostToDevice, s), "copy inputs");
  } else {
    CK(cudaMemcpyAsync(d_in, pts, np * sizeof(float), cudaMemcpyHostToDevice, s), "copy points");
    if (N) {
      CK(cudaMemcpyAsync(d_in + np, x, nx * sizeof(float), cudaMemcpyHostToDevice, s), "copy charge positions");
      CK(cudaMemcpyAsync(d_in + np + nx, q, nq * sizeof(float), cudaMemcpyHostToDevice, s), "copy charges");
    }
  }
  CK(launch_widen(static_cast<int64_t>(n_in), d_in, d64, w.g.zeroed,
                  w.point ? 0 : static_cast<int64_t>(w.zero_ints()), s),
     "widen inputs");
  rc = w.launch(d64, d64 + np, d64 + np + nx, d_val, s, true);
  if (rc != CPETGB_OK) return rc;
  int* tail = reinterpret_cast<int*>(d_rows + out_bytes - 16);
  CK(launch_rows(fmt, fmt == kRowsPlain ? static_cast<int64_t>(n_val) : P, d_in, d_val, d_rows, c->status, tail, s),
     "row conversion");
  int st = 0;
  if (host.p) {
    unsigned char* h = static_cast<unsigned char*>(host.p) + in_bytes;
    CK(cudaMemcpyAsync(h, d_rows, out_bytes, cudaMemcpyDeviceToHost, s), "copy rows");
    CK(cudaStreamSynchronize(s), "stream synchronize");
    host.waited = true;
    std::memcpy(rows, h, row_bytes);
    std::memcpy(&st, h + out_bytes - 16, sizeof(int));
  } else {
    CK(cudaMemcpyAsync(rows, d_rows, row_bytes, cudaMemcpyDeviceToHost, s), "copy rows");
    CK(cudaMemcpyAsync(&st, tail, sizeof(int), cudaMemcpyDeviceToHost, s), "status read");
    CK(cudaStreamSynchronize(s), "stream synchronize");
  }
  return status_code(c, st);
}

// source = kCharges: q[N] charges; kDipoles: q is mu[N][3], the dipole moments.
int topo_impl(int prec, int mem, int L, int N, const double* starts, const int32_t* n_iter,
              double step, const double* half, const double* x, const double* q, double* result,
              double* ends, int32_t* steps, void* stream, int source = kCharges) {
  if (!valid_prec(prec)) return fail(CPETGB_EINVAL, "bad precision %d", prec);
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (L < 0 || N < 0) return fail(CPETGB_EINVAL, "negative line or charge count");
  if (!half) return fail(CPETGB_EINVAL, "half_dims is NULL");
  for (int k = 0; k < 3; ++k)
    if (!std::isfinite(half[k]) || half[k] < 0)
      return fail(CPETGB_EINVAL, "half_dims[%d] must be finite and >= 0", k);
  if (!std::isfinite(step)) return fail(CPETGB_EINVAL, "step must be finite");
  if (L == 0) return CPETGB_OK;
  if (!starts || !n_iter || !result) return fail(CPETGB_EINVAL, "line pointer is NULL");
  if (N > 0 && (!x || !q)) return fail(CPETGB_EINVAL, "charge pointer is NULL");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mem == CPETGB_HOST && !s) s = c->stream;

  Scratch S(s);
  const double *ds = starts, *dx = x, *dq = q;
  const int32_t* dn = n_iter;
  double *dres = result, *dends = ends;
  int32_t* dsteps = steps;
  if (mem == CPETGB_HOST) {
    CK(h2d(const_cast<double**>(&ds), S, starts, size_t(L) * 3), "copy starts");
    CK(h2d(const_cast<int32_t**>(&dn), S, n_iter, size_t(L)), "copy n_iter");
    if (N) {
      CK(h2d(const_cast<double**>(&dx), S, x, size_t(N) * 3), "copy charge positions");
      CK(h2d(const_cast<double**>(&dq), S, q, size_t(N) * (source == kDipoles ? 3 : 1)),
         "copy charges");
    }
    CK(S.get(&dres, size_t(L) * 2), "alloc result");
    if (ends) CK(S.get(&dends, size_t(L) * 3), "alloc ends");
    if (steps) CK(S.get(&dsteps, size_t(L)), "alloc steps");
  }
  const int pad = topo_charge_pad(prec);
  const int64_t n_pad = ((std::max(N, 1) + int64_t(pad) - 1) / pad) * pad;
  unsigned char* packed = nullptr;
  int* queue = nullptr;  // the queue counter and, per round, the count of lines handed over
  TopoState* left = nullptr;
  const double diag_steps = topo_diag_steps(half, step);
  int rounds = topo_team_rounds(c->sms, L, diag_steps);
  const bool whole = topo_resident_count(prec, source, static_cast<int>(n_pad)) == n_pad;
  const bool fresh = topo_fresh(prec, source, whole, double(n_pad), L, c->sms, true);
  const bool records = fresh ? rounds > 1 : topo_hands_over(prec, source, whole, static_cast<int>(n_pad), diag_steps);
  const int left_cap = records ? topo_left_capacity(c->sms, L, fresh) : 0;
  CK(S.get(&packed, size_t(n_pad) * topo_source_bytes(prec, source)), "alloc packed charges");
  CK(S.get(&queue, size_t(1 + rounds)), "alloc queue");
  CK(cudaMemsetAsync(queue, 0, (1 + rounds) * sizeof(int), s), "zero queue");
  if (left_cap)
    CK(left_or_none([&] { return S.get(&left, 2 * size_t(left_cap)); }, &left, &rounds), "alloc hand-over records");
  if (reinterpret_cast<uintptr_t>(packed) % 16 != 0)
    return fail(CPETGB_ECUDA, "scratch allocation is not 16-byte aligned");
  if (source == kDipoles)
    CK(launch_pack_dipoles(prec, N, n_pad, dx, dq, packed, s), "pack dipoles");
  else
    CK(launch_pack_topo(prec, N, n_pad, dx, dq, packed, s), "pack charges");
  TopoParams p;
  p.source = source;
  p.n_lines = L;
  p.n_charges = N;
  p.step = step;
  for (int k = 0; k < 3; ++k) p.half[k] = half[k];
  p.starts = ds;
  p.n_iter = dn;
  p.packed = packed;
  p.result = dres;
  p.ends = dends;
  p.steps = dsteps;
  p.queue = queue;
  p.left = left;
  p.left_records = left_cap;
  p.left_count = queue + 1;
  p.rounds = rounds;
  p.fresh = fresh;
  p.status = c->status;
  CK(launch_topo(prec, p, c->sms, s), "topo kernel launch");
  if (mem == CPETGB_HOST) {
    CK(cudaMemcpyAsync(result, dres, size_t(L) * 2 * sizeof(double), cudaMemcpyDeviceToHost, s),
       "copy result");
    if (ends)
      CK(cudaMemcpyAsync(ends, dends, size_t(L) * 3 * sizeof(double), cudaMemcpyDeviceToHost, s),
         "copy ends");
    if (steps)
      CK(cudaMemcpyAsync(steps, dsteps, size_t(L) * sizeof(int32_t), cudaMemcpyDeviceToHost, s),
         "copy steps");
    return finish(c, s);
  }
  return CPETGB_OK;
}

struct TopoTables {
  std::vector<TopoFrame> frames;
  std::vector<int64_t> src;  // per frame {charge offset, charge count} into x/q
  int64_t tot_lines = 0, tot_ch = 0, packed_elems = 0;
  int64_t sum_lines = 0;      // lines of all frames (frames may share ranges)
  double line_sources = 0.0;  // sources of all lines
  int64_t left_records = 0;   // hand-over records of all frames
  int rounds = 1;             // team kernel launches
  bool fresh = false;         // every line in them from its start point
  double diag_steps = 0.0;    // the frames' largest box diagonal in steps
  int max_res = 0, max_team_res = 0, max_pairs = 0;
  bool all_resident = true;  // every frame entirely in shared memory (tuner class 1)
};

// Frame table of a streamline launch: padded sizes, packed offsets (FP32C
// frames occupy n_pad float4 -- the pair block A then B --, FP64 frames n_pad
// Charge64), how many charges of each frame stay resident in shared memory, and
// each frame's hand-over records (at most kMaxLeft in all; frames beyond that
// have none and their lines end where they started).

int build_topo_tables(int prec, int F, const int64_t* desc, const double* params, TopoTables& t) {
  if (!valid_prec(prec)) return fail(CPETGB_EINVAL, "bad precision %d", prec);
  if (F < 0 || (F > 0 && (!desc || !params))) return fail(CPETGB_EINVAL, "bad frame table");
  const int pad = topo_charge_pad(prec);
  t.frames.assign(F, TopoFrame{});
  t.src.assign(2 * size_t(F), 0);
  for (int f = 0; f < F; ++f) {
    const int64_t co = desc[4 * f], n = desc[4 * f + 1], lo = desc[4 * f + 2], L = desc[4 * f + 3];
    if (co < 0 || n < 0 || lo < 0 || L < 0 || n > INT_MAX / 2 || L > INT_MAX)
      return fail(CPETGB_EINVAL, "frame %d: negative or oversized offset/count", f);
    const double* pr = params + 4 * f;
    if (!std::isfinite(pr[0])) return fail(CPETGB_EINVAL, "frame %d: step must be finite", f);
    for (int k = 1; k < 4; ++k)
      if (!std::isfinite(pr[k]) || pr[k] < 0)
        return fail(CPETGB_EINVAL, "frame %d: half-widths must be finite and >= 0", f);
    TopoFrame& fr = t.frames[f];
    fr.n_pad = static_cast<int32_t>(((std::max<int64_t>(n, 1) + pad - 1) / pad) * pad);
    fr.packed_off = t.packed_elems;
    t.packed_elems += fr.n_pad;
    fr.line_off = lo;
    fr.n_lines = static_cast<int32_t>(L);
    fr.resident = topo_resident_count(prec, kCharges, fr.n_pad);
    fr.team_resident = topo_team_resident(prec, kCharges, fr.n_pad);
    t.max_team_res = std::max(t.max_team_res, int(fr.team_resident));
    t.sum_lines += L;
    t.line_sources += double(L) * double(fr.n_pad);
    t.diag_steps = std::max(t.diag_steps, topo_diag_steps(pr + 1, pr[0]));
    fr.step = pr[0];
    for (int k = 0; k < 3; ++k) fr.half[k] = pr[1 + k];
    t.max_res = std::max(t.max_res, int(fr.resident));
    if (fr.resident < fr.n_pad) t.all_resident = false;
    t.max_pairs = std::max(t.max_pairs, int(fr.n_pad));
    t.src[2 * f] = co;
    t.src[2 * f + 1] = n;
    t.tot_lines = std::max(t.tot_lines, lo + L);
    t.tot_ch = std::max(t.tot_ch, co + n);
  }
  if (t.tot_lines > INT_MAX) return fail(CPETGB_EINVAL, "too many lines");
  return CPETGB_OK;
}

void plan_hand_over(int prec, int sms, TopoTables& t) {
  t.rounds = topo_team_rounds(sms, t.sum_lines, t.diag_steps);
  t.fresh = topo_fresh(prec, kCharges, t.all_resident, t.line_sources / double(std::max<int64_t>(t.sum_lines, 1)),
                       t.sum_lines, sms, true);
  for (TopoFrame& fr : t.frames) {
    const bool records = t.fresh ? t.rounds > 1
                                 : topo_hands_over(prec, kCharges, fr.resident == fr.n_pad, fr.n_pad,
                                                   topo_diag_steps(fr.half, fr.step));
    const int64_t cap = records ? topo_left_capacity(sms, fr.n_lines, t.fresh) : 0;
    fr.left_off = static_cast<int32_t>(t.left_records);
    fr.left_cap = t.left_records + cap <= kMaxLeft ? static_cast<int32_t>(cap) : 0;
    t.left_records += fr.left_cap;
  }
}

int topo_batch_impl(int prec, int mem, int F, const int64_t* desc, const double* params,
                    const double* starts, const int32_t* n_iter, const double* x, const double* q,
                    double* result, double* ends, int32_t* steps, void* stream) {
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  TopoTables t;
  int rc0 = build_topo_tables(prec, F, desc, params, t);
  if (rc0 != CPETGB_OK) return rc0;
  std::vector<TopoFrame>& frames = t.frames;
  std::vector<int64_t>& src = t.src;
  const int64_t tot_lines = t.tot_lines, tot_ch = t.tot_ch, packed_elems = t.packed_elems;
  const int max_res = t.max_res, max_pairs = t.max_pairs;
  const bool all_resident = t.all_resident;
  if (tot_lines == 0) return CPETGB_OK;
  if (!starts || !n_iter || !result) return fail(CPETGB_EINVAL, "line pointer is NULL");
  if (tot_ch > 0 && (!x || !q)) return fail(CPETGB_EINVAL, "charge pointer is NULL");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  plan_hand_over(prec, c->sms, t);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mem == CPETGB_HOST && !s) s = c->stream;
  const size_t L = size_t(tot_lines);
  Scratch S(s);
  const double *ds = starts, *dx = x, *dq = q;
  const int32_t* dn = n_iter;
  double *dres = result, *dends = ends;
  int32_t* dsteps = steps;
  if (mem == CPETGB_HOST) {
    CK(h2d(const_cast<double**>(&ds), S, starts, L * 3), "copy starts");
    CK(h2d(const_cast<int32_t**>(&dn), S, n_iter, L), "copy n_iter");
    if (tot_ch) {
      CK(h2d(const_cast<double**>(&dx), S, x, size_t(tot_ch) * 3), "copy charge positions");
      CK(h2d(const_cast<double**>(&dq), S, q, size_t(tot_ch)), "copy charges");
    }
    CK(S.get(&dres, L * 2), "alloc result");
    if (ends) CK(S.get(&dends, L * 3), "alloc ends");
    if (steps) CK(S.get(&dsteps, L), "alloc steps");
  }
  unsigned char* packed = nullptr;
  TopoFrame* d_frames = nullptr;
  int64_t* d_src = nullptr;
  int* queues = nullptr;
  CK(S.get(&packed, size_t(std::max<int64_t>(packed_elems, 1)) * packed_size(prec)),
     "alloc packed charges");
  if (reinterpret_cast<uintptr_t>(packed) % 16 != 0)
    return fail(CPETGB_ECUDA, "scratch allocation is not 16-byte aligned");
  CK(h2d_table(&d_frames, S, static_cast<const TopoFrame*>(frames.data()), frames.size()), "copy frame table");
  CK(h2d_table(&d_src, S, static_cast<const int64_t*>(src.data()), src.size()), "copy frame sources");
  TopoState* left = nullptr;
  CK(S.get(&queues, size_t(1 + t.rounds) * F), "alloc queues");
  CK(cudaMemsetAsync(queues, 0, sizeof(int) * size_t(1 + t.rounds) * F, s), "zero queues");
  if (t.left_records)
    CK(left_or_none([&] { return S.get(&left, 2 * size_t(t.left_records)); }, &left, &t.rounds),
       "alloc hand-over records");
  CK(launch_pack_topo_frames(prec, F, d_frames, d_src, dx, dq, packed, max_pairs, s),
     "pack charges");
  TopoParams p{};
  p.n_lines = static_cast<int>(tot_lines);
  p.starts = ds;
  p.n_iter = dn;
  p.packed = packed;
  p.result = dres;
  p.ends = dends;
  p.steps = dsteps;
  p.queue = queues;
  p.left = left;
  p.left_records = t.left_records;
  p.left_count = queues + F;
  p.rounds = t.rounds;
  p.fresh = t.fresh;
  p.status = c->status;
  p.frames = d_frames;
  p.n_frames = F;
  p.max_resident_pad = max_res;
  p.max_team_resident = t.max_team_res;
  p.sum_lines = t.sum_lines;
  p.all_resident = all_resident ? 1 : 0;
  CK(launch_topo_frames(prec, p, c->sms, s), "topo kernel launch");
  if (mem == CPETGB_HOST) {
    CK(cudaMemcpyAsync(result, dres, L * 2 * sizeof(double), cudaMemcpyDeviceToHost, s),
       "copy result");
    if (ends)
      CK(cudaMemcpyAsync(ends, dends, L * 3 * sizeof(double), cudaMemcpyDeviceToHost, s),
         "copy ends");
    if (steps)
      CK(cudaMemcpyAsync(steps, dsteps, L * sizeof(int32_t), cudaMemcpyDeviceToHost, s),
         "copy steps");
    return finish(c, s);
  }
  return CPETGB_OK;
}

int hist_impl(int mem, int L, const double* result, int nb0, int nb1, const double* range,
              uint64_t* counts, double* edges, void* stream) {
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (L < 0 || nb0 < 1 || nb1 < 1 || nb0 + nb1 > 4096)
    return fail(CPETGB_EINVAL, "bad histogram shape (%d lines, %d x %d bins)", L, nb0, nb1);
  if (!range || !counts || (L > 0 && !result)) return fail(CPETGB_EINVAL, "NULL pointer");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mem == CPETGB_HOST && !s) s = c->stream;
  Scratch S(s);
  const double* dv = result;
  unsigned long long* dc = reinterpret_cast<unsigned long long*>(counts);
  double* de = edges;
  const size_t nbins = size_t(nb0) * nb1;
  if (mem == CPETGB_HOST) {
    if (L) CK(h2d(const_cast<double**>(&dv), S, result, size_t(L) * 2), "copy values");
    CK(S.get(&dc, nbins), "alloc counts");
  }
  if (mem == CPETGB_HOST || !edges) CK(S.get(&de, size_t(nb0 + nb1 + 2)), "alloc edges");
  CK(cudaMemsetAsync(dc, 0, nbins * sizeof(unsigned long long), s), "zero counts");
  CK(launch_hist2d(L, dv, nb0, nb1, range, de, dc, c->status, s), "histogram launch");
  if (mem == CPETGB_HOST) {
    CK(cudaMemcpyAsync(counts, dc, nbins * sizeof(uint64_t), cudaMemcpyDeviceToHost, s),
       "copy counts");
    if (edges)
      CK(cudaMemcpyAsync(edges, de, size_t(nb0 + nb1 + 2) * sizeof(double),
                         cudaMemcpyDeviceToHost, s),
         "copy edges");
    return finish(c, s);
  }
  return CPETGB_OK;
}

int hist_sets_impl(int mem, int n_sets, const int64_t* offsets, const double* values, int nb0,
                   int nb1, const double* range, uint64_t* counts, double* hists, void* stream) {
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (n_sets < 0 || nb0 < 1 || nb1 < 1 || nb0 + nb1 > 4096)
    return fail(CPETGB_EINVAL, "bad histogram shape (%d sets, %d x %d bins)", n_sets, nb0, nb1);
  if (n_sets == 0) return CPETGB_OK;
  if (!offsets || !range || (!counts && !hists)) return fail(CPETGB_EINVAL, "NULL pointer");
  if (offsets[0] != 0) return fail(CPETGB_EINVAL, "offsets[0] must be 0");
  int64_t max_set = 0;
  for (int f = 0; f < n_sets; ++f) {
    if (offsets[f + 1] < offsets[f]) return fail(CPETGB_EINVAL, "offsets decrease at set %d", f);
    max_set = std::max(max_set, offsets[f + 1] - offsets[f]);
  }
  const int64_t L = offsets[n_sets];
  if (L > 0 && !values) return fail(CPETGB_EINVAL, "values pointer is NULL");
  for (int k = 0; k < 4; ++k)
    if (!std::isfinite(range[k])) return fail(CPETGB_ERANGE, "histogram range must be finite");
  if (range[0] > range[1] || range[2] > range[3])
    return fail(CPETGB_ERANGE, "histogram range is inverted");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mem == CPETGB_HOST && !s) s = c->stream;
  Scratch S(s);
  const size_t nbins = size_t(nb0) * nb1, total = nbins * size_t(n_sets);
  const double* dv = values;
  unsigned long long* dc = reinterpret_cast<unsigned long long*>(counts);
  double* dh = hists;
  double* de = nullptr;
  int64_t* doff = nullptr;
  if (mem == CPETGB_HOST && L) CK(h2d(const_cast<double**>(&dv), S, values, size_t(L) * 2), "copy values");
  if (mem == CPETGB_HOST || !counts) CK(S.get(&dc, total), "alloc counts");
  if (mem == CPETGB_HOST && hists) CK(S.get(&dh, total), "alloc histograms");
  CK(S.get(&de, size_t(nb0 + nb1 + 2)), "alloc edges");
  CK(h2d_table(&doff, S, offsets, size_t(n_sets) + 1), "copy offsets");
  CK(cudaMemsetAsync(dc, 0, total * sizeof(unsigned long long), s), "zero counts");
  CK(launch_hist2d_sets(n_sets, doff, max_set, dv, nb0, nb1, range, de, dc, hists ? dh : nullptr,
                        c->status, s),
     "histogram launch");
  if (mem == CPETGB_HOST) {
    if (counts)
      CK(cudaMemcpyAsync(counts, dc, total * sizeof(uint64_t), cudaMemcpyDeviceToHost, s),
         "copy counts");
    if (hists)
      CK(cudaMemcpyAsync(hists, dh, total * sizeof(double), cudaMemcpyDeviceToHost, s),
         "copy histograms");
    return finish(c, s);
  }
  return CPETGB_OK;
}

int prepare_frame_impl(int mem, int n, const double* x, const double* q, const int32_t* resid,
                       const int32_t* resnum, const double* center, const double* inv,
                       double radius, const double* half, const double* shift, double* x_out,
                       double* q_out, int* n_out, void* stream) {
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (n < 0) return fail(CPETGB_EINVAL, "negative atom count");
  if (!center || !n_out) return fail(CPETGB_EINVAL, "center / n_out pointer is NULL");
  if (!std::isfinite(radius)) return fail(CPETGB_EINVAL, "radius must be finite (<= 0: no filter)");
  for (int k = 0; k < 3; ++k)
    if (!std::isfinite(center[k]) || (half && !(half[k] >= 0.0)) || (shift && !std::isfinite(shift[k])))
      return fail(CPETGB_EINVAL, "center, box half-widths and shift must be finite (half-widths >= 0)");
  if (inv)
    for (int k = 0; k < 9; ++k)
      if (!std::isfinite(inv[k])) return fail(CPETGB_EINVAL, "inverse basis must be finite");
  *n_out = 0;
  if (n == 0) return CPETGB_OK;
  if (!x || !q || !x_out || !q_out) return fail(CPETGB_EINVAL, "array pointer is NULL");
  if (radius > 0.0 && (!resid || !resnum))
    return fail(CPETGB_EINVAL, "the residue radius filter needs resid and resnum");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!s) s = c->stream;
  Scratch S(s);
  const double *dx = x, *dq = q;
  const int32_t *dr = resid, *dn = resnum;
  double *dxo = x_out, *dqo = q_out;
  if (mem == CPETGB_HOST) {
    CK(h2d(const_cast<double**>(&dx), S, x, size_t(n) * 3), "copy positions");
    CK(h2d(const_cast<double**>(&dq), S, q, size_t(n)), "copy charges");
    if (radius > 0.0) {
      CK(h2d(const_cast<int32_t**>(&dr), S, resid, size_t(n)), "copy resid");
      CK(h2d(const_cast<int32_t**>(&dn), S, resnum, size_t(n)), "copy resnum");
    }
    CK(S.get(&dxo, size_t(n) * 3), "alloc positions");
    CK(S.get(&dqo, size_t(n)), "alloc charges");
  }
  unsigned char* scratch = nullptr;
  int64_t* dcount = nullptr;
  CK(S.get(&scratch, prep_scratch_bytes(n)), "alloc scratch");
  CK(S.get(&dcount, 1), "alloc count");
  CK(launch_prepare_frame(n, dx, dq, dr, dn, center, inv, radius, half, shift, dxo, dqo, scratch,
                          dcount, s),
     "frame preparation");
  int64_t count = 0;
  CK(cudaMemcpyAsync(&count, dcount, sizeof(int64_t), cudaMemcpyDeviceToHost, s), "read count");
  CK(cudaStreamSynchronize(s), "stream synchronize");
  *n_out = static_cast<int>(count);
  if (mem == CPETGB_HOST && count) {
    CK(cudaMemcpyAsync(x_out, dxo, size_t(count) * 3 * sizeof(double), cudaMemcpyDeviceToHost, s),
       "copy positions");
    CK(cudaMemcpyAsync(q_out, dqo, size_t(count) * sizeof(double), cudaMemcpyDeviceToHost, s),
       "copy charges");
    return finish(c, s);
  }
  return CPETGB_OK;
}

int format_text_impl(int fmt, int mem, int64_t n_rows, int n_cols, const float* values, char* text,
                     int64_t capacity, int64_t* length, void* stream) {
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (n_rows < 0 || n_cols < 1) return fail(CPETGB_EINVAL, "need n_rows >= 0 and n_cols >= 1");
  if (!length) return fail(CPETGB_EINVAL, "length pointer is NULL");
  if (n_rows > 0 && !values) return fail(CPETGB_EINVAL, "values pointer is NULL");
  if (n_rows > (int64_t(1) << 40) / n_cols) return fail(CPETGB_EINVAL, "matrix too large");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!s) s = c->stream;
  Scratch S(s);
  const float* dv = values;
  if (mem == CPETGB_HOST && n_rows)
    CK(h2d(const_cast<float**>(&dv), S, values, size_t(n_rows) * n_cols), "copy values");
  int64_t* off = nullptr;
  int64_t* scratch = nullptr;
  CK(S.get(&off, size_t(n_rows) + 1), "alloc offsets");
  CK(S.get(&scratch, size_t(fixed3_scan_scratch(n_rows + 1))), "alloc scan scratch");
  CK(launch_text_offsets(fmt, n_rows, n_cols, dv, off, scratch, s), "length pass");
  int64_t total = 0;
  CK(cudaMemcpyAsync(&total, off + n_rows, sizeof(int64_t), cudaMemcpyDeviceToHost, s), "read length");
  CK(cudaStreamSynchronize(s), "stream synchronize");
  *length = total;
  if (!text) return CPETGB_OK;
  if (capacity < total) return fail(CPETGB_ERANGE, "text buffer holds %lld bytes, %lld needed",
                                    (long long)capacity, (long long)total);
  char* dt = text;
  if (mem == CPETGB_HOST) CK(S.get(&dt, size_t(std::max<int64_t>(total, 1))), "alloc text");
  CK(launch_text_write(fmt, n_rows, n_cols, dv, off, dt, s), "write pass");
  if (mem == CPETGB_HOST) {
    if (total) CK(cudaMemcpyAsync(text, dt, size_t(total), cudaMemcpyDeviceToHost, s), "copy text");
    return finish(c, s);
  }
  return CPETGB_OK;
}

// kind 0: chi-square over histogram rows [n][feat]; kind 1: field rows [n][feat][3].
int distance_impl(int kind, int prec, int mem, int n, int feat, const double* src, double* out,
                  void* stream) {
  if (!valid_prec(prec)) return fail(CPETGB_EINVAL, "bad precision %d", prec);
  if (!valid_mem(mem)) return fail(CPETGB_EINVAL, "bad memory kind %d", mem);
  if (n < 0 || feat < 0) return fail(CPETGB_EINVAL, "negative matrix or feature count");
  if (n > 65535 * 64) return fail(CPETGB_EINVAL, "at most %d rows", 65535 * 64);
  if (n == 0) return CPETGB_OK;
  if (!out || (feat > 0 && !src)) return fail(CPETGB_EINVAL, "NULL pointer");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mem == CPETGB_HOST && !s) s = c->stream;
  Scratch S(s);
  const size_t nc = kind == 0 ? 1 : 3;
  const double* dsrc = src;
  double* dout = out;
  if (mem == CPETGB_HOST) {
    if (feat) CK(h2d(const_cast<double**>(&dsrc), S, src, size_t(n) * feat * nc), "copy rows");
    CK(S.get(&dout, size_t(n) * n), "alloc matrix");
  }
  const int splits = distance_splits(n, feat, c->sms);
  unsigned char *partial = nullptr, *f32_rows = nullptr;
  if (splits > 1) CK(S.get(&partial, distance_partial_bytes(prec, kind, n, splits)), "alloc partial sums");
  if (prec != CPETGB_FP64 && feat > 0)
    CK(S.get(&f32_rows, distance_f32_bytes(kind, n, feat)), "alloc float rows");
  if (reinterpret_cast<uintptr_t>(f32_rows) % 16 != 0)  // bulk async copies need 16-byte sources
    return fail(CPETGB_ECUDA, "scratch allocation is not 16-byte aligned");
  CK(launch_distance_matrix(prec, kind, n, feat, dsrc, dout, splits, partial, f32_rows, c->status, s),
     "distance launch");
  if (mem == CPETGB_HOST) {
    CK(cudaMemcpyAsync(out, dout, size_t(n) * n * sizeof(double), cudaMemcpyDeviceToHost, s),
       "copy matrix");
    return finish(c, s);
  }
  return CPETGB_OK;
}

std::vector<double> widen(const float* p, size_t n) {
  std::vector<double> v(n);
  for (size_t i = 0; i < n; ++i) v[i] = p[i];
  return v;
}

template <typename T>
cudaError_t plan_alloc(std::vector<void*>& bufs, T** p, size_t count) {
  *p = nullptr;
  void* v = nullptr;
  cudaError_t e = cudaMalloc(&v, std::max<size_t>(count, 1) * sizeof(T));
  if (e == cudaSuccess) {
    bufs.push_back(v);
    *p = static_cast<T*>(v);
  }
  return e;
}

}  // namespace

// A prepared launch: device tables and scratch allocated once, the launch
// sequence captured into a CUDA graph and replayed by cpetgb_plan_launch.
struct cpetgb_plan {
  int device = -1;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<void*> bufs;
  ~cpetgb_plan() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    for (void* p : bufs) cudaFree(p);
  }
};

namespace {

// Captures `body` (launches on the capture stream) into plan->graph/exec.
template <typename Body>
int capture_plan(cpetgb_plan* pl, Body body) {
  cudaStream_t cs = nullptr;
  CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "capture stream");
  cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    cudaStreamDestroy(cs);
    return cuda_fail(e, "begin capture");
  }
  const int rc = body(cs);
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(cs, &g);
  cudaStreamDestroy(cs);
  if (rc != CPETGB_OK) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return cuda_fail(e, "end capture");
  pl->graph = g;
  CK(cudaGraphInstantiate(&pl->exec, g, 0), "graph instantiate");
  return CPETGB_OK;
}

int grid_plan_impl(cpetgb_plan** out_plan, int kind, int prec, int clamp, int n_frames,
                   const int64_t* desc, const double* pts, const double* x, const double* q,
                   double* out) {
  if (!out_plan) return fail(CPETGB_EINVAL, "plan pointer is NULL");
  *out_plan = nullptr;
  if (kind != CPETGB_FIELD && kind != CPETGB_ESP) return fail(CPETGB_EINVAL, "bad grid kind %d", kind);
  if (!valid_prec(prec)) return fail(CPETGB_EINVAL, "bad precision %d", prec);
  if (n_frames < 0 || (n_frames > 0 && !desc)) return fail(CPETGB_EINVAL, "bad frame table");
  int64_t tot_pts = 0, tot_ch = 0;
  for (int f = 0; f < n_frames; ++f) {
    const int64_t co = desc[4 * f], n = desc[4 * f + 1], po = desc[4 * f + 2], P = desc[4 * f + 3];
    if (co < 0 || n < 0 || po < 0 || P < 0 || n > INT_MAX || P > INT_MAX)
      return fail(CPETGB_EINVAL, "frame %d: negative or oversized offset/count", f);
    tot_pts = std::max(tot_pts, po + P);
    tot_ch = std::max(tot_ch, co + n);
  }
  if (tot_pts > 0 && (!pts || !out)) return fail(CPETGB_EINVAL, "points/output pointer is NULL");
  if (tot_ch > 0 && (!x || !q)) return fail(CPETGB_EINVAL, "charge pointer is NULL");
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  GridTable gp;
  int ppt = 4, ips = 8;
  tuned_grid_shape(prec, kind, grid_pair_evals(n_frames, desc), &ppt, &ips);
  rc = plan_grid(prec, n_frames, desc, c->sms, ppt, ips, gp);
  if (rc != CPETGB_OK) return rc;
  GridLaunch g = grid_launch(kind, prec, clamp, ppt, n_frames, desc, gp, tot_ch, c);
  g.points = pts;
  g.x = x;
  g.q = q;
  g.out = out;
  cpetgb_plan* pl = new cpetgb_plan();
  cudaGetDevice(&pl->device);
  const bool point = grid_point_fits(g);
  unsigned char *packed = nullptr, *dfq = nullptr;
  GridFrame* d_frames = nullptr;
  cudaError_t e = plan_alloc(pl->bufs, &packed, size_t(std::max<int64_t>(tot_ch, 1)) * kGridRecord);
  if (e == cudaSuccess) e = plan_alloc(pl->bufs, &d_frames, gp.frames.size());
  if (e == cudaSuccess && !gp.frames.empty())
    e = cudaMemcpy(d_frames, gp.frames.data(), gp.frames.size() * sizeof(GridFrame), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = plan_alloc(pl->bufs, &g.zeroed, grid_zero_ints(n_frames, g.tau > 0.0));
  if (e == cudaSuccess && gp.n_slots)
    e = plan_alloc(pl->bufs, &g.partial, size_t(gp.n_slots) * grid_slot_doubles(kind, ppt));
  if (e == cudaSuccess && g.tau > 0.0) {
    e = plan_alloc(pl->bufs, &dfq, size_t(tot_ch) * 32);
    if (e == cudaSuccess) e = plan_alloc(pl->bufs, &g.list, size_t(refine_list_len(n_frames, desc)) * 2);
  }
  if (e != cudaSuccess) {
    delete pl;
    return cuda_fail(e, "plan allocation");
  }
  g.packed = packed;
  g.frames = d_frames;
  g.dfq = dfq;
  e = preload_grid_kernels(prec, kind, clamp ? 1 : 0, ppt);
  if (e != cudaSuccess) {
    delete pl;
    return cuda_fail(e, "kernel load");
  }
  rc = capture_plan(pl, [&](cudaStream_t cs) -> int {
    if (point)
      CK(launch_grid_point(g, cs), "point kernel launch");
    else
      CK(launch_grid(g, cs), "grid launch");
    return CPETGB_OK;
  });
  if (rc != CPETGB_OK) {
    delete pl;
    return rc;
  }
  *out_plan = pl;
  return CPETGB_OK;
}

int topo_plan_impl(cpetgb_plan** out_plan, int prec, int F, const int64_t* desc,
                   const double* params, const double* starts, const int32_t* n_iter,
                   const double* x, const double* q, double* result, double* ends, int32_t* steps) {
  if (!out_plan) return fail(CPETGB_EINVAL, "plan pointer is NULL");
  *out_plan = nullptr;
  TopoTables t;
  int rc = build_topo_tables(prec, F, desc, params, t);
  if (rc != CPETGB_OK) return rc;
  if (t.tot_lines > 0 && (!starts || !n_iter || !result))
    return fail(CPETGB_EINVAL, "line pointer is NULL");
  if (t.tot_ch > 0 && (!x || !q)) return fail(CPETGB_EINVAL, "charge pointer is NULL");
  Ctx* c = context(&rc);
  if (!c) return rc;
  plan_hand_over(prec, c->sms, t);
  cpetgb_plan* pl = new cpetgb_plan();
  cudaGetDevice(&pl->device);
  unsigned char* packed = nullptr;
  TopoFrame* d_frames = nullptr;
  int64_t* d_src = nullptr;
  int* queues = nullptr;
  TopoState* left = nullptr;
  cudaError_t e =
      plan_alloc(pl->bufs, &packed, size_t(std::max<int64_t>(t.packed_elems, 1)) * packed_size(prec));
  if (e == cudaSuccess) e = plan_alloc(pl->bufs, &d_frames, t.frames.size());
  if (e == cudaSuccess) e = plan_alloc(pl->bufs, &d_src, t.src.size());
  if (e == cudaSuccess) e = plan_alloc(pl->bufs, &queues, size_t(1 + t.rounds) * std::max(F, 1));
  if (e == cudaSuccess && t.left_records)
    e = left_or_none([&] { return plan_alloc(pl->bufs, &left, 2 * size_t(t.left_records)); }, &left, &t.rounds);
  if (e == cudaSuccess && F > 0)
    e = cudaMemcpy(d_frames, t.frames.data(), t.frames.size() * sizeof(TopoFrame),
                   cudaMemcpyHostToDevice);
  if (e == cudaSuccess && F > 0)
    e = cudaMemcpy(d_src, t.src.data(), t.src.size() * sizeof(int64_t), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    delete pl;
    return cuda_fail(e, "plan allocation");
  }
  if (reinterpret_cast<uintptr_t>(packed) % 16 != 0) {
    delete pl;
    return fail(CPETGB_ECUDA, "plan allocation is not 16-byte aligned");
  }
  TopoParams p{};
  p.n_lines = static_cast<int>(t.tot_lines);
  p.starts = starts;
  p.n_iter = n_iter;
  p.packed = packed;
  p.result = result;
  p.ends = ends;
  p.steps = steps;
  p.queue = queues;
  p.left = left;
  p.left_records = t.left_records;
  p.left_count = queues + F;
  p.rounds = t.rounds;
  p.fresh = t.fresh;
  p.status = c->status;
  p.frames = d_frames;
  p.n_frames = F;
  p.max_resident_pad = t.max_res;
  p.max_team_resident = t.max_team_res;
  p.sum_lines = t.sum_lines;
  p.all_resident = t.all_resident ? 1 : 0;
  const int max_pairs = t.max_pairs;
  rc = capture_plan(pl, [&](cudaStream_t cs) -> int {
    CK(cudaMemsetAsync(queues, 0, sizeof(int) * size_t(1 + p.rounds) * std::max(F, 1), cs), "zero queues");
    CK(launch_pack_topo_frames(prec, F, d_frames, d_src, x, q, packed, max_pairs, cs),
       "pack charges");
    CK(launch_topo_frames(prec, p, c->sms, cs), "topo kernel launch");
    return CPETGB_OK;
  });
  if (rc != CPETGB_OK) {
    delete pl;
    return rc;
  }
  *out_plan = pl;
  return CPETGB_OK;
}

}  // namespace

int cpetgb::set_error(int code, const char* msg) { return fail(code, "%s", msg); }

void cpetgb::make_staging() {
  StagingPool& pool = staging_pool();
  std::lock_guard<std::mutex> lock(pool.mu);
  pool.make();
}

int cpetgb::tuned_topo_slots(int prec, bool resident, int n_lines) {
  const int v = tune_choose(tune_key(kOpTopo, prec, resident ? 1 : 0, double(n_lines)));
  return v == 1 ? 2 : 4;
}

void cpetgb::tuned_grid_shape(int prec, int kind, double pair_evals, int* ppt, int* items_per_sm) {
  int v = tune_choose(tune_key(kOpGrid, prec, kind, pair_evals));
  if (v < 0 || v >= kGridVariants) v = 1;  // untuned: 4 points per thread, 8 items per SM
  if (v >= 10) {
    *ppt = ((v - 10) / 2) == 1 ? 8 : 4;
    *items_per_sm = ((v - 10) % 2) == 0 ? 128 : 256;
    return;
  }
  static const int ips[5] = {4, 8, 16, 32, 64};
  *ppt = (v / 5) == 1 ? 8 : 4;
  *items_per_sm = ips[v % 5];
}

extern "C" {

int cpetgb_version(void) { return kVersion; }

int cpetgb_last_error(char* buf, size_t len) {
  if (!buf || len == 0) return CPETGB_EINVAL;
  std::snprintf(buf, len, "%s", g_err.c_str());
  return CPETGB_OK;
}

int cpetgb_device_sms(void) {
  int rc;
  Ctx* c = context(&rc);
  return c ? c->sms : rc;
}

int cpetgb_synchronize(void* stream) {
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  return finish(c, static_cast<cudaStream_t>(stream));
}

int cpetgb_check_wait_limit(double seconds) {
  if (!(seconds > 0.0) || seconds > 2.0)
    return fail(CPETGB_EINVAL, "wait limit must be in (0, 2] s, got %g", seconds);
  int rc;
  Ctx* c = context(&rc);
  if (!c) return rc;
  const unsigned long long ns = static_cast<unsigned long long>(seconds * 1e9);
  CK(launch_wait_limit_check(c->status, ns, c->stream), "wait check launch");
  return finish(c, c->stream);
}

int cpetgb_set_hand_over_records(int on) {
  g_hand_over = on != 0;
  return CPETGB_OK;
}

int cpetgb_set_field_refinement(double tau) {
  if (!(tau >= 0.0) || !std::isfinite(tau) || tau > 1.0)
    return fail(CPETGB_EINVAL, "refinement threshold must be in [0, 1], got %g", tau);
  g_refine_tau.store(tau);
  return CPETGB_OK;
}

double cpetgb_field_refinement(void) { return g_refine_tau.load(); }

int cpetgb_set_default_precision(int precision) {
  if (!valid_prec(precision)) return fail(CPETGB_EINVAL, "bad precision %d", precision);
  g_default_prec.store(precision);
  return CPETGB_OK;
}

int cpetgb_get_default_precision(void) { return g_default_prec.load(); }

int cpetgb_field_grid(int precision, int mem, int n_points, int n_charges, const double* points,
                      const double* x, const double* q, int clamp, double* field, void* stream) {
  if (n_points < 0 || n_charges < 0) return fail(CPETGB_EINVAL, "negative size");
  const int64_t desc[4] = {0, n_charges, 0, n_points};
  return grid_batch_impl(CPETGB_FIELD, precision, mem, clamp, 1, desc, points, x, q, field, stream);
}

int cpetgb_esp_grid(int precision, int mem, int n_points, int n_charges, const double* points,
                    const double* x, const double* q, double* esp, void* stream) {
  if (n_points < 0 || n_charges < 0) return fail(CPETGB_EINVAL, "negative size");
  const int64_t desc[4] = {0, n_charges, 0, n_points};
  return grid_batch_impl(CPETGB_ESP, precision, mem, 0, 1, desc, points, x, q, esp, stream);
}

int cpetgb_grid_batch(int kind, int precision, int mem, int clamp, int n_frames,
                      const int64_t* desc, const double* points, const double* x,
                      const double* q, double* out, void* stream) {
  return grid_batch_impl(kind, precision, mem, clamp, n_frames, desc, points, x, q, out, stream);
}

int cpetgb_topo_lines(int precision, int mem, int n_lines, int n_charges, const double* starts,
                      const int32_t* n_iter, double step, const double* half_dims,
                      const double* x, const double* q, double* result, double* ends,
                      int32_t* steps, void* stream) {
  return topo_impl(precision, mem, n_lines, n_charges, starts, n_iter, step, half_dims, x, q,
                   result, ends, steps, stream);
}

int cpetgb_topo_dipole_lines(int precision, int mem, int n_lines, int n_dipoles,
                             const double* starts, const int32_t* n_iter, double step,
                             const double* half_dims, const double* x, const double* mu,
                             double* result, double* ends, int32_t* steps, void* stream) {
  return topo_impl(precision, mem, n_lines, n_dipoles, starts, n_iter, step, half_dims, x, mu,
                   result, ends, steps, stream, kDipoles);
}

int cpetgb_topo_batch(int precision, int mem, int n_frames, const int64_t* desc,
                      const double* params, const double* starts, const int32_t* n_iter,
                      const double* x, const double* q, double* result, double* ends,
                      int32_t* steps, void* stream) {
  return topo_batch_impl(precision, mem, n_frames, desc, params, starts, n_iter, x, q, result, ends,
                         steps, stream);
}

int cpetgb_grid_plan_create(cpetgb_plan** plan, int kind, int precision, int clamp, int n_frames,
                            const int64_t* desc, const double* points, const double* x,
                            const double* q, double* out) {
  return grid_plan_impl(plan, kind, precision, clamp, n_frames, desc, points, x, q, out);
}

int cpetgb_topo_plan_create(cpetgb_plan** plan, int precision, int n_frames, const int64_t* desc,
                            const double* params, const double* starts, const int32_t* n_iter,
                            const double* x, const double* q, double* result, double* ends,
                            int32_t* steps) {
  return topo_plan_impl(plan, precision, n_frames, desc, params, starts, n_iter, x, q, result, ends,
                        steps);
}

int cpetgb_tune_key(int op, int precision, int cls, double size) {
  if ((op != kOpGrid && op != kOpTopo) || !valid_prec(precision) || cls < 0 || cls > 15 ||
      !(size >= 0))
    return fail(CPETGB_EINVAL, "bad tuning key arguments");
  return tune_key(op, precision, cls, size);
}

int cpetgb_tune_variants(int op) {
  if (op == kOpGrid) return kGridVariants;
  if (op == kOpTopo) return kTopoVariants;
  return fail(CPETGB_EINVAL, "bad operation %d", op);
}

int cpetgb_topo_resident_limit(int precision, int dipoles) {
  if (!valid_prec(precision)) return fail(CPETGB_EINVAL, "bad precision %d", precision);
  int rc;
  if (!context(&rc)) return rc;
  return static_cast<int>(topo_resident_limit(precision, dipoles ? kDipoles : kCharges));
}

int cpetgb_tune_set(int key, int variant) {
  const int op = key >> 12;
  const int n = op == kOpGrid ? kGridVariants : (op == kOpTopo ? kTopoVariants : 0);
  if (key < 0 || variant < -1 || variant >= n) return fail(CPETGB_EINVAL, "bad tuning entry");
  std::lock_guard<std::mutex> lock(g_tune_mu);
  if (variant < 0)
    g_tune.erase(key);
  else
    g_tune[key] = variant;
  return CPETGB_OK;
}

int cpetgb_tune_get(int key) { return tune_lookup(key); }

int cpetgb_plan_launch(cpetgb_plan* plan, void* stream) {
  if (!plan || !plan->exec) return fail(CPETGB_EINVAL, "plan is NULL or empty");
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev != plan->device)
    return fail(CPETGB_EINVAL, "plan belongs to device %d; current device is %d", plan->device, dev);
  CK(cudaGraphLaunch(plan->exec, static_cast<cudaStream_t>(stream)), "graph launch");
  return CPETGB_OK;
}

int cpetgb_plan_destroy(cpetgb_plan* plan) {
  delete plan;
  return CPETGB_OK;
}

int cpetgb_topo_hist2d(int mem, int n_lines, const double* result, int nb_dist, int nb_curv,
                       const double* range, uint64_t* counts, double* edges, void* stream) {
  return hist_impl(mem, n_lines, result, nb_dist, nb_curv, range, counts, edges, stream);
}

int cpetgb_prepare_frame(int mem, int n_atoms, const double* x, const double* q,
                         const int32_t* resid, const int32_t* resnum, const double* center,
                         const double* inv_basis, double radius, const double* box_half,
                         const double* box_shift, double* x_out, double* q_out, int* n_out,
                         void* stream) {
  return prepare_frame_impl(mem, n_atoms, x, q, resid, resnum, center, inv_basis, radius, box_half,
                            box_shift, x_out, q_out, n_out, stream);
}

int cpetgb_format_fixed3(int mem, int64_t n_rows, int n_cols, const float* values, char* text,
                         int64_t capacity, int64_t* length, void* stream) {
  return format_text_impl(kTextFixed3, mem, n_rows, n_cols, values, text, capacity, length, stream);
}

int cpetgb_format_sci18(int mem, int64_t n_rows, int n_cols, const float* values, char* text,
                        int64_t capacity, int64_t* length, void* stream) {
  return format_text_impl(kTextSci18, mem, n_rows, n_cols, values, text, capacity, length, stream);
}

int cpetgb_topo_hist2d_sets(int mem, int n_sets, const int64_t* offsets, const double* values,
                            int nb_dist, int nb_curv, const double* range, uint64_t* counts,
                            double* hists, void* stream) {
  return hist_sets_impl(mem, n_sets, offsets, values, nb_dist, nb_curv, range, counts, hists,
                        stream);
}

int cpetgb_chi2_distance_matrix(int precision, int mem, int n, int bins, const double* hists,
                                double* out, void* stream) {
  return distance_impl(0, precision, mem, n, bins, hists, out, stream);
}

int cpetgb_field_distance_matrix(int precision, int mem, int n, int n_points,
                                 const double* fields, double* out, void* stream) {
  return distance_impl(1, precision, mem, n, n_points, fields, out, stream);
}

// ---- float32 drop-ins ----------------------------------------------------

int cpetgb_compute_looped_field_p(int precision, int total_points, int n_charges,
                                  const float* x_0, const float* x, const float* Q, float* E) {
  return grid_f32_impl(CPETGB_FIELD, precision, 1, total_points, n_charges, x_0, x, Q, kRowsPlain, E);
}

int cpetgb_compute_esp_grid_p(int precision, int total_points, int n_charges, const float* x_0,
                              const float* x, const float* Q, float* ESP) {
  return grid_f32_impl(CPETGB_ESP, precision, 0, total_points, n_charges, x_0, x, Q, kRowsPlain, ESP);
}

int cpetgb_box_field_rows(int precision, int n_points, int n_charges, const float* points,
                          const float* x, const float* q, float* rows) {
  return grid_f32_impl(CPETGB_FIELD, precision, 1, n_points, n_charges, points, x, q, kRowsField, rows);
}

int cpetgb_box_esp_rows(int precision, int n_points, int n_charges, const float* points,
                        const float* x, const float* q, uint16_t* rows) {
  return grid_f32_impl(CPETGB_ESP, precision, 0, n_points, n_charges, points, x, q, kRowsEspHalf, rows);
}

int cpetgb_calc_esp_base_p(int precision, float* ESP, const float* x_init, int n_charges,
                           const float* x, const float* Q) {
  if (!ESP || !x_init) return fail(CPETGB_EINVAL, "NULL pointer");
  float v = 0.f;
  const int rc = cpetgb_compute_esp_grid_p(precision, 1, n_charges, x_init, x, Q, &v);
  if (rc != CPETGB_OK) return rc;
  ESP[0] += v;
  return CPETGB_OK;
}

int cpetgb_calc_field_p(int precision, float* E, const float* x_init, int n_charges,
                        const float* x, const float* Q) {
  if (!E || !x_init) return fail(CPETGB_EINVAL, "NULL pointer");
  return grid_f32_impl(CPETGB_FIELD, precision, 0, 1, n_charges, x_init, x, Q, kRowsPlain, E);
}

int cpetgb_thread_operation_batch_p(int precision, int n_lines, int n_charges,
                                    const int32_t* n_iter, float step_size, const float* x_0,
                                    const float* dimensions, const float* x, const float* Q,
                                    float* ret) {
  if (n_lines < 0 || n_charges < 0) return fail(CPETGB_EINVAL, "negative size");
  if (n_lines == 0) return CPETGB_OK;
  if (!n_iter || !x_0 || !dimensions || !ret || (n_charges && (!x || !Q)))
    return fail(CPETGB_EINVAL, "NULL pointer");
  auto s = widen(x_0, size_t(n_lines) * 3);
  auto xx = widen(x, size_t(n_charges) * 3);
  auto qq = widen(Q, size_t(n_charges));
  const double half[3] = {dimensions[0], dimensions[1], dimensions[2]};
  std::vector<double> res(size_t(n_lines) * 2);
  const int rc = cpetgb_topo_lines(precision, CPETGB_HOST, n_lines, n_charges,
                                   s.data(), n_iter, double(step_size), half, xx.data(),
                                   qq.data(), res.data(), nullptr, nullptr, nullptr);
  if (rc != CPETGB_OK) return rc;
  for (size_t i = 0; i < res.size(); ++i) ret[i] = static_cast<float>(res[i]);
  return CPETGB_OK;
}

int cpetgb_thread_operation_p(int precision, int n_charges, int n_iter, float step_size,
                              const float* x_0, const float* dimensions, const float* x,
                              const float* Q, float* ret) {
  const int32_t it = n_iter;
  return cpetgb_thread_operation_batch_p(precision, 1, n_charges, &it, step_size, x_0, dimensions,
                                         x, Q, ret);
}

int cpetgb_thread_operation_dipole_p(int precision, int n_dipoles, int n_iter, float step_size,
                                     const float* x_0, const float* dimensions, const float* x,
                                     const float* mu, float* ret) {
  if (n_dipoles < 0) return fail(CPETGB_EINVAL, "negative size");
  if (!x_0 || !dimensions || !ret || (n_dipoles && (!x || !mu)))
    return fail(CPETGB_EINVAL, "NULL pointer");
  auto s = widen(x_0, 3);
  auto xx = widen(x, size_t(n_dipoles) * 3);
  auto mm = widen(mu, size_t(n_dipoles) * 3);
  const double half[3] = {dimensions[0], dimensions[1], dimensions[2]};
  const int32_t it = n_iter;
  double res[2];
  const int rc = cpetgb_topo_dipole_lines(precision, CPETGB_HOST, 1, n_dipoles,
                                          s.data(), &it, double(step_size), half, xx.data(),
                                          mm.data(), res, nullptr, nullptr, nullptr);
  if (rc != CPETGB_OK) return rc;
  ret[0] = static_cast<float>(res[0]);
  ret[1] = static_cast<float>(res[1]);
  return CPETGB_OK;
}

// The reference-shaped entry points: the same calls in the library's default precision.
int cpetgb_compute_looped_field(int total_points, int n_charges, const float* x_0,
                                const float* x, const float* Q, float* E) {
  return cpetgb_compute_looped_field_p(g_default_prec.load(), total_points, n_charges, x_0, x, Q,
                                       E);
}

int cpetgb_compute_esp_grid(int total_points, int n_charges, const float* x_0, const float* x,
                            const float* Q, float* ESP) {
  return cpetgb_compute_esp_grid_p(g_default_prec.load(), total_points, n_charges, x_0, x, Q,
                                   ESP);
}

int cpetgb_calc_esp_base(float* ESP, const float* x_init, int n_charges, const float* x,
                         const float* Q) {
  return cpetgb_calc_esp_base_p(g_default_prec.load(), ESP, x_init, n_charges, x, Q);
}

int cpetgb_calc_field(float* E, const float* x_init, int n_charges, const float* x,
                      const float* Q) {
  return cpetgb_calc_field_p(g_default_prec.load(), E, x_init, n_charges, x, Q);
}

int cpetgb_thread_operation_batch(int n_lines, int n_charges, const int32_t* n_iter,
                                  float step_size, const float* x_0, const float* dimensions,
                                  const float* x, const float* Q, float* ret) {
  return cpetgb_thread_operation_batch_p(g_default_prec.load(), n_lines, n_charges, n_iter,
                                         step_size, x_0, dimensions, x, Q, ret);
}

int cpetgb_thread_operation(int n_charges, int n_iter, float step_size, const float* x_0,
                            const float* dimensions, const float* x, const float* Q,
                            float* ret) {
  return cpetgb_thread_operation_p(g_default_prec.load(), n_charges, n_iter, step_size, x_0,
                                   dimensions, x, Q, ret);
}

int cpetgb_thread_operation_dipole(int n_dipoles, int n_iter, float step_size, const float* x_0,
                                   const float* dimensions, const float* x, const float* mu,
                                   float* ret) {
  return cpetgb_thread_operation_dipole_p(g_default_prec.load(), n_dipoles, n_iter, step_size,
                                          x_0, dimensions, x, mu, ret);
}

}  // extern "C"
