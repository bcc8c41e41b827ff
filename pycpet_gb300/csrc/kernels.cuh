// kernels.cuh -- launch interface between the C-ABI layer (api.cu) and the
// kernels (grid.cu, topo.cu, hist.cu).  Host-side declarations only.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cpetgb {

enum Precision : int { kFP64 = 0, kFP32C = 1 };

// Status word written by kernels (device memory); 0 = fine, first error wins.
enum DevStatus : int {
  kDevOk = 0,
  kDevWaitTimeout = 1,   // an mbarrier wait exceeded its limit
  kDevBadArgument = 2,   // histogram range not finite or inverted
  kDevBadCap = 3,        // a streamline step cap above kMaxLineCap
};

// Largest accepted per-line step cap: keeps every streamline kernel bounded.
constexpr int kMaxLineCap = 1 << 24;
enum GridKind : int { kField = 0, kEsp = 1 };

// Packed charge layouts in HBM (positions relative to the box centre).
struct alignas(32) Charge64 {
  double x, y, z, q;
};
// Point dipole (FP64 streamline form): position and moment.
struct alignas(16) Dipole64 {
  double x, y, z, mx, my, mz;
};
static_assert(sizeof(Dipole64) == 48, "Dipole64 layout");
// Sources of a streamline launch.
enum Source : int { kCharges = 0, kDipoles = 1 };
// FP32C uses float4 {x, y, z, q}.

constexpr int kGridThreads = 128;
// A frame of at most this many points goes to the few-points kernel.  FP32C: 30
// points x 50 frames 476 -> 206 us, but 200 points x 20,000 charges 27 -> 52 us
// (potential; its charges come from L2 there); FP64, where a thread per point
// leaves most of the slow pipe to padding, 200 points 481 -> 236 us.
constexpr int kGridFewPoints = 256;
constexpr int kGridFewPointsFp32 = 32;
// Launches with fewer pairs than this don't look for meshes: the look costs about
// 5 us, a quarter of so small a launch's kernel less.
constexpr double kGridMeshPairsFp32 = 2.0e7, kGridMeshPairsFp64 = 1.0e6;
// Nor is a frame of fewer charges than this looked at: the look reads every point
// twice, and a column saves little per charge.  Potential of 159^3 points x 256 charges:
// 269 us without a look, 282 with it as columns; x 500 charges 487 as columns, 511 as
// points in no order (look included).  In FP64 20 charges already repay it (1,418 us
// against 1,818).
constexpr int kGridMeshChargesFp32 = 512, kGridMeshChargesFp64 = 16;

// One frame of a grid launch (device table, sorted by charge chunk, longest
// first).  Its points are cut into tiles of kGridThreads threads with 4 or 8
// points each, its charges into n_split chunks; a CTA takes one tile and one
// chunk (item = split * n_tiles + tile within the frame).
struct GridFrame {
  int64_t charge_off;   // first charge of the frame in x / q / packed
  int64_t point_off;    // first point of the frame (points / output rows)
  int32_t n_charges;
  int32_t n_points;
  int32_t n_tiles;
  int32_t n_split;
  int32_t chunk;        // charges per split (the last may have fewer)
  int32_t slot_base;    // partial sums of (split, tile): slot_base + item; -1: n_split == 1, none
  int32_t item_base;    // items, tiles and preparation blocks of the frames before this one
  int32_t tile_base;
  int32_t prep_base;
  int32_t few;          // 1: few-points kernel (one tile)
  int32_t pad[2];
};
static_assert(sizeof(GridFrame) == 64, "GridFrame layout");

// A grid launch.  Scratch (device): packed 32 bytes per charge; partial
// n_slots * grid_slot_doubles(kind, ppt); lattice and, for the refinement, list
// (2 int64 per point) and dfq (32 bytes per charge); zeroed: grid_zero_ints()
// ints, cleared by launch_grid unless the caller has (cleared).
struct GridLaunch {
  int prec, kind, clamp, ppt;
  int n_frames;
  const GridFrame* frames;    // device; not read when n_frames == 1
  GridFrame one;              // the frame itself when n_frames == 1 (no table to copy, none to load)
  int n_items;                // items of all frames
  int n_tiles;
  int n_prep;                 // preparation blocks of all frames (0: no look for meshes)
  int few_items;              // items of the frames with few != 0 (they come first)
  int64_t n_charges;          // extent of x / q
  int max_points;             // largest frame
  const double *points, *x, *q;
  double* out;
  void* packed;
  double* partial;
  int* zeroed;
  int* status;
  double tau;                 // refinement threshold; 0: no refinement
  int64_t* list;
  void* dfq;
  int num_sms;
};
constexpr int kGridPrepPoints = 1024;  // points per preparation block of a frame
size_t grid_slot_doubles(int kind, int ppt);
size_t grid_zero_ints(int n_frames, bool refine);

// grid.cu
// A launch of one frame of so few (point, run) units that one CTA does all of it
// in one kernel, without scratch (g.one, points, x, q, out set).
bool grid_point_fits(const GridLaunch& g);
cudaError_t launch_grid_point(const GridLaunch& g, cudaStream_t s);
cudaError_t launch_grid(const GridLaunch& g, cudaStream_t s, bool cleared = false);
// Loads the module code of the grid kernels: those of one form (before a graph
// capture), or all (before a persistent kernel: a first launch loads a kernel's
// code, which waits until the device is idle).
cudaError_t preload_grid_kernels(int prec, int kind, int clamp, int ppt);
cudaError_t preload_grid_kernels();
// Packs x[n][3], q[n] as Charge64 (the FP64 streamline layout) and fills [n,
// n_pad) with zero charges placed far outside any box (they contribute exactly
// zero).
cudaError_t launch_pack_f64(int64_t n, int64_t n_pad, const double* x, const double* q, void* packed,
                            cudaStream_t s);

// topo.cu
// One frame of a streamline launch (device table for multi-frame launches).
struct TopoFrame {
  int64_t packed_off;  // first packed element (FP32C: float4 index of the pair block; FP64: Charge64)
  int64_t line_off;    // first line of the frame in starts / n_iter / result
  int32_t n_pad;       // padded charge count (a multiple of topo_charge_pad(prec))
  int32_t n_lines;
  int32_t resident;    // charges staged in shared memory: n_pad, a prefix, or 0
  int32_t team_resident;  // the same in the team kernel (topo_team.cu)
  int32_t left_off;    // the frame's hand-over records: first one and how many (0: none)
  int32_t left_cap;
  double step;
  double half[3];
};
static_assert(sizeof(TopoFrame) == 72, "TopoFrame layout");

// A line in flight, handed from the persistent kernel to the team kernel.
struct TopoState {
  double x0[3], xip[3], xipp[3], xend[3], xe1[3];
  double pos[3];
  int32_t line, phase, steps, cap;
};
static_assert(sizeof(TopoState) == 160, "TopoState layout");

struct TopoParams {
  int n_lines;
  int n_charges;
  double step;
  double half[3];
  const double* starts;      // [L][3]
  const int32_t* n_iter;     // [L]
  const void* packed;        // packed charges
  double* result;            // [L][2]  {distance, mean curvature}
  double* ends;              // [L][3] or null
  int32_t* steps;            // [L] or null (Euler steps of the main loop)
  int* queue;                // work-queue counter(s), one per frame (zeroed by the caller)
  TopoState* left = nullptr;   // two lists of left_records hand-over records, or null: no hand-over
  int64_t left_records = 0;
  int* left_count = nullptr;   // records written: [rounds][n_frames] counters (zeroed by the caller)
  int rounds = 1;              // team kernel launches (topo_team_rounds); 1 without lists
  bool fresh = false;          // all lines go to the team kernel from their start points (topo_fresh)
  int* status;
  const TopoFrame* frames;   // device frame table (multi-frame launches) or null
  int n_frames;              // frames in the table
  int max_resident_pad;      // largest TopoFrame::resident of the launch (shared-memory size)
  int max_team_resident = 0;  // largest TopoFrame::team_resident of the launch
  int64_t sum_lines = 0;      // lines of all frames of the table
  int all_resident = 0;      // 1: every frame entirely in shared memory (tuner class)
  int source = kCharges;     // kDipoles: packed holds dipoles (single-frame launches only)
};
// Single frame: p.frames == null, the frame is described by n_charges/step/half.
cudaError_t launch_topo(int prec, const TopoParams& p, int num_sms, cudaStream_t s);
// Multi-frame: p.frames/n_frames/queue[n_frames]/max_resident_pad set by the caller.
cudaError_t launch_topo_frames(int prec, const TopoParams& p, int num_sms, cudaStream_t s);
// Packs the charges of every frame of a table (host copy `frames`, device copy `d_frames`,
// source offsets src_off[f] into x/q) into the streamline layout.
cudaError_t launch_pack_topo_frames(int prec, int n_frames, const TopoFrame* d_frames,
                                    const int64_t* d_src, const double* x, const double* q,
                                    void* packed, int max_pairs, cudaStream_t s);
// Hand-over records of a frame of n_lines in each list (TopoFrame::left_cap).
int topo_left_capacity(int num_sms, int64_t n_lines, bool fresh);

// topo_team.cu: lines stepped by teams of warps, in p.rounds launches.  fresh !=
// 0: the lines of the frames' tables from their start points; 0: the lines
// handed over (p.left).
cudaError_t launch_topo_team(int prec, const TopoParams& p, const TopoFrame& f0, int fresh,
                             int num_sms, cudaStream_t s);
int topo_team_resident(int prec, int source, int n_pad);
// Launches of the team kernel for sum_lines lines whose box diagonal is crossed
// in diag_steps steps (the largest of the launch's frames).
int topo_team_rounds(int num_sms, int64_t sum_lines, double diag_steps);
double topo_diag_steps(const double* half, double step);
// the lines a CTA of the team kernel steps together; a CTA of the persistent kernel
// hands its last lines over once it holds no more than this many
constexpr int kTeamLinesPerSm = 16;
constexpr int64_t kMaxLeft = int64_t(1) << 18;  // hand-over records of a launch: two lists of 42 MB
// Whether a launch's lines go to the team kernel from their start points
// (resident: every frame's sources fit shared memory; n_pad: a line's sources, on
// average; lists: hand-over records may be asked for).  Decided once, by who plans the
// launch; that there is no memory for the records in the end does not change it.
bool topo_fresh(int prec, int source, bool resident, double n_pad, int64_t sum_lines, int num_sms, bool lists);
// Whether a frame's last lines are worth handing over (diag_steps: steps across its box).
bool topo_hands_over(int prec, int source, bool resident, int n_pad, double diag_steps);

// max sources (charges or dipoles) held resident in shared memory
size_t topo_resident_limit(int prec, int source = kCharges);
// sources of a frame of n_pad held in shared memory: n_pad when it fits, else
// a prefix of whole Kahan runs; 0 for FP64 (TopoFrame::resident)
int topo_resident_count(int prec, int source, int n_pad);
// bytes per packed source (FP32C charge 16, dipole 24; FP64 charge 32, dipole 48)
size_t topo_source_bytes(int prec, int source);
// Packs point dipoles x[n][3], mu[n][3] in the streamline layout (single frame).
cudaError_t launch_pack_dipoles(int prec, int64_t n, int64_t n_pad, const double* x,
                                const double* mu, void* packed, cudaStream_t s);
int topo_charge_pad(int prec);         // packed charge arrays are padded to this multiple
// Packs charges in the streamline kernel's layout (FP32C: pair layout; FP64: Charge64).
cudaError_t launch_pack_topo(int prec, int64_t n, int64_t n_pad, const double* x, const double* q,
                             void* packed, cudaStream_t s);

// peaks.cu: one CTA whose bounded mbarrier wait can never be satisfied runs
// out after limit_ns and records kDevWaitTimeout in *status.
cudaError_t launch_wait_limit_check(int* status, unsigned long long limit_ns, cudaStream_t s);

// rows.cu: conversions of the float32 host calls.  launch_rows writes n float32
// values (kRowsPlain) or n points' rows, and copies the status word to *tail;
// launch_widen also clears n_zero ints.
enum RowFormat : int { kRowsPlain = 0, kRowsField = 1, kRowsEspHalf = 2 };
cudaError_t launch_widen(int64_t n, const float* in, double* out, int* zeroed, int64_t n_zero, cudaStream_t s);
cudaError_t launch_rows(int fmt, int64_t n, const float* pts, const double* val, void* rows, const int* status,
                        int* tail, cudaStream_t s);
cudaError_t preload_row_kernels();  // as preload_grid_kernels()
// api.cu: allocates the float32 host calls' pinned buffers.
void make_staging();

// api.cu: records `msg` as the calling thread's last error and returns `code`.
int set_error(int code, const char* msg);

// Streamline serving engine (topo.cu kernel, engine.cu host side).
// A chunk of lines of one request; written by the host into host-mapped memory.
struct EngineChunk {
  int32_t frame;       // engine frame slot (index into the frame table)
  int32_t request;     // request slot (index into the done counters)
  int32_t line_begin;  // global line indices [line_begin, line_end)
  int32_t line_end;
  double step;
  double half[3];
};
static_assert(sizeof(EngineChunk) == 48, "EngineChunk layout");

struct EngineParams {
  TopoParams p;                 // line arrays (starts, n_iter, result, ends, steps) and status
  const TopoFrame* frames;      // frame table (packed_off, n_pad) in device memory
  const EngineChunk* chunks;    // chunk ring (host-mapped)
  int chunk_capacity;
  const int* tail;              // chunks published (host-mapped, written by the host)
  int* head;                    // chunks claimed (device memory)
  int* head_mirror;             // claims seen by the host (host-mapped, monotonic)
  int* done;                    // finished lines per request slot (host-mapped)
  int* busy;                    // warps of this launch holding lines (device memory, 0 at launch)
  int* closing;                 // 1 once this launch takes no more chunks (device memory, 0 at launch)
};
cudaError_t launch_engine(int prec, const EngineParams& e, int ctas, cudaStream_t s);
int engine_threads();

// api.cu: the tuned variants (autotuner table, defaults when untuned).
int tuned_topo_slots(int prec, bool resident, int n_lines);    // 2 or 4 line slots per warp
void tuned_grid_shape(int prec, int kind, double pair_evals, int* ppt, int* items_per_sm);

// hist.cu
cudaError_t launch_hist2d(int n, const double* vals, int nb0, int nb1, const double* range,
                          double* edges, unsigned long long* counts, int* status,
                          cudaStream_t s);
cudaError_t launch_hist2d_sets(int n_sets, const int64_t* d_off, int64_t max_set,
                               const double* vals, int nb0, int nb1, const double* range,
                               double* edges, unsigned long long* counts, double* hists,
                               int* status, cudaStream_t s);

// prep.cu: residue radius filter, rotation, box filter, shift, compaction of one
// frame (device pointers; center/inv/half/shift on the host, inv/half/shift may
// be null); the survivor count lands in d_count (device int64).
size_t prep_scratch_bytes(int n);
cudaError_t launch_prepare_frame(int n, const double* x, const double* q, const int32_t* resid,
                                 const int32_t* resnum, const double* center, const double* inv,
                                 double radius, const double* half, const double* shift,
                                 double* x_out, double* q_out, void* scratch, int64_t* d_count,
                                 cudaStream_t s);

// format.cu: in-place exclusive scan of int64 values (scratch: scan_scratch_i64(n)).
int64_t scan_scratch_i64(int64_t n);
cudaError_t scan_exclusive_i64(int64_t n, int64_t* x, int64_t* scratch, cudaStream_t s);
// format.cu: text of a float32 matrix in numpy.savetxt's layout (values joined
// by single spaces, "\n" after each row), "%.3f" or "%.18e".
enum TextFormat : int { kTextFixed3 = 0, kTextSci18 = 1 };
int64_t fixed3_scan_scratch(int64_t n);
cudaError_t launch_text_offsets(int fmt, int64_t n_rows, int n_cols, const float* v,
                                int64_t* offsets, int64_t* scratch, cudaStream_t s);
cudaError_t launch_text_write(int fmt, int64_t n_rows, int n_cols, const float* v,
                              const int64_t* offsets, char* out, cudaStream_t s);

// distance.cu: kind 0 = chi-square over histogram rows [n][feat]; kind 1 =
// summed Euclidean norms over field rows [n][feat][3]; out [n][n].
// splits > 1 (distance_splits) needs partial scratch of distance_partial_bytes;
// FP32C also needs f32_rows scratch of distance_f32_bytes(kind, n, feat) bytes.
int distance_splits(int n, int feat, int num_sms);
size_t distance_f32_bytes(int kind, int n, int feat);
size_t distance_partial_bytes(int prec, int kind, int n, int splits);
cudaError_t launch_distance_matrix(int prec, int kind, int n, int feat, const double* src,
                                   double* out, int splits, void* partial, void* f32_rows,
                                   int* status, cudaStream_t s);
// chi2.cu: kind 0 in FP32C.  Scratch 16-byte aligned.
size_t chi2_rows_bytes(int n, int bins);
size_t chi2_partial_bytes(int n, int splits);
cudaError_t launch_chi2_f32(int n, int bins, const double* hists, double* out, int splits, void* partial,
                            void* rows, int* status, cudaStream_t s);

}  // namespace cpetgb
