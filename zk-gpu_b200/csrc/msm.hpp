// MSM plan (host side of Msm, src/msm.rs:25-298).
#pragma once
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "msm_common.hpp"
#include "runtime.hpp"

namespace zkg {

uint32_t default_window(size_t n);
uint32_t auto_seg_len(size_t entries, int group, int sms);  // points per segment, unless the caller chooses
void upload_bases(zkg_ctx* ctx, const uint32_t* xy, size_t words, bool mont256, zkg_buf* out);
// out (windows * n points) <- the fixed-base table of n resident bases for window size c: row w
// holds 2^(c w) P_i (windows = ceil(255 / c)); queued on the context stream.
void fixed_base_table(zkg_ctx* ctx, int group, const zkg_buf* bases, size_t n, uint32_t c, zkg_buf* out);
// The device's GLV split of `count` host scalars (8 words each): per scalar |k1| and |k2| (4
// words each) and their signs (1 word each), to host memory.
void glv_split(zkg_ctx* ctx, const uint32_t* scalars, size_t count, uint32_t* out);

struct MsmPlan;

// A plan's place among those that hold spare memory (give_back_spare); leaves it when destroyed.
struct SpareEntry {
  MsmPlan* plan = nullptr;
  void list(MsmPlan* p);
  void unlist();
  ~SpareEntry() { unlist(); }
};

struct MsmPlan {
  enum Stage {
    kStageCount,
    kStageScan,
    kStageScatter,
    kStageAccumulate,
    kStageMerge,
    kStageReduce,
    kStageWindows,
    kStageCombine,
    kStages
  };

  zkg_ctx* ctx;
  int group;
  size_t n;
  uint32_t c, windows = 0, half = 0;
  bool affine;  // may have affine rounds (their scratch doubles the plan's memory or more)
  // Accumulation kernel form: 0 = integer field products inlined, 1 = through one out-of-line
  // product, 2 = out of line, independent products two per call (G2: one reduction per component of
  // an Fq2 product), 3 / 5 / 6 = bucket arithmetic in
  // double-precision limbs (msm_f64.cuh: two products per call, or for G1 the accumulator in
  // shared memory with one / two per call), 4 = for G1 the plan's own choice (inlined integer
  // products), for G2 limbs with one product per call. Every form fetches the next base into
  // shared memory with cp.async. Defaults (measured, MsmPlan's constructor): G1 4, G2 2. Tunable.
  int acc_variant = 4;
  // Warp aggregation of the counting pass's atomics (slot_peers in msm_kernels.cuh): 0 = every
  // group of equal slots, 1 = the first lane's group, 2 = none, 3 = the group of the first equal
  // neighbour pair. The scatter pass always merges every group.
  int sort_agg = 3;
  // Counting sort: 0 = scalar-major scatter through atomic cursors, 1 = ranked (the counting
  // pass records each digit's rank in its slot, the placing pass runs window by window;
  // msm_rank / msm_place). 1 is the default where it applies (c <= 16).
  int sort_form = 1;
  bool ranked_sort() const { return fixed_base || glv || (sort_form == 1 && c <= 16); }
  // Fixed-base mode: `bases` of run() is a table from fixed_base_table() (windows * n points,
  // row w = 2^(c w) P_i), every window's digits share one set of 2^(c-1) buckets, and the
  // result is that set's running sum: no per-window reductions and no combination doublings.
  // Needs c <= 16 (the ranked sort).
  bool fixed_base = false;
  // GLV mode (G1, c <= 16): every scalar splits as k1 + k2 lambda with 127-bit halves, and the
  // MSM runs over the 2n points P_i, phi(P_i) (phi(P_i) in glv_bases, made from `bases` on every
  // run; each half-scalar's sign in its digits) with
  // W = ceil(128 / c) windows of floor(128 / W) or floor(128 / W) + 1 bits (glv_window_width):
  // about the same number of bucket additions, half the windows, so half the reductions and half
  // the combination doublings.
  // On by default where it applies (glv_default); zkg_msm_set_glv switches it; fixed-base mode
  // switches it off.
  bool glv = false;
  bool glv_default() const;
  // Points per pass. Entry positions and point indices are 32-bit, so one pass holds fewer than
  // 2^32 (window, point) entries; a run over more points goes in passes of `chunk` points whose
  // results are added (the reference's limit, n < 2^31, is kept). The plan's scratch is sized
  // for one pass, so a smaller chunk (zkg_msm_set_chunk) also bounds its device memory.
  size_t chunk = 0, run_n = 0;  // run_n: the points of the pass being queued
  // Where the last pass left its entry count in `counts` (the switches between runs move active_slots());
  // kNoEntries before a run and after a change of layout.
  static constexpr size_t kNoEntries = ~(size_t)0;
  size_t entries_at = kNoEntries;
  size_t chunk_req = 0;         // 0: the largest pass the mode allows
  size_t max_chunk() const;
  void set_chunk(size_t points);
  size_t passes() const { return (n + chunk - 1) / chunk; }
  size_t points() const { return glv ? 2 * run_n : run_n; }
  size_t active_slots() const { return fixed_base ? half : slots; }
  uint32_t active_windows() const { return fixed_base ? 1u : windows; }
  size_t slots = 0;
  // What the accumulation kernel sums: groups of 2^group_log entries, each of which the affine rounds
  // (msm_affine.cuh) have made one point, or the entries themselves (group_log = 0); in segments of
  // seg_len, one partial sum (head) each at most, merged in merge_levels launches. The rounds belong to the plan's own
  // accumulation form; the scratch holds both layouts, so that switching the form moves nothing.
  // The rounds' own scratch (affine_sums, affine_lane) is spare memory: taken where the device has
  // room, given back when an allocation fails for want of it (G1 2^20 320 MiB without it, 1220 with).
  struct Segments {
    uint32_t group_log = 0, seg_len = 0, merge_levels = 0;
    size_t groups = 0, heads = 0;
  };
  Segments rounds, plain;
  int own_variant() const { return group == ZKG_G1 ? 4 : 2; }
  const Segments& segments() const { return rounds.group_log && acc_variant == own_variant() ? rounds : plain; }
  uint32_t affine_rounds(size_t entries) const;
  uint32_t batch_groups = 0;  // of a batch of rounds, at most, which bounds their scratch
  uint32_t scan_tiles_n = 0;
  ReduceLevels levels;
  std::vector<uint32_t> level_m;

  DeviceArray counts, slot_start, cursor, tile_sums, sorted, buckets;
  DeviceArray ranks, digits;  // the ranked sort's rank (32 bits) and digit (16 bits) per (window, point), window-major
  DeviceArray glv_bases;      // GLV mode: phi(P_0)..phi(P_{n-1})
  DeviceArray affine_sums;    // the rounds' result, one affine point per group
  // Batches alternate between the run's stream and `side`, each with its own scratch: a round's
  // products of denominators, one per thread, and a batch's points between rounds, all x then all y.
  struct AffineLane {
    DeviceArray inverses, mid[2];
  };
  AffineLane affine_lane[2];
  struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    ~SideStream() {
      if (stream) cudaStreamDestroy(stream);
      if (fork) cudaEventDestroy(fork);
      if (join) cudaEventDestroy(join);
    }
  } side;
  DeviceArray heads[2], head_keys[2];
  uint32_t marg_lo = 0, marg_hi = 0, marg_stride = 0;  // the last level's column and row bits (msm_marginals)
  DeviceArray marginals, bit_sums;
  DeviceArray tots, runs[2], window_sums, result, partial;  // partial: a later pass's result
  zkg_buf result_handle;
  StageTimer timer;

  MsmPlan(zkg_ctx* ctx, int group, size_t n, uint32_t c, uint32_t item_points, bool affine = true);
  ~MsmPlan() {
    if (result_handle.last_use) cudaEventDestroy(result_handle.last_use);
    if (result_handle.pending_read) cudaEventDestroy(result_handle.pending_read);
  }
  MsmPlan(const MsmPlan&) = delete;
  MsmPlan& operator=(const MsmPlan&) = delete;
  size_t xyzz_words() const;
  size_t affine_words() const;
  void check_buffers(const zkg_buf* bases, const zkg_buf* scalars) const;
  void set_fixed_base(bool enable);
  void set_glv(bool enable);
  // Whether the plan may have affine rounds; lays the scratch out anew.
  void set_rounds(bool enable);
  uint32_t run_rounds() const { return segments().group_log; }  // of a run as the plan is now
  // Frees the rounds' scratch and goes on without them (queued runs finish first); the rest of the
  // scratch stays where it is. Graphs captured with the rounds must not be launched any more.
  void drop_rounds();
  size_t rounds_bytes() const;    // of the rounds' scratch
  size_t spare_bytes() const;     // the same, or 0 while a captured graph may hold it
  size_t give_back();             // drop_rounds if there are spare bytes; their number
  // Queues every stage on stream s (no host synchronisation).
  void enqueue(const uint32_t* bases, const uint32_t* scalars, cudaStream_t s);
  void run(const zkg_buf* bases, const zkg_buf* scalars);
  std::vector<std::pair<std::string, double>> profile(const zkg_buf* bases, const zkg_buf* scalars);
  static const char* stage_name(int which);

 private:
  template <class F>
  void stage(int which, const uint32_t* bases, const uint32_t* scalars, cudaStream_t s);
  template <class FC>
  void tail_stage(int which, cudaStream_t s);
  template <class F>
  void affine_stage(const uint32_t* bases, const uint32_t* bases2, uint32_t split, cudaStream_t s);
  // Windows, slots, segments, merge and reduction levels and their scratch, for the current
  // mode (points() and the scalar width); the result buffer is kept.
  void layout();
  void layout_rounds(uint32_t group_log);
  uint32_t* combine_out = nullptr;  // where the combination of the pass being queued goes
  bool first_pass = true;
  void begin_pass(size_t off, const uint32_t*& bases, const uint32_t*& scalars);
  template <int AGG>
  void rank(const uint32_t* bases, const uint32_t* scalars, cudaStream_t s);
  uint32_t item_points_req = 0;
  void release_rounds();
  void drop_rounds_locked();
  // Every array of the scratch is there; not after a change of layout that ran out of memory, until one
  // that fits.
  bool laid_out = false;
  void check_laid_out() const;

 public:
  // Held while a run is queued and while the rounds' scratch is given back, by whichever thread.
  mutable std::mutex queue_mu;

 private:
  bool captured = false;  // a graph may hold the rounds' scratch
  SpareEntry spare;       // last: the plan is off the list before its arrays go
};

}  // namespace zkg

struct zkg_msm {
  zkg::MsmPlan plan;
  template <class... A>
  explicit zkg_msm(A&&... a) : plan(std::forward<A>(a)...) {}
};
