// MSM plan and driver: the host side of Msm (src/msm.rs:82-298), sm_100a kernels in
// msm_kernels.cuh.
//
// A plan owns every scratch buffer for a fixed (group, n, c, L); runs are queued on the
// context stream with no host synchronisation (data-dependent sizes such as the number of
// nonzero digits stay on the device: kernels read them and exit early), so a plan can be
// reused any number of times and captured in a CUDA graph.
#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "host_field.hpp"
#include "msm.hpp"
#include "msm_affine.cuh"
#include "msm_f64.cuh"
#include "msm_kernels.cuh"

namespace zkg {

// Dynamic shared memory of msm_accumulate_f64: the G2 form keeps its accumulators there
// (4 coordinates x 10 doubles x 128 threads); G1 keeps them in registers.
template <class E>
static size_t f64_acc_smem(bool smem_acc = std::is_same<E, f64::Fq2D>::value) {
  return smem_acc ? (size_t)4 * f64::AccSmem<E>::N * 128 * sizeof(double) : 0;
}

// Allows the G2 form's dynamic shared memory beside its static staging buffers (72 KiB a block).
static void set_acc_smem_limits() {
  const int bytes = (int)f64_acc_smem<f64::Fq2D>();
  check_cuda(cudaFuncSetAttribute(msm_accumulate_f64<f64::Fq2D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  bytes),
             "accumulation smem attribute");
  check_cuda(cudaFuncSetAttribute(msm_accumulate_f64<f64::Fq2D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  bytes),
             "accumulation smem attribute");
}

uint32_t default_window(size_t n) {
  // clamp(log2(max(n,1)) - 5, 11, 16) (src/msm.rs:78-80)
  size_t v = n < 1 ? 1 : n;
  int lg = 63 - __builtin_clzll((unsigned long long)v);
  int c = lg - 5;
  if (c < 11) c = 11;
  if (c > 16) c = 16;
  return (uint32_t)c;
}

// Points accumulated per thread when the caller does not choose. Long segments lengthen the chains of
// additions, short ones add heads and merges: about 32 below 2^23 (window, point) entries, 64 below 2^26,
// 128 above, and then as many as make the threads whole waves of the accumulation kernel (four blocks of
// 128 an SM for G1, two for G2), whose last wave otherwise runs nearly empty: G2 2^18 4.75 ms at 32 points
// (4.3 waves), 4.49 at 48 (2.9). Where 16 or fewer suffice, as many as leave one merge tile an SM (two
// for G2), and at least 4: G1 2^14 0.488 ms at 8, 0.466 at 12.
uint32_t auto_seg_len(size_t entries, int group, int sms) {
  const size_t few = (size_t)sms * 256, wave = (size_t)sms * (group == ZKG_G1 ? 512 : 256);
  const size_t small = (entries + few - 1) / few;
  if (small <= 16) return (uint32_t)std::max<size_t>(small, 4);
  const size_t target = entries < (size_t)1 << 23 ? 32 : entries < (size_t)1 << 26 ? 64 : 128;
  const size_t waves = std::max<size_t>(1, (entries + wave * target / 2) / (wave * target));
  if (waves > 16) return (uint32_t)target;  // a part of a wave in so many is nothing
  return (uint32_t)((entries + wave * waves - 1) / (wave * waves));
}

// Entries of one batch of affine rounds. A batch's points between rounds take 48 bytes an entry (G2 96),
// and there are two batches' scratch; G1 2^24 40.4 ms with batches of 2^24, 39.2 with 2^25. Each stream has as
// many batches: accumulation at G1 2^22 8.77 ms in three of them, 8.45 in two.
static size_t affine_batch(int group) { return (size_t)1 << (group == ZKG_G1 ? 25 : 24); }

// Pairs per thread of a round over `pairs` pairs: about 32, such that the threads fill whole waves of
// msm_affine_sums (four blocks an SM, two for G2) or, for small rounds, fewer down to 4.
static uint32_t affine_per_thread(size_t pairs, int group, int sms) {
  const size_t wave = (size_t)sms * (group == ZKG_G1 ? 4 : 2) * kAffineThreads;
  const size_t waves = std::max<size_t>(1, (pairs + wave * 16) / (wave * 32));
  return (uint32_t)std::max<size_t>(4, (pairs + wave * waves - 1) / (wave * waves));
}

// Rounds of affine additions for `entries` entries over the plan's slots (msm_affine.cuh). Each round
// takes half of the additions that are left from the mixed to the cheaper affine form, but costs three
// launches a batch, the latency of an inversion and half a group of padding a slot more. Accumulation and
// merge, ms, with 0 / 2 / 3 / 4 rounds: G1 2^17 0.55 / 0.55 / 0.60 / 0.74, 2^18 0.92 / 0.82 / 0.89 / 1.12, 2^20
// 2.96 / 2.54 / 2.53 / 2.94, 2^22 9.95 / 9.01 / 8.97 / 9.37, 2^24 39.0 / 35.3 / 34.2 / 33.9; G2 2^16 0.88 / 0.89 /
// 1.01 / 1.44, 2^18 2.78 / 2.30 / 2.60 / 3.63, 2^20 8.73 / 7.12 / 7.90 / 11.5, 2^22 32.3 / 28.1 / 27.1. The
// entries are the most there can be: sparse scalars (three in five zero digits) gain from larger sizes
// on than uniform ones, so the line lies at 2^19 and G2 2^18 points (a sparse G1 MSM of 300007 points:
// 1.01 ms without rounds, 1.09 with two). There they lose little yet: whole MSMs, ms, without / with two
// rounds, uniform and sparse: G1 2^19 2.35 / 2.18 and 1.44 / 1.47, 2^20 3.73 / 3.32 and 2.26 / 2.08; G2 2^18
// 3.95 / 3.47 and 2.50 / 2.63, 2^19 6.57 / 5.76 and 4.04 / 3.89. A fixed-base plan is laid out by the slots of
// all windows although its runs fill one set: G1 2^19 2.27 / 2.18 and 1.37 / 1.46, 2^20 3.43 / 3.31 and 2.03 /
// 2.05.
uint32_t MsmPlan::affine_rounds(size_t entries) const {
  if (!affine) return 0;
  const size_t per_slot = entries / slots;
  uint32_t r = 0;
  if (entries >= (size_t)1 << (group == ZKG_G1 ? 23 : 22) && per_slot >= 48) r = 2;
  if (entries >= (size_t)1 << 26 && per_slot >= 128) r = 3;
  if (entries >= (size_t)1 << 28 && per_slot >= 512) r = 4;
  while (r > 0 && entries + slots * ((1u << r) - 1) > 0xfffffffeull) r--;  // places are 32-bit
  return r;
}

MsmPlan::MsmPlan(zkg_ctx* c_, int group_, size_t n_, uint32_t c, uint32_t item_points, bool affine)
    : ctx(c_), group(group_), n(n_), c(c), affine(affine) {
  if (n < 1) fail(ZKG_EINVAL, "an MSM needs at least one point");
  if (c < 9 || c > 20) fail(ZKG_EINVAL, "window size c must be in 9..=20, got " + std::to_string(c));
  if (group != ZKG_G1 && group != ZKG_G2) fail(ZKG_EINVAL, "group must be ZKG_G1 or ZKG_G2");
  if (n >= (size_t)kNegBit) fail(ZKG_EINVAL, "an MSM holds fewer than 2^31 points");
  item_points_req = item_points;

  use(ctx);
  if (group == ZKG_G2) {
    set_acc_smem_limits();
  }
  glv = glv_default();
  // The plan's own choice, form 4 for G1 and form 2 for G2: integer products with interleaved
  // accumulators (field.cuh), inlined for G1; for G2 out of line, one reduction per component.
  // Accumulation, ms: G1 2^16 / 2^20 / 2^22 0.30 / 2.80 / 9.72, against 0.32 / 2.96 / 10.28 for one
  // product per call, 0.31 / 2.94 / 10.24 for two and 0.40 / 3.88 / 13.05 for double-precision
  // limbs; G2 2^20 8.41, against 9.79 for pairs of reduced products, 9.79 for one product per call,
  // 11.1 inlined and 17.3 for limbs (8.41 with two blocks an SM, 9.88 with three, which spill).
  acc_variant = own_variant();
  chunk = std::min(n, max_chunk());
  layout();
  result.alloc(xyzz_words(), "msm result");
  result_handle.ctx = ctx;
  result_handle.ptr = result.ptr;
  result_handle.words = xyzz_words();
  result_handle.owned = false;
  check_cuda(cudaMemsetAsync(result.ptr, 0, xyzz_words() * 4, ctx->stream), "msm result init");
}

size_t MsmPlan::max_chunk() const {
  // fewer than 2^32 - 1 (window, point) entries per pass; GLV: 2 chunk points below 2^31 too
  if (glv) return std::min<size_t>(0xfffffffeull / (2 * ((128 + c - 1) / c)), ((size_t)kNegBit >> 1) - 1);
  return 0xfffffffeull / ((255 + c - 1) / c);
}

void MsmPlan::set_chunk(size_t points) {
  if (fixed_base) fail(ZKG_EINVAL, "a fixed-base plan runs in one pass");
  use(ctx);
  chunk_req = points;
  const size_t want = std::min(n, std::min(points ? points : n, max_chunk()));
  if (want != chunk || !laid_out) {
    chunk = want;
    layout();
  }
}

// The plans that hold spare memory, of every device.
struct SpareList {
  std::mutex mu;
  std::vector<MsmPlan*> plans;
};
static SpareList& spare_list() {
  static SpareList* list = new SpareList;  // outlives plans of any lifetime
  return *list;
}
void SpareEntry::list(MsmPlan* p) {
  SpareList& l = spare_list();
  std::lock_guard<std::mutex> lock(l.mu);
  plan = p;
  l.plans.push_back(p);
}
void SpareEntry::unlist() {
  if (!plan) return;
  SpareList& l = spare_list();
  std::lock_guard<std::mutex> lock(l.mu);
  l.plans.erase(std::remove(l.plans.begin(), l.plans.end(), plan), l.plans.end());
  plan = nullptr;
}

bool give_back_spare(size_t bytes) {
  int device = 0;
  size_t free_bytes = 0, total = 0;
  if (cudaGetDevice(&device) != cudaSuccess || cudaMemGetInfo(&free_bytes, &total) != cudaSuccess) return false;
  SpareList& l = spare_list();
  std::lock_guard<std::mutex> lock(l.mu);
  size_t all = free_bytes;
  for (const MsmPlan* p : l.plans)
    if (p->ctx->device == device) all += p->spare_bytes();
  if (all < bytes) return false;
  for (MsmPlan* p : l.plans)
    if (p->ctx->device == device && p->give_back()) return true;
  return false;
}

void MsmPlan::release_rounds() {
  affine_sums.release();
  for (AffineLane& lane : affine_lane) {
    lane.inverses.release();
    lane.mid[0].release();
    lane.mid[1].release();
  }
}

size_t MsmPlan::rounds_bytes() const {
  size_t words = affine_sums.words;
  for (const AffineLane& lane : affine_lane) words += lane.inverses.words + lane.mid[0].words + lane.mid[1].words;
  return 4 * words;
}

void MsmPlan::drop_rounds_locked() {
  rounds = plain;
  release_rounds();  // cudaFree waits for the runs that use it
}

void MsmPlan::drop_rounds() {
  spare.unlist();
  std::lock_guard<std::mutex> lock(queue_mu);
  drop_rounds_locked();
  captured = false;
}

size_t MsmPlan::spare_bytes() const {
  std::lock_guard<std::mutex> lock(queue_mu);
  return captured ? 0 : rounds_bytes();
}

size_t MsmPlan::give_back() {
  std::lock_guard<std::mutex> lock(queue_mu);
  const size_t bytes = captured ? 0 : rounds_bytes();
  if (bytes) drop_rounds_locked();
  return bytes;
}

void MsmPlan::set_rounds(bool enable) {
  use(ctx);
  affine = enable;
  layout();
}

// Where the affine rounds' scratch does not fit the device beside the rest, the plan goes without.
void MsmPlan::layout() {
  spare.unlist();
  captured = laid_out = false;
  release_rounds();
  const size_t np = glv ? 2 * chunk : chunk;
  windows = glv ? (128 + c - 1) / c : (255 + c - 1) / c;
  half = 1u << (c - 1);
  slots = (size_t)windows * half;
  entries_at = kNoEntries;
  if (const uint32_t group_log = affine_rounds(windows * np)) {
    try {
      layout_rounds(group_log);
      laid_out = true;
      spare.list(this);
      return;
    } catch (const Error& e) {
      if (e.code != ZKG_ENOMEM) throw;
      release_rounds();
    }
  }
  layout_rounds(0);
  laid_out = true;
}

void MsmPlan::check_laid_out() const {
  if (!laid_out)
    fail(ZKG_ENOMEM, "the MSM plan has no scratch: its last change of layout ran out of device memory");
}

void MsmPlan::layout_rounds(uint32_t group_log) {
  const size_t np = glv ? 2 * chunk : chunk;  // points of the largest pass
  const size_t xw = xyzz_words();
  const size_t max_entries = (size_t)windows * np;
  const size_t tile = group == ZKG_G1 ? MergeTile<FqCP>::value : MergeTile<Fq2L>::value;
  auto segments_of = [&](uint32_t log) {
    Segments g;
    g.group_log = log;
    g.groups = (max_entries + slots * (((size_t)1 << log) - 1)) >> log;  // at most: every slot's last group all but empty
    g.seg_len = item_points_req ? item_points_req : auto_seg_len(g.groups, group, ctx->sm_count);
    g.heads = (g.groups + g.seg_len - 1) / g.seg_len;
    for (size_t len = g.heads; len > 1; len = (len + tile - 1) / tile) g.merge_levels++;
    return g;
  };
  plain = segments_of(0);
  rounds = segments_of(group_log);
  counts.alloc(slots + 1, "msm counts");  // and the run's entry count
  slot_start.alloc(slots + 1, "msm slot_start");
  cursor.alloc(slots, "msm cursor");
  scan_tiles_n = (uint32_t)((slots + kScanTile - 1) / kScanTile);
  if (scan_tiles_n > (uint32_t)kScanTile) fail(ZKG_EINVAL, "too many bucket slots");
  tile_sums.alloc(scan_tiles_n, "msm scan tiles");
  sorted.alloc(rounds.groups << group_log, "msm sorted");
  if (c <= 16) {
    ranks.alloc(max_entries, "msm ranks");
    digits.alloc((max_entries + 1) / 2, "msm ranked digits");  // 16 bits per entry
  }
  buckets.alloc(slots * xw, "msm buckets");

  // Running sums: the fewest buckets per thread that leave one chunked level before the marginals, at
  // most 8.
  const uint32_t chunk_log = half > 4 * kMarginalMax ? 3 : half > 2 * kMarginalMax ? 2 : 1;
  const size_t heads_max = std::max(plain.heads, rounds.heads), second = (heads_max + tile - 1) / tile;
  heads[0].alloc(heads_max * xw, "msm heads");
  head_keys[0].alloc(heads_max, "msm head keys");
  heads[1].alloc(std::max<size_t>(second, 1) * xw, "msm heads");
  head_keys[1].alloc(std::max<size_t>(second, 1), "msm head keys");

  // Running-sum levels: m_0 = B; m_{l+1} = ceil(m_l / C) - 1 (C = 2^chunk_log) down to at most
  // kMarginalMax values, the last level's (level_m.back()).
  std::memset(&levels, 0, sizeof(levels));
  levels.chunk_log = chunk_log;
  const uint32_t bucket_chunk = 1u << chunk_log;
  uint32_t m = half;
  size_t tot_points = 0, run_points = 0;
  level_m.clear();
  while (m > kMarginalMax) {
    if (levels.count >= (uint32_t)kMaxReduceLevels) fail(ZKG_EINVAL, "too many reduction levels");
    const uint32_t chunks = (m + bucket_chunk - 1) / bucket_chunk;
    const uint32_t blocks = (chunks + kReduceThreads - 1) / kReduceThreads;  // one tot point per block
    level_m.push_back(m);
    levels.tot_len[levels.count] = blocks;
    levels.tot_offset[levels.count] = (uint32_t)tot_points;
    tot_points += (size_t)blocks * windows;
    m = chunks - 1;
    levels.count++;
    run_points = std::max<size_t>(run_points, (size_t)m * windows);
  }
  level_m.push_back(m);
  uint32_t bits = 0;
  while ((1u << bits) < m) bits++;
  marg_lo = (bits + 1) / 2;
  marg_hi = bits - marg_lo;
  marg_stride = (1u << marg_lo) + (1u << marg_hi) + levels.count;
  tots.alloc(std::max<size_t>(tot_points, 1) * xw, "msm tots");
  runs[0].alloc(std::max<size_t>(run_points, 1) * xw, "msm runs");
  runs[1].alloc(std::max<size_t>(run_points, 1) * xw, "msm runs");
  marginals.alloc((size_t)windows * marg_stride * xw, "msm marginals");
  bit_sums.alloc((size_t)windows * (bits + 1) * xw, "msm bit sums");
  window_sums.alloc((size_t)windows * xw, "msm window sums");
  if (glv) glv_bases.alloc(chunk * affine_words(), "msm GLV bases (phi)");
  else glv_bases.release();
  if (passes() > 1) partial.alloc(xw, "msm pass result");
  else partial.release();
  if (group_log) {  // last, when the rest has what it needs
    // as many batches for each stream, of affine_batch's size and an eighth more at most
    const size_t two = (affine_batch(group) >> group_log) * 9 / 4, twos = (rounds.groups + two - 1) / two;
    batch_groups = (uint32_t)((rounds.groups + 2 * twos - 1) / (2 * twos));
    affine_sums.alloc(rounds.groups * affine_words(), "msm affine sums", true);
    size_t threads = 0;  // of the largest round
    for (uint32_t r = 1; r <= group_log; r++) {
      const size_t pairs = (size_t)batch_groups << (group_log - r);
      const size_t per = affine_per_thread(pairs, group, ctx->sm_count);
      threads = std::max<size_t>(threads, (size_t)grid_for((pairs + per - 1) / per, kAffineThreads) * kAffineThreads);
    }
    for (AffineLane& lane : affine_lane) {
      lane.inverses.alloc(threads * (affine_words() / 2), "msm affine inverses", true);
      for (uint32_t k = 0; k < 2; k++) {  // rounds 1 and 2 write the largest arrays
        if (group_log > k + 1)
          lane.mid[k].alloc(((size_t)batch_groups << (group_log - 1 - k)) * affine_words(), "msm affine points", true);
      }
    }
    if (!side.stream) check_cuda(cudaStreamCreateWithFlags(&side.stream, cudaStreamNonBlocking), "msm side stream");
    if (!side.fork) check_cuda(cudaEventCreateWithFlags(&side.fork, cudaEventDisableTiming), "msm side event");
    if (!side.join) check_cuda(cudaEventCreateWithFlags(&side.join, cudaEventDisableTiming), "msm side event");
  }
}

size_t MsmPlan::xyzz_words() const { return group == ZKG_G1 ? 32 : 64; }
size_t MsmPlan::affine_words() const { return group == ZKG_G1 ? 16 : 32; }

void MsmPlan::check_buffers(const zkg_buf* bases, const zkg_buf* scalars) const {
  // Msm::check_buffers (src/msm.rs:271-282): byte counts in the messages, like the reference.
  size_t sb = scalars->words * 4, need_s = n * 32;
  if (sb < need_s)
    fail(ZKG_ESIZE, "scalars buffer holds " + std::to_string(sb) + " bytes; " + std::to_string(n) +
                        " scalars need " + std::to_string(need_s));
  const size_t points = fixed_base ? (size_t)windows * n : n;  // a fixed-base table has a row per window
  size_t bb = bases->words * 4, need_b = points * affine_words() * 4;
  if (bb < need_b)
    fail(ZKG_ESIZE, "bases buffer holds " + std::to_string(bb) + " bytes; " + std::to_string(points) +
                        " points need " + std::to_string(need_b));
}

// GLV is the G1 default wherever it applies: measured faster than the plain windows at every
// default window on B200 (2^16: 0.70 against 0.87 ms; 2^18: 1.38 / 1.57; 2^20: 3.32 / 3.46;
// 2^22: 10.3 / 10.7; 2^24: 39.2 / 39.7), half the reduction and combination work for the same
// bucket additions.
bool MsmPlan::glv_default() const {
  return group == ZKG_G1 && c <= 16;
}

void MsmPlan::set_glv(bool enable) {
  if (enable == glv && laid_out) return;
  if (enable) {
    if (group != ZKG_G1) fail(ZKG_EINVAL, "GLV splitting is for G1 (the endomorphism (x, y) -> (beta x, y))");
    if (c > 16) fail(ZKG_EINVAL, "GLV splitting needs a window size c <= 16, got " + std::to_string(c));
    if (fixed_base) fail(ZKG_EINVAL, "GLV splitting and fixed-base tables do not combine");
  }
  use(ctx);
  const bool old = glv;
  const size_t old_chunk = chunk;
  glv = enable;
  try {
    chunk = std::min(n, std::min(chunk_req ? chunk_req : n, max_chunk()));
    layout();
  } catch (...) {
    glv = old;
    chunk = old_chunk;
    layout();
    throw;
  }
}

void MsmPlan::set_fixed_base(bool enable) {
  if (enable && c > 16) fail(ZKG_EINVAL, "fixed-base tables need a window size c <= 16, got " + std::to_string(c));
  const size_t plain_windows = (255 + c - 1) / c;  // a table has a row per plain window
  if (enable && plain_windows * n >= (size_t)kNegBit)
    fail(ZKG_EINVAL, "a fixed-base table holds fewer than 2^31 points");
  if (enable && glv) set_glv(false);  // the table's rows are the plain windows
  if (enable && (chunk != n || !laid_out)) {  // one pass: the table's rows are n points apart
    chunk = n;
    layout();
  }
  fixed_base = enable;
}

void fixed_base_table(zkg_ctx* ctx, int group, const zkg_buf* bases, size_t n, uint32_t c, zkg_buf* out) {
  if (n < 1) fail(ZKG_EINVAL, "an MSM needs at least one point");
  if (c < 9 || c > 20) fail(ZKG_EINVAL, "window size c must be in 9..=20, got " + std::to_string(c));
  if (group != ZKG_G1 && group != ZKG_G2) fail(ZKG_EINVAL, "group must be ZKG_G1 or ZKG_G2");
  const uint32_t windows = (255 + c - 1) / c;
  const size_t aw = group == ZKG_G1 ? 16 : 32;
  if (bases->words < n * aw) fail(ZKG_ESIZE, "bases buffer too small for n points");
  if (out->words < (size_t)windows * n * aw) fail(ZKG_ESIZE, "table buffer too small for windows * n points");
  use(ctx);
  if (group == ZKG_G1)
    msm_fixed_base_table<Fq><<<grid_for(n, 128), 128, 0, ctx->stream>>>(bases->ptr, n, c, windows, out->ptr);
  else
    msm_fixed_base_table<Fq2><<<grid_for(n, 128), 128, 0, ctx->stream>>>(bases->ptr, n, c, windows, out->ptr);
  check_launch("msm_fixed_base_table");
}

// The ranked sort's counting pass (msm_rank), plain or with the GLV split.
template <int AGG>
void MsmPlan::rank(const uint32_t* bases, const uint32_t* scalars, cudaStream_t s) {
  const unsigned b256 = 256;
  if (glv) {
    msm_glv_phi<<<grid_for(run_n, b256), b256, 0, s>>>(bases, run_n, glv_bases.ptr);
    check_launch("msm_glv_phi");
    msm_rank_glv<AGG><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, counts.ptr,
                                                              digits.as<uint16_t>(), ranks.ptr);
  } else {
    msm_rank<AGG><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, fixed_base, counts.ptr,
                                                          digits.as<uint16_t>(), ranks.ptr);
  }
}

template <class F>
void MsmPlan::stage(int which, const uint32_t* bases, const uint32_t* scalars, cudaStream_t s) {
  const unsigned b256 = 256;
  const Segments& seg = segments();
  switch (which) {
    case kStageCount:
      check_cuda(cudaMemsetAsync(counts.ptr, 0, (active_slots() + 1) * 4, s), "msm counts clear");
      if (ranked_sort()) {
        if (sort_agg == 0)
          rank<0>(bases, scalars, s);
        else if (sort_agg == 1)
          rank<1>(bases, scalars, s);
        else if (sort_agg == 2)
          rank<2>(bases, scalars, s);
        else
          rank<3>(bases, scalars, s);
        check_launch("msm_rank");
      } else if (sort_agg == 1)
        msm_count<1><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, counts.ptr);
      else if (sort_agg == 2)
        msm_count<2><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, counts.ptr);
      else if (sort_agg == 3)
        msm_count<3><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, counts.ptr);
      else
        msm_count<0><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, counts.ptr);
      check_launch("msm_count");
      break;
    case kStageScan:
    {
      const size_t ns = active_slots();
      const uint32_t tiles = (uint32_t)((ns + kScanTile - 1) / kScanTile);
      scan_tile_sums<<<tiles, kScanBlock, 0, s>>>(counts.ptr, ns, seg.group_log, tile_sums.ptr, counts.ptr + ns);
      check_launch("scan_tile_sums");
      scan_tiles<<<1, kScanBlock, 0, s>>>(tile_sums.ptr, tiles, slot_start.ptr + ns);
      check_launch("scan_tiles");
      scan_apply<<<tiles, kScanBlock, 0, s>>>(counts.ptr, ns, seg.group_log, tile_sums.ptr, slot_start.ptr, cursor.ptr,
                                              sorted.ptr);
      check_launch("scan_apply");
      break;
    }
    case kStageScatter:
      if (ranked_sort()) {
        const dim3 grid((unsigned)grid_for(points(), b256), windows);
        msm_place<<<grid, b256, 0, s>>>(digits.as<uint16_t>(), ranks.ptr, points(), half, fixed_base, glv ? 1 : 0,
                                        slot_start.ptr, seg.group_log, sorted.ptr);
        check_launch("msm_place");
        break;
      }
      // every group merged: measured best or equal for the scatter on every distribution
      msm_scatter<0><<<grid_for(run_n, b256), b256, 0, s>>>(scalars, run_n, c, windows, cursor.ptr, sorted.ptr);
      check_launch("msm_scatter");
      break;
    case kStageAccumulate: {
      // GLV: points run_n..2 run_n - 1 are the phi(P_i) of glv_bases
      const uint32_t* bases2 = glv ? glv_bases.ptr : bases;
      const uint32_t split = glv ? (uint32_t)run_n : 0xffffffffu;
      if (seg.group_log) {
        using A = typename std::conditional<std::is_same<F, Fq>::value, Fq, typename PairedOf<F>::type>::type;
        affine_stage<A>(bases, bases2, split, s);
        msm_accumulate<A><<<grid_for(seg.heads, 128), 128, 0, s>>>(
            affine_sums.ptr, affine_sums.ptr, 0xffffffffu, nullptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len,
            buckets.ptr, heads[0].ptr, head_keys[0].ptr);
        check_launch("msm_accumulate");
        break;
      }
      if ((acc_variant == 5 || acc_variant == 6) && std::is_same<F, Fq>::value) {
        // G1 with the accumulator in shared memory, four blocks per SM
        const size_t acc_smem = f64_acc_smem<f64::FqD>(true);
        if (acc_variant == 5)
          msm_accumulate_f64<f64::FqD, false, true><<<grid_for(seg.heads, 128), 128, acc_smem, s>>>(
              bases, bases2, split, sorted.ptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
        else
          msm_accumulate_f64<f64::FqD, true, true><<<grid_for(seg.heads, 128), 128, acc_smem, s>>>(
              bases, bases2, split, sorted.ptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
      } else if (acc_variant == 3 || (acc_variant > 3 && std::is_same<F, Fq2>::value)) {
        using E = typename std::conditional<std::is_same<F, Fq>::value, f64::FqD, f64::Fq2D>::type;
        const size_t acc_smem = f64_acc_smem<E>();
        if (acc_variant == 3 || acc_variant == 6)
          msm_accumulate_f64<E, true><<<grid_for(seg.heads, 128), 128, acc_smem, s>>>(
              bases, bases2, split, sorted.ptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
        else
          msm_accumulate_f64<E, false><<<grid_for(seg.heads, 128), 128, acc_smem, s>>>(
              bases, bases2, split, sorted.ptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
      }
      else if (acc_variant == 1)
        msm_accumulate<typename CompactOf<F>::type><<<grid_for(seg.heads, 128), 128, 0, s>>>(
            bases, bases2, split, sorted.ptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
      else if (acc_variant == 2)
        msm_accumulate<typename PairedOf<F>::type><<<grid_for(seg.heads, 128), 128, 0, s>>>(
            bases, bases2, split, sorted.ptr, slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
      else
        msm_accumulate<F><<<grid_for(seg.heads, 128), 128, 0, s>>>(bases, bases2, split, sorted.ptr, slot_start.ptr,
                                                                   (uint32_t)active_slots(),
                                                                   seg.seg_len, buckets.ptr, heads[0].ptr, head_keys[0].ptr);
      check_launch("msm_accumulate");
      break;
    }
    case kStageCombine:
      {
        // a warp for each pair of windows (msm_combine_lanes)
        using A = typename std::conditional<std::is_same<F, Fq>::value, Fq, typename CompactOf<F>::type>::type;
        const uint32_t width = glv ? 128u / windows : c, extra = glv ? 128u % windows : 0u;
        const uint32_t warps = std::max(1u, active_windows() / 2);
        auto launch = [&](auto kernel) {
          kernel<<<1, 32 * warps, 0, s>>>(window_sums.ptr, active_windows(), width, extra, combine_out);
        };
        constexpr uint32_t few = CombineWarps<A>::value;
        if (warps <= few) launch(msm_combine_lanes<A, few>);
        else launch(msm_combine_lanes<A, kCombineWindows / 2>);
      }
      check_launch("msm_combine_lanes");
      if (!first_pass) {  // a later pass: add its point into the result
        msm_add_partial<F><<<1, 32, 0, s>>>(result.ptr, partial.ptr);
        check_launch("msm_add_partial");
      }
      break;
    case kStageMerge:
    case kStageReduce:
    case kStageWindows:
      // out-of-line products in every form (PairedOf)
      tail_stage<typename PairedOf<F>::type>(which, s);
      break;
  }
}

// The affine rounds over the run's groups, batch by batch. Batches go to the run's stream and to `side` in turn, so
// that one's reads and inversions meet the other's products: accumulation at 2^24 36.7 ms in one
// stream, 33.7 in two, 2^20 2.52 and 2.43; G2 2^20 7.03 and 6.94.
template <class F>
void MsmPlan::affine_stage(const uint32_t* bases, const uint32_t* bases2, uint32_t split, cudaStream_t s) {
  const uint32_t aw = (uint32_t)affine_words();
  check_cuda(cudaEventRecord(side.fork, s), "fork");
  check_cuda(cudaStreamWaitEvent(side.stream, side.fork, 0), "fork");
  const uint32_t log = rounds.group_log, batches = (uint32_t)((rounds.groups + batch_groups - 1) / batch_groups);
  for (uint32_t b = 0; b < batches; b++) {
    const AffineLane& lane = affine_lane[b & 1];
    const cudaStream_t st = (b & 1) ? side.stream : s;
    auto between = [&](uint32_t k) {  // lane.mid[k]: x of its points, then y
      const size_t points = (size_t)batch_groups << (log - 1 - k);
      return PointArray{lane.mid[k].ptr, lane.mid[k].ptr + points * (aw / 2), aw / 2};
    };
    for (uint32_t r = 1; r <= log; r++) {
      const uint32_t pairs_log = log - r;
      const size_t pairs = (size_t)batch_groups << pairs_log;  // at most
      const uint32_t per_thread = affine_per_thread(pairs, group, ctx->sm_count);
      const unsigned blocks = grid_for((pairs + per_thread - 1) / per_thread, kAffineThreads);
      const PointArray out = r == log ? PointArray{affine_sums.ptr, affine_sums.ptr + aw / 2, aw} : between((r - 1) & 1);
      const PointArray in = r == 1 ? out : between(r & 1);
      const AffineRound<F> a{bases, bases2, split, sorted.ptr, in, out, slot_start.ptr, (uint32_t)active_slots(), b, batches,
                             log, pairs_log, blocks * kAffineThreads, lane.inverses.ptr};
      const size_t smem = 5 * kAffineThreads * sizeof(F);
      if (r == 1) msm_affine_prefixes<F, true><<<blocks, kAffineThreads, 0, st>>>(a);
      else msm_affine_prefixes<F, false><<<blocks, kAffineThreads, 0, st>>>(a);
      check_launch("msm_affine_prefixes");
      msm_affine_invert<F><<<grid_for(blocks, kInvertEach), kAffineThreads, 2 * kAffineThreads * sizeof(F), st>>>(a);
      check_launch("msm_affine_invert");
      if (r == 1) msm_affine_sums<F, true><<<blocks, kAffineThreads, smem, st>>>(a);
      else msm_affine_sums<F, false><<<blocks, kAffineThreads, smem, st>>>(a);
      check_launch("msm_affine_sums");
    }
  }
  check_cuda(cudaEventRecord(side.join, side.stream), "join");
  check_cuda(cudaStreamWaitEvent(s, side.join, 0), "join");
}

template <class FC>
void MsmPlan::tail_stage(int which, cudaStream_t s) {
  switch (which) {
    case kStageMerge: {
      // `few`: a thread takes 6 us for an addition (G2 18), a group of lanes 2 (2.6) of which a block
      // runs 16 (8) at once, so up to 48 (56) additions groups are the faster; 32 for G1 measured the
      // same or better from 2^18 to 2^24, where threads do more of them per second
      constexpr uint32_t tile = MergeTile<FC>::value;
      const size_t smem = (size_t)tile * (sizeof(Xyzz<FC>) + 12);
      const Segments& seg = segments();
      size_t len = seg.heads;  // the largest a level can be (the entry count is on the device)
      for (uint32_t l = 0; l < seg.merge_levels; l++) {
        const size_t out_len = (len + tile - 1) / tile;
        const int src = l & 1, dst = src ^ 1;
        const uint32_t few = group == ZKG_G1 ? 32 : 56;
        msm_merge<FC><<<(unsigned)out_len, kMergeThreads, smem, s>>>(slot_start.ptr, (uint32_t)active_slots(), seg.seg_len, l, few,
                                                                    heads[src].ptr, head_keys[src].ptr, heads[dst].ptr,
                                                                    head_keys[dst].ptr, buckets.ptr);
        check_launch("msm_merge");
        len = out_len;
      }
      break;
    }
    case kStageReduce: {
      const uint32_t* in = buckets.ptr;
      uint32_t in_stride = half;
      for (uint32_t l = 0; l < levels.count; l++) {
        uint32_t m = level_m[l];
        uint32_t chunks = (m + (1u << levels.chunk_log) - 1) >> levels.chunk_log;
        uint32_t* run_out = runs[l & 1].ptr;
        const dim3 grid(levels.tot_len[l], active_windows());
        msm_reduce_level<FC><<<grid, kReduceThreads, kReduceThreads * sizeof(Xyzz<FC>), s>>>(
            in, in_stride, m, levels.chunk_log, l == 0 ? slot_start.ptr : nullptr,
            tots.ptr + (size_t)levels.tot_offset[l] * xyzz_words(), levels.tot_len[l], run_out,
            chunks > 1 ? chunks - 1 : 1);
        check_launch("msm_reduce_level");
        in = run_out;
        in_stride = chunks > 1 ? chunks - 1 : 1;
      }
      break;
    }
    case kStageWindows: {
      // the last level's vector: the buckets, or the last chunked level's running sums
      const uint32_t l = levels.count, m = level_m[l];
      const uint32_t* in = l == 0 ? buckets.ptr : runs[(l - 1) & 1].ptr;
      const uint32_t rows = (m + (1u << marg_lo) - 1) >> marg_lo, threads = SubsetThreads<FC>::value;
      msm_marginals<FC><<<dim3((1u << marg_lo) + rows + l, active_windows()), threads, 0, s>>>(
          in, l == 0 ? half : m, m, marg_lo, l == 0 ? slot_start.ptr : nullptr, tots.ptr, levels, marginals.ptr,
          marg_stride);
      check_launch("msm_marginals");
      msm_bit_sums<FC><<<dim3(marg_lo + marg_hi + 1, active_windows()), threads, 0, s>>>(
          marginals.ptr, marg_stride, m, marg_lo, marg_hi, bit_sums.ptr);
      check_launch("msm_bit_sums");
      msm_window_fold<FC><<<active_windows(), 32 * std::max(1u, (marg_lo + marg_hi + 1) / 2), 0, s>>>(
          bit_sums.ptr, marg_lo + marg_hi, marginals.ptr + ((size_t)(1u << marg_lo) + rows) * xyzz_words(), marg_stride, l,
          levels.chunk_log, window_sums.ptr);
      check_launch("msm_window_fold");
      break;
    }
    case kStageCombine:  // launched by stage() (msm_combine_lanes)
      break;
  }
}

const char* MsmPlan::stage_name(int which) {
  static const char* names[kStages] = {"count", "scan", "scatter", "accumulate", "merge", "reduce", "window sums", "combine"};
  return names[which];
}

// Selects pass `off` (its first point): run_n, where the combination writes, and the pass's
// slice of the bases (a fixed-base plan has one pass) and scalars.
void MsmPlan::begin_pass(size_t off, const uint32_t*& bases, const uint32_t*& scalars) {
  run_n = std::min(chunk, n - off);
  entries_at = active_slots();
  first_pass = off == 0;
  combine_out = first_pass ? result.ptr : partial.ptr;
  bases += off * affine_words();
  scalars += off * 8;
}

void MsmPlan::enqueue(const uint32_t* bases, const uint32_t* scalars, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(queue_mu);
  check_laid_out();
  if (segments().group_log && !captured) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    check_cuda(cudaStreamIsCapturing(s, &status), "stream capture status");
    captured = status != cudaStreamCaptureStatusNone;
  }
  for (size_t off = 0; off < n; off += chunk) {
    const uint32_t *b = bases, *sc = scalars;
    begin_pass(off, b, sc);
    for (int st = 0; st < kStages; st++) {
      size_t ev = timer.enabled ? timer.begin(st, s) : 0;
      if (group == ZKG_G1) stage<Fq>(st, b, sc, s);
      else stage<Fq2>(st, b, sc, s);
      if (timer.enabled) timer.end(ev, s);
    }
  }
  if (timer.enabled) timer.runs++;
}

void MsmPlan::run(const zkg_buf* bases, const zkg_buf* scalars) {
  check_buffers(bases, scalars);
  use(ctx);
  enqueue(bases->ptr, scalars->ptr, ctx->stream);
}

std::vector<std::pair<std::string, double>> MsmPlan::profile(const zkg_buf* bases, const zkg_buf* scalars) {
  check_buffers(bases, scalars);
  use(ctx);
  std::lock_guard<std::mutex> lock(queue_mu);
  check_laid_out();
  std::vector<std::pair<std::string, double>> out;
  cudaEvent_t a, b;
  check_cuda(cudaEventCreate(&a), "event");
  check_cuda(cudaEventCreate(&b), "event");
  for (int st = 0; st < kStages; st++) out.emplace_back(stage_name(st), 0.0);
  for (size_t off = 0; off < n; off += chunk) {  // stage times summed over the passes
    const uint32_t *bp = bases->ptr, *sp = scalars->ptr;
    begin_pass(off, bp, sp);
    for (int st = 0; st < kStages; st++) {
      check_cuda(cudaEventRecord(a, ctx->stream), "event record");
      if (group == ZKG_G1) stage<Fq>(st, bp, sp, ctx->stream);
      else stage<Fq2>(st, bp, sp, ctx->stream);
      check_cuda(cudaEventRecord(b, ctx->stream), "event record");
      check_cuda(cudaEventSynchronize(b), "msm stage");
      float ms = 0;
      check_cuda(cudaEventElapsedTime(&ms, a, b), "event time");
      out[st].second += (double)ms;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return out;
}

// ------------------------------------------------------------------ GLV split check

// out[10 i ..]: |k1| (4 words), |k2| (4 words), sign of k1, sign of k2, by glv::split_half.
__global__ void glv_split_kernel(const uint32_t* __restrict__ scalars, size_t count, uint32_t* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  for (int h = 0; h < 2; h++) {
    uint32_t s[8];
    load_scalar(scalars, i, s);
    const bool neg = glv::split_half(s, h == 1);
    for (int k = 0; k < 4; k++) out[10 * i + 4 * h + k] = s[k];
    out[10 * i + 8 + h] = neg ? 1u : 0u;
  }
}

void glv_split(zkg_ctx* ctx, const uint32_t* scalars, size_t count, uint32_t* out) {
  use(ctx);
  DeviceArray in, res;
  in.alloc(count * 8, "GLV split input");
  res.alloc(count * 10, "GLV split output");
  check_cuda(cudaMemcpyAsync(in.ptr, scalars, count * 32, cudaMemcpyHostToDevice, ctx->stream), "copy");
  glv_split_kernel<<<grid_for(count, 128), 128, 0, ctx->stream>>>(in.ptr, count, res.ptr);
  check_launch("glv_split_kernel");
  check_cuda(cudaMemcpyAsync(out, res.ptr, count * 40, cudaMemcpyDeviceToHost, ctx->stream), "copy");
  check_cuda(cudaStreamSynchronize(ctx->stream), "GLV split");
}

// ------------------------------------------------------------------ base upload

// Rescales every coordinate in place on the device: v -> v * scale / 2^256.
static void rescale(zkg_ctx* ctx, zkg_buf* buf, const host::U256& scale_mont) {
  Fq s;
  host::words32(scale_mont, s.w);
  size_t coords = buf->words / 8;
  if (coords == 0) return;
  fq_rescale<<<grid_for(coords, 256), 256, 0, ctx->stream>>>(buf->ptr, coords, s);
  check_launch("fq_rescale");
}

void upload_bases(zkg_ctx* ctx, const uint32_t* xy, size_t words, bool mont256, zkg_buf* out) {
  (void)xy;
  (void)words;
  // Msm::upload_bases: scale = R^2 turns plain x into x*R (src/msm.rs:182-188).
  // Msm::upload_bases_montgomery_256: the input is x*2^256 = x*R already (src/msm.rs:190-197).
  if (!mont256) rescale(ctx, out, host::fq().r2);
}

}  // namespace zkg
