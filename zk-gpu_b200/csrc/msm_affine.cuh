// Bucket sums by rounds of affine additions (G1 and G2): the accumulation's first stage.
//
// With the sorted entries of every slot padded to a multiple of A = 2^R, entries 2p and 2p + 1
// always belong to one bucket, and so do the pairs' sums in turn: R rounds of pairwise additions
// leave one affine point per group of A entries, and msm_accumulate sums those. An affine addition
// costs lambda = (y2 - y1) / (x2 - x1), one square and one product, and the quotients' inverses are
// shared (Montgomery's trick: three products an element), so 5 products and 1 square against the
// mixed addition's 6 products, 2 squares and a double product: 764 against 1196 slots of the wide
// multiply-add pipe (G2 1904 against 3016), which bounds both. The points pass through memory between
// rounds, and the first round reads its points at random, twice.
//
// Tried and slower: a round in one kernel, its blocks inverting on their own (157 ps a pair in the first
// round, 130 later, against 140 and 114 in three launches) or through a warp of their own (153, 133);
// four lanes copying one record together (the sums 2.0 against 1.5 ms a batch); the L2::64B hint on
// random reads, which halves their DRAM traffic (1.65 against 1.52 ms).
#pragma once
#include "field_inverse.cuh"
#include "msm_kernels.cuh"

namespace zkg {

constexpr uint32_t kAffineThreads = 128;

// What a pair of points sums to: the general case, an operand at infinity, equal or opposite points.
enum PairKind { kPairAdd, kPairSecond, kPairFirst, kPairDouble, kPairInfinity };

// Where a round's points lie: x of point i at x + i * stride words, y at y + i * stride.
struct PointArray {
  uint32_t *x, *y;
  uint32_t stride;
};

// A round over batch `batch` of `batches` equal shares of the run's groups (slot_start counts groups,
// slot_start[num_slots] of them): pair p of the batch is points 2p and 2p + 1 of `in`, or in the first
// round entries 2p and 2p + 1 of `sorted` from the batch's first group on; its sum goes to point p of
// `out`, from the first group on in the last round (pairs_log = 0: one pair a group). The shares and the
// pairs a thread takes follow the run's own count, so that every block has its part whatever the scalars.
template <class F>
struct AffineRound {
  const uint32_t *bases, *bases2;
  uint32_t split;
  const uint32_t* sorted;
  PointArray in, out;
  const uint32_t* slot_start;
  uint32_t num_slots, batch, batches, group_log, pairs_log;
  uint32_t threads;    // of the round's first and third launch
  uint32_t* inverses;  // per thread, the product of its denominators and then its inverse

  struct Share {
    uint32_t group0, pairs, per_thread;
  };
  __device__ __forceinline__ Share share() const {
    const uint32_t total = __ldg(&slot_start[num_slots]);
    const uint32_t each = (total + batches - 1) / batches;
    const uint32_t group0 = min(batch * each, total), pairs = min(each, total - group0) << pairs_log;
    return Share{group0, pairs, max(4u, (pairs + threads - 1) / threads)};
  }
  // The entries of pair p (first round; later rounds have none).
  template <bool FIRST>
  __device__ __forceinline__ uint2 entries_of(uint32_t group0, uint32_t p) const {
    if constexpr (FIRST) return __ldg(reinterpret_cast<const uint2*>(sorted) + ((size_t)group0 << (group_log - 1)) + p);
    else return make_uint2(0, 0);
  }
  // Point i of the round, or the entry's point; a place without an entry reads point 0's words,
  // which coordinate() turns into zeros.
  __device__ __forceinline__ const uint32_t* point_of(uint32_t entry) const {
    constexpr int AW = PointWords<F>::affine;
    const uint32_t pt = entry & ~kNegBit;
    if (entry == kPadEntry) return bases;
    return pt < split ? bases + (size_t)pt * AW : bases2 + (size_t)(pt - split) * AW;
  }
  template <bool FIRST>
  __device__ __forceinline__ const uint32_t* x_at(uint32_t entry, size_t i) const {
    if constexpr (FIRST) return point_of(entry);
    else return in.x + i * in.stride;
  }
  template <bool FIRST>
  __device__ __forceinline__ const uint32_t* y_at(uint32_t entry, size_t i) const {
    if constexpr (FIRST) return point_of(entry) + PointWords<F>::affine / 2;
    else return in.y + i * in.stride;
  }
  template <bool FIRST>
  __device__ __forceinline__ F coordinate(const F& v, uint32_t entry) const {
    if constexpr (FIRST) return entry == kPadEntry ? F::zero() : v;
    else return v;
  }
  template <bool FIRST>
  __device__ __forceinline__ F load_y(uint32_t entry, size_t i) const {
    const F y = coordinate<FIRST>(load_elem<F>(y_at<FIRST>(entry, i)), entry);
    return FIRST && (entry & kNegBit) ? neg(y) : y;
  }
};

template <class F>
__device__ __forceinline__ PairKind pair_kind(const F& x1, const F& x2, const F& y1, const F& y2) {
  if (x1.is_zero() && y1.is_zero()) return kPairSecond;
  if (x2.is_zero() && y2.is_zero()) return kPairFirst;
  if (!(x1 == x2)) return kPairAdd;
  return y1 == y2 && !y1.is_zero() ? kPairDouble : kPairInfinity;
}

// Words of a thread's next points, brought into shared memory by cp.async while the present pair is
// worked on: 16-byte piece c of thread t at piece c * kAffineThreads + t (no bank conflicts).
template <class F>
struct Staged {
  static constexpr int kPieces = sizeof(F) / 16;  // of one coordinate
  uint4* base;                                    // this thread's first piece
  __device__ __forceinline__ void fetch(int coordinate, const uint32_t* g) const {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(base + coordinate * kPieces * kAffineThreads);
#pragma unroll
    for (int c = 0; c < kPieces; c++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa + 16 * kAffineThreads * c), "l"(g + 4 * c)
                   : "memory");
  }
  __device__ __forceinline__ F get(int coordinate) const {
    F r;
    uint32_t* w = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
    for (int c = 0; c < kPieces; c++) {
      const uint4 v = base[(coordinate * kPieces + c) * kAffineThreads];
      w[4 * c] = v.x;
      w[4 * c + 1] = v.y;
      w[4 * c + 2] = v.z;
      w[4 * c + 3] = v.w;
    }
    return r;
  }
};
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// A round's threads take per_thread pairs each, kAffineThreads apart, in three launches.
//
// First: the product of each thread's denominators, each prefix kept where the pair's sum will go, the
// whole product to inverses[thread]. Bound by memory: 64 bytes read and 32 written for one product, in
// the first round two random reads (44 G/s; 38-52 is what a gather alone reaches over 0.5-2 GiB).
template <class F, bool FIRST>
__global__ void __launch_bounds__(kAffineThreads) msm_affine_prefixes(AffineRound<F> a) {
  constexpr int CW = PointWords<F>::affine / 2;
  __shared__ uint4 staged[2 * Staged<F>::kPieces * kAffineThreads];
  const Staged<F> sm{staged + threadIdx.x};
  const auto [group0, pairs, per_thread] = a.share();
  const uint32_t g = blockIdx.x * kAffineThreads + threadIdx.x;
  const uint32_t p0 = blockIdx.x * kAffineThreads * per_thread + threadIdx.x;
  if (p0 >= pairs) return;
  const uint32_t count = min(per_thread, (pairs - p0 + kAffineThreads - 1) / kAffineThreads);
  const uint32_t out0 = a.pairs_log == 0 ? group0 : 0u;
  auto fetch = [&](uint2 en, uint32_t p) {
    sm.fetch(0, a.template x_at<FIRST>(en.x, 2 * (size_t)p));
    sm.fetch(1, a.template x_at<FIRST>(en.y, 2 * (size_t)p + 1));
    stage_commit();
  };
  uint2 en = a.template entries_of<FIRST>(group0, p0), next = en;
  fetch(en, p0);
  if (count > 1) next = a.template entries_of<FIRST>(group0, p0 + kAffineThreads);
  F run;
  for (uint32_t k = 0; k < count; k++) {
    const uint32_t p = p0 + k * kAffineThreads;
    stage_wait();
    const F x1 = a.template coordinate<FIRST>(sm.get(0), en.x), x2 = a.template coordinate<FIRST>(sm.get(1), en.y);
    const uint2 cur = en;
    if (k + 1 < count) {
      en = next;
      fetch(en, p + kAffineThreads);
      if (k + 2 < count) next = a.template entries_of<FIRST>(group0, p + 2 * kAffineThreads);
    }
    F d = x2 - x1;
    if (x1.is_zero() || x2.is_zero() || d.is_zero()) {
      const F y1 = a.template load_y<FIRST>(cur.x, 2 * (size_t)p);
      const PairKind kind = pair_kind(x1, x2, y1, a.template load_y<FIRST>(cur.y, 2 * (size_t)p + 1));
      if (kind != kPairAdd) d = kind == kPairDouble ? dbl(y1) : F::one();
    }
    if (k == 0) {
      run = d;
    } else {
      store_elem(a.out.x + (size_t)(out0 + p) * a.out.stride, run);
      run = run * d;
    }
  }
  store_elem(a.inverses + (size_t)g * CW, run);
}

// Second: inverses[g] <- 1 / inverses[g] for the round's threads. A thread multiplies kInvertEach of
// them up (kAffineThreads apart), the block's products meet pairwise down to 32, one inversion runs in
// each lane of the first warp, and the way back. Bound by latency: G1 44 us with a block an SM, 64 with
// four, of which the inversion takes a lone thread 14.
constexpr uint32_t kInvertEach = 8;
template <class F>
__global__ void __launch_bounds__(kAffineThreads) msm_affine_invert(AffineRound<F> a) {
  constexpr int CW = PointWords<F>::affine / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  F* const tree = reinterpret_cast<F*>(smem_raw);  // 2 * kAffineThreads elements
  const auto [group0, pairs, per_thread] = a.share();
  const uint32_t tile = kAffineThreads * per_thread;  // pairs of a block of the other launches
  const uint32_t threads = pairs / tile * kAffineThreads + min(pairs % tile, kAffineThreads);  // that have a pair
  const uint32_t g0 = blockIdx.x * kAffineThreads * kInvertEach, t = threadIdx.x;
  if (g0 >= threads) return;
  auto at = [&](uint32_t k) { return a.inverses + (size_t)(g0 + k * kAffineThreads + t) * CW; };
  auto value = [&](uint32_t k) { return g0 + k * kAffineThreads + t < threads ? load_elem<F>(at(k)) : F::one(); };
  F pre[kInvertEach], run = value(0);
#pragma unroll 1
  for (uint32_t k = 1; k < kInvertEach; k++) {
    pre[k] = run;
    run = run * value(k);
  }
  tree[kAffineThreads + t] = run;
  __syncthreads();
  for (uint32_t n = kAffineThreads / 2; n >= 32; n >>= 1) {
    if (t < n) tree[n + t] = tree[2 * (n + t)] * tree[2 * (n + t) + 1];
    __syncthreads();
  }
  if (t < 32) tree[32 + t] = affine_inverse(tree[32 + t]);
  __syncthreads();
  for (uint32_t n = 64; n <= kAffineThreads; n <<= 1) {
    F x;
    if (t < n) x = tree[(n + t) >> 1] * tree[(n + t) ^ 1];
    __syncthreads();
    if (t < n) tree[n + t] = x;
    __syncthreads();
  }
  run = tree[kAffineThreads + t];
#pragma unroll 1
  for (uint32_t k = kInvertEach - 1; k > 0; k--) {
    const F v = value(k);
    if (g0 + k * kAffineThreads + t < threads) store_elem(at(k), run * pre[k]);
    run = run * v;
  }
  if (g0 + t < threads) store_elem(at(0), run);
}

// Third: backwards through each thread's pairs, the inverse of a pair's denominator from the running
// inverse and the pair's prefix, and the pair's sum. Bound by the multiply pipe (83% busy; 84 ps a pair
// for G1, 70 at the pipe's full rate).
template <class F, bool FIRST>
__global__ void __launch_bounds__(kAffineThreads, sizeof(F) == 32 ? 4 : 2) msm_affine_sums(AffineRound<F> a) {
  constexpr int CW = PointWords<F>::affine / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];  // 5 coordinates a thread
  const Staged<F> sm{reinterpret_cast<uint4*>(smem_raw) + threadIdx.x};
  const auto [group0, pairs, per_thread] = a.share();
  const uint32_t g = blockIdx.x * kAffineThreads + threadIdx.x;
  const uint32_t p0 = blockIdx.x * kAffineThreads * per_thread + threadIdx.x;
  if (p0 >= pairs) return;
  const uint32_t count = min(per_thread, (pairs - p0 + kAffineThreads - 1) / kAffineThreads);
  const uint32_t out0 = a.pairs_log == 0 ? group0 : 0u;
  auto result = [&](uint32_t* array, uint32_t p) { return array + (size_t)(out0 + p) * a.out.stride; };
  auto fetch = [&](uint2 en, uint32_t p) {
    sm.fetch(0, a.template x_at<FIRST>(en.x, 2 * (size_t)p));
    sm.fetch(1, a.template x_at<FIRST>(en.y, 2 * (size_t)p + 1));
    sm.fetch(2, a.template y_at<FIRST>(en.x, 2 * (size_t)p));
    sm.fetch(3, a.template y_at<FIRST>(en.y, 2 * (size_t)p + 1));
    sm.fetch(4, result(a.out.x, p));  // the prefix (not written for a thread's first pair, and not used)
    stage_commit();
  };
  const uint32_t last = p0 + (count - 1) * kAffineThreads;
  uint2 en = a.template entries_of<FIRST>(group0, last), next = en;
  fetch(en, last);
  if (count > 1) next = a.template entries_of<FIRST>(group0, last - kAffineThreads);
  F run = load_elem<F>(a.inverses + (size_t)g * CW);
  for (uint32_t k = count; k-- > 0;) {
    const uint32_t p = p0 + k * kAffineThreads;
    stage_wait();
    const F x1 = a.template coordinate<FIRST>(sm.get(0), en.x), x2 = a.template coordinate<FIRST>(sm.get(1), en.y);
    F y1 = a.template coordinate<FIRST>(sm.get(2), en.x), y2 = a.template coordinate<FIRST>(sm.get(3), en.y);
    const F prefix = sm.get(4);
    if constexpr (FIRST) {
      if (en.x & kNegBit) y1 = neg(y1);
      if (en.y & kNegBit) y2 = neg(y2);
    }
    if (k > 0) {
      en = next;
      fetch(en, p - kAffineThreads);
      if (k > 1) next = a.template entries_of<FIRST>(group0, p - 2 * kAffineThreads);
    }
    F d = x2 - x1, num = y2 - y1;
    PairKind kind = kPairAdd;
    if (x1.is_zero() || x2.is_zero() || d.is_zero()) {
      kind = pair_kind(x1, x2, y1, y2);
      if (kind == kPairDouble) {
        d = dbl(y1);
        const F xx = sqr(x1);
        num = dbl(xx) + xx;
      } else if (kind != kPairAdd) {
        d = F::one();
      }
    }
    F inv = run;
    if (k > 0) mul2(run, prefix, run, d, inv, run);
    const F lambda = num * inv;
    F x3 = (sqr(lambda) - x1) - x2;
    F y3 = lambda * (x1 - x3) - y1;
    if (kind == kPairSecond) {
      x3 = x2;
      y3 = y2;
    } else if (kind == kPairFirst) {
      x3 = x1;
      y3 = y1;
    } else if (kind == kPairInfinity) {
      x3 = y3 = F::zero();
    }
    store_elem(result(a.out.x, p), x3);
    store_elem(result(a.out.y, p), y3);
  }
}

}  // namespace zkg
