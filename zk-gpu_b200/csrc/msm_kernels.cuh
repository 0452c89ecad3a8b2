// MSM device kernels (signed-digit Pippenger), templated on the coordinate field
// (Fq for G1, Fq2 for G2).
//
// Pipeline for one run (reference stage in brackets):
//   1. recode + count   per point, W signed c-bit digits; warp-aggregated histogram of
//                       (window, |digit|) slots                    [msm_digits.wgsl, count]
//   2. scan             exclusive prefix sum over all W*B slots -> slot_start, cursor
//                                                                  [msm_scan.wgsl]
//   3. recode + scatter point index (sign in bit 31) written to its slot's range, one u32 per
//                       nonzero digit, warp-aggregated cursors     [msm_digits.wgsl, scatter]
//   4. accumulate       the sorted array is cut into equal segments of L entries, one per
//                       thread, regardless of bucket boundaries: every thread does exactly L
//                       mixed additions, so skewed bucket sizes cannot unbalance the warps.
//                       A bucket that starts in a segment is written by that segment's thread;
//                       the parts of a bucket that continue into later segments ("heads")
//                       are emitted per segment with the bucket's slot as key.
//                                                                  [msm_accumulate.wgsl]
//   5. merge levels     heads with equal keys are contiguous; each level sums the runs within tiles
//                       of 256 (G2: 128) of them, adds runs that start in a tile into the bucket,
//                       and passes runs that continue from the previous tile to the next level
//                                                                  [msm_merge/finalize.wgsl]
//   6. reduce level     per window S_w = sum_b (b+1) * bucket_b; above 4096 buckets by chunked
//                       running sums: chunk k of C buckets gives tot_k = sum_j (j+1) B_j and
//                       run_k = sum_j B_j; S_w = sum_k tot_k + C * sum_k k * run_k, and the
//                       second sum is the same problem over run_1.. [msm_reduce_chunks.wgsl]
//   7. window sums      per window the last vector's columns and rows, their bits' sums, and the
//                       fold of those by doublings                [msm_sum.wgsl]
//   8. combine          neighbouring windows pairwise, each pair's upper one doubled by the width of
//                       the lower                                  [msm_combine.wgsl]
#pragma once
#include "curve.cuh"
#include "curve_lanes.cuh"
#include "msm_common.hpp"

namespace zkg {


template <class F>
struct PointWords {
  static constexpr int affine = 2 * FieldWords<F>::value;
  static constexpr int xyzz = 4 * FieldWords<F>::value;
};

// ------------------------------------------------------------------ recoding

// Window w's raw c bits of the scalar (8 LE words). c <= 20 < 32, so two words suffice.
__device__ __forceinline__ uint32_t window_bits(const uint32_t s[8], uint32_t pos, uint32_t c) {
  uint32_t word = pos >> 5, off = pos & 31;
  uint32_t v = 0;
  if (word < 8) v = s[word] >> off;
  if (off + c > 32 && word + 1 < 8) v |= s[word + 1] << (32 - off);
  return v & ((1u << c) - 1);
}

__device__ __forceinline__ void load_scalar(const uint32_t* scalars, size_t i, uint32_t s[8]) {
  const uint4* p = reinterpret_cast<const uint4*>(scalars + 8 * i);
  uint4 lo = __ldg(p), hi = __ldg(p + 1);
  s[0] = lo.x; s[1] = lo.y; s[2] = lo.z; s[3] = lo.w;
  s[4] = hi.x; s[5] = hi.y; s[6] = hi.z; s[7] = hi.w;
}

// Digit recoding of msm_digits.wgsl:19-37: v = window + carry; v >= 2^(c-1) gives the
// negative digit v - 2^c (magnitude 2^c - v) and a carry into the next window. Returns the
// slot (w * B + |digit| - 1) or kNoKey for a zero digit; *neg gets the sign.
struct Recoder {
  uint32_t s[8];
  uint32_t carry = 0;
  __device__ __forceinline__ uint32_t next(uint32_t w, uint32_t c, uint32_t half, bool* neg) {
    uint32_t v = window_bits(s, w * c, c) + carry;
    carry = 0;
    uint32_t mag = v;
    *neg = false;
    if (v >= half) {
      mag = (1u << c) - v;
      *neg = true;
      carry = 1;
    }
    return mag ? w * half + mag - 1 : kNoKey;
  }
};

// Recoding of a GLV half (127-bit magnitude in four words; the words are picked by selects, so
// two of these stay in registers in one thread).
struct GlvRecoder {
  uint32_t s[4];
  uint32_t carry = 0;
  __device__ __forceinline__ uint32_t word(uint32_t i) const {
    return i == 0 ? s[0] : i == 1 ? s[1] : i == 2 ? s[2] : i == 3 ? s[3] : 0u;
  }
  __device__ __forceinline__ uint32_t window_bits(uint32_t pos, uint32_t width) const {
    const uint32_t wd = pos >> 5, off = pos & 31;
    uint32_t v = word(wd) >> off;
    if (off + width > 32) v |= word(wd + 1) << (32 - off);
    return v & ((1u << width) - 1);
  }
  // Recoder::next for a window of `width` bits starting at bit `pos` (width <= c: the GLV
  // windows), the digit negated when `flip` (a negative half-scalar: its digits are those of |k| with the
  // sign turned). A flipped half is recoded with v > 2^(width-1) negative instead of >=, so its
  // digits lie in (-2^(width-1), 2^(width-1)] and, turned, in [-2^(width-1), 2^(width-1)) like
  // every other digit: the positive magnitude 2^(c-1), whose 16-bit code is kRankZero at c = 16,
  // never occurs.
  __device__ __forceinline__ uint32_t next_at(uint32_t w, uint32_t pos, uint32_t width, uint32_t half, bool flip,
                                              bool* neg) {
    const uint32_t v = window_bits(pos, width) + carry;
    const uint32_t h = 1u << (width - 1);
    carry = 0;
    uint32_t mag = v;
    bool neg_d = false;
    if (flip ? v > h : v >= h) {
      mag = (1u << width) - v;
      neg_d = true;
      carry = 1;
    }
    *neg = neg_d != flip;
    return mag ? w * half + mag - 1 : kNoKey;
  }
};

// GLV windows: the 128 bits of the halves split as evenly as possible over W windows, the first
// 128 mod W of them floor(128 / W) + 1 bits wide and the rest floor(128 / W) (at most c bits
// each, since W = ceil(128 / c)). Equal c-bit windows would leave the top one with as little as
// 0.2 significant bits (|k| < 2^126.2), whose few buckets would take every entry's counting
// atomic; here every window keeps at least floor(128 / W) - 1.8 bits, and the top one still
// cannot carry out.
__device__ __forceinline__ uint32_t glv_window_pos(uint32_t w, uint32_t windows) {
  const uint32_t base = 128u / windows, extra = 128u % windows;
  return w * base + (w < extra ? w : extra);
}
__device__ __forceinline__ uint32_t glv_window_width(uint32_t w, uint32_t windows) {
  return 128u / windows + (w < 128u % windows ? 1u : 0u);
}

// Lanes of a warp that share a slot, for one atomic per group. AGG 0: every group
// (__match_any_sync); 1: only the group of the first lane that has a slot (one shuffle and one
// ballot: skewed inputs put most repeats into one hot slot per window); 2: none; 3: the group of
// the first lane whose right neighbour has the same slot (a slot held by a sizeable share of
// the warp almost always shows up in an adjacent pair; uniform digits almost never do, and
// then no group forms). Lanes without a slot (kNoKey) get an empty mask.
template <int AGG>
__device__ __forceinline__ unsigned slot_peers(uint32_t slot) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned active = __activemask();
  if (AGG == 0) {
    const unsigned m = __match_any_sync(active, slot);  // every lane of the mask takes part
    return slot == kNoKey ? 0u : m;
  }
  if (AGG == 1) {
    const unsigned valid = __ballot_sync(active, slot != kNoKey);
    if (!valid) return 0u;
    const int first = __ffs(valid) - 1;
    const uint32_t hot = __shfl_sync(active, slot, first);
    const unsigned group = __ballot_sync(active, slot == hot) & valid;
    if (slot == kNoKey) return 0u;
    return slot == hot ? group : (1u << lane);
  }
  if (AGG == 3) {
    const unsigned valid = __ballot_sync(active, slot != kNoKey);
    const uint32_t right = __shfl_down_sync(active, slot, 1);
    const unsigned pairs = __ballot_sync(active, slot != kNoKey && lane < 31 && slot == right);
    if (slot == kNoKey) return 0u;
    if (!pairs) return 1u << lane;
    const uint32_t hot = __shfl_sync(valid | pairs, slot, __ffs(pairs) - 1);
    const unsigned group = __ballot_sync(valid, slot == hot);
    return slot == hot ? group : (1u << lane);
  }
  return slot == kNoKey ? 0u : (1u << lane);
}

// Pass 1: histogram of (window, bucket) slots; lanes of a warp that hit the same slot are
// merged into one atomic as slot_peers<AGG> groups them (equal scalars, zero-heavy or
// r-1-heavy inputs hammer single slots).
template <int AGG>
__global__ void msm_count(const uint32_t* __restrict__ scalars, size_t n, uint32_t c, uint32_t windows,
                          uint32_t* __restrict__ counts) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool live = i < n;
  Recoder rc;
  if (live) load_scalar(scalars, i, rc.s);
  uint32_t half = 1u << (c - 1);
  const unsigned lane = threadIdx.x & 31;
  for (uint32_t w = 0; w < windows; w++) {
    bool neg;
    uint32_t slot = live ? rc.next(w, c, half, &neg) : kNoKey;
    const unsigned peers = slot_peers<AGG>(slot);
    if (peers && (int)lane == __ffs(peers) - 1) atomicAdd(&counts[slot], (uint32_t)__popc(peers));
  }
}

// Pass 3: scatter point indices (sign in bit 31) into slot order. Within a slot the order is
// whatever the atomics give; bucket sums are exact, so the result does not depend on it.
// Issuing 4 or 8 windows' atomics together measured 1-3% slower at 2^24, so the pass is not
// bound by the atomics' round trips; its scattered 4-byte stores (a 32-byte sector each) are
// the likely bound.
template <int AGG>
__global__ void msm_scatter(const uint32_t* __restrict__ scalars, size_t n, uint32_t c, uint32_t windows,
                            uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool live = i < n;
  Recoder rc;
  if (live) load_scalar(scalars, i, rc.s);
  uint32_t half = 1u << (c - 1);
  const unsigned lane = threadIdx.x & 31;
  for (uint32_t w = 0; w < windows; w++) {
    bool neg = false;
    uint32_t slot = live ? rc.next(w, c, half, &neg) : kNoKey;
    const unsigned peers = slot_peers<AGG>(slot);
    if (AGG == 2) {
      if (peers) sorted[atomicAdd(&cursor[slot], 1u)] = (uint32_t)i | (neg ? kNegBit : 0u);
      continue;
    }
    // every lane takes part in the shuffle below: groups are disjoint, each with its own leader
    const int leader = peers ? __ffs(peers) - 1 : (int)lane;
    uint32_t base = 0;
    if (peers && (int)lane == leader) base = atomicAdd(&cursor[slot], (uint32_t)__popc(peers));
    base = __shfl_sync(__activemask(), base, leader);
    if (peers) sorted[base + __popc(peers & ((1u << lane) - 1))] = (uint32_t)i | (neg ? kNegBit : 0u);
  }
}

// ------------------------------------------------------------------ GLV split (G1)
//
// BN254 G1 has the endomorphism phi(x, y) = (beta x, y), beta a cube root of unity in Fq, and
// phi(P) = lambda P for every P of G1 (a group of prime order r) with lambda the matching cube
// root of unity in Fr. A scalar splits as k = k1 + k2 lambda (mod r) with short k1, k2
// (Gallant, Lambert, Vanstone, CRYPTO 2001), so sum k_i P_i = sum (k1_i P_i + k2_i phi(P_i)): an
// MSM over 2n points whose scalars have 127-bit magnitudes, half the windows of the 254-bit one.
//
// Lattice split: v1 = (a1, b1), v2 = (a2, b2) are short vectors with a + b lambda = 0 (mod r) and
// a1 b2 - a2 b1 = r (the extended Euclidean algorithm on (r, lambda)); c1 = round(b2 k / r), c2 =
// round(-b1 k / r), k1 = k - c1 a1 - c2 a2, k2 = -c1 b1 - c2 b2. The roundings use g1 =
// round(2^256 b2 / r) and g2 = round(2^256 (-b1) / r): c = floor((k g + 2^255) / 2^256) is within
// 1/2 + k / 2^257 < 5/8 of the exact quotient for k < r, so (k1, k2) = -e1 v1 - e2 v2 with |e1|,
// |e2| < 5/8, and |k1|, |k2| < 5/8 (a1 + a2) < 2^126.2 (a2 = -b1 < 2^64, b2 < 2^127). Signed
// c-bit digits of such a magnitude need ceil(128 / c) windows: the top window's bits stay below
// 2^(c - 1.8), so its digit never carries out.
namespace glv {
__device__ constexpr uint64_t kR[4] = {0x43e1f593f0000001ull, 0x2833e84879b97091ull, 0xb85045b68181585dull,
                            0x30644e72e131a029ull};
__device__ constexpr uint64_t kA1[2] = {0x8211bbeb7d4f1128ull, 0x6f4d8248eeb859fcull};
__device__ constexpr uint64_t kB2[2] = {0x0be4e1541221250bull, 0x6f4d8248eeb859fdull};
__device__ constexpr uint64_t kShort[1] = {0x89d3256894d213e3ull};  // a2 = -b1
__device__ constexpr uint64_t kG1[3] = {0x5398fd0300ff6565ull, 0x4ccef014a773d2d2ull, 0x2ull};
__device__ constexpr uint64_t kG2[2] = {0xd91d232ec7e0b3d7ull, 0x2ull};
// beta = 0x30644e72e131a0295e6dd9e7e0acccb0c28f069fbb966e3de4bd44e5607cfd48 (beta^3 = 1 mod q,
// paired with lambda = 0x30644e72e131a029048b6e193fd84104cc37a73fec2bc5e9b8ca0b2d36636f23 mod
// r), here times 2^256 mod q (Montgomery form).
__device__ constexpr uint32_t kBetaMont[8] = {0x13e80b9cu, 0x3350c88eu, 0xdb5e56b9u, 0x7dce557cu,
                                   0xb615564au, 0x6001b4b8u, 0x020217e0u, 0x2682e617u};

// The low L limbs of a * b (64-bit limbs, little-endian).
template <int L, int LA, int LB>
__device__ __forceinline__ void mul_lo(const uint64_t (&a)[LA], const uint64_t (&b)[LB], uint64_t (&r)[L]) {
#pragma unroll
  for (int k = 0; k < L; k++) r[k] = 0;
#pragma unroll
  for (int i = 0; i < LA; i++) {
    uint64_t carry = 0;
#pragma unroll
    for (int j = 0; j < LB; j++) {
      if (i + j < L) {
        const uint64_t lo = a[i] * b[j], hi = __umul64hi(a[i], b[j]);
        uint64_t t = r[i + j] + lo;
        uint64_t cy = t < lo;
        t += carry;
        cy += t < carry;
        r[i + j] = t;
        carry = hi + cy;  // r + a b + carry < 2^128: no overflow
      }
    }
    if (i + LB < L) r[i + LB] = carry;
  }
}

// a - b mod 2^(64 L).
template <int L>
__device__ __forceinline__ void sub_mod(uint64_t (&a)[L], const uint64_t (&b)[L]) {
  uint64_t borrow = 0;
#pragma unroll
  for (int i = 0; i < L; i++) {
    const uint64_t x = a[i] - b[i];
    const uint64_t b1 = a[i] < b[i];
    a[i] = x - borrow;
    borrow = b1 | (x < borrow);
  }
}

// floor((k g + 2^255) / 2^256), taking the LC limbs of the quotient.
template <int LG, int LC>
__device__ __forceinline__ void round_quotient(const uint64_t (&k)[4], const uint64_t (&g)[LG], uint64_t (&c)[LC]) {
  uint64_t p[4 + LG];
  mul_lo<4 + LG>(k, g, p);
  const uint64_t t = p[3] + (1ull << 63);
  uint64_t carry = t < p[3];
#pragma unroll
  for (int i = 4; i < 4 + LG; i++) {
    p[i] += carry;
    carry = carry && p[i] == 0;
  }
#pragma unroll
  for (int i = 0; i < LC; i++) c[i] = p[4 + i];
}

// |v| (a signed 192-bit value, |v| < 2^127) into out (words 0..3; 4..7 zero); whether v < 0.
__device__ __forceinline__ bool store_half(uint64_t (&v)[3], uint32_t out[8]) {
  const bool neg = v[2] >> 63;
  if (neg) {
    uint64_t m[3] = {0, 0, 0};
    sub_mod(m, v);
    v[0] = m[0];
    v[1] = m[1];
  }
  out[0] = (uint32_t)v[0];
  out[1] = (uint32_t)(v[0] >> 32);
  out[2] = (uint32_t)v[1];
  out[3] = (uint32_t)(v[1] >> 32);
#pragma unroll
  for (int i = 4; i < 8; i++) out[i] = 0;
  return neg;
}

// s (8 words, any 256-bit value; reduced mod r first, which changes no multiple of a point of
// G1) -> |k1| in k1, |k2| in k2 (words 0..3, words 4..7 zero) and their signs.
__device__ __forceinline__ void split(const uint32_t s[8], uint32_t k1[8], bool& neg1, uint32_t k2[8], bool& neg2) {
  uint64_t k[4];
#pragma unroll
  for (int i = 0; i < 4; i++) k[i] = s[2 * i] | (uint64_t)s[2 * i + 1] << 32;
#pragma unroll
  for (int t = 0; t < 5; t++) {  // 2^256 < 6 r
    uint64_t d[4] = {k[0], k[1], k[2], k[3]};
    uint64_t borrow = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint64_t x = d[i] - kR[i];
      const uint64_t b1 = d[i] < kR[i];
      d[i] = x - borrow;
      borrow = b1 | (x < borrow);
    }
    if (!borrow) {
#pragma unroll
      for (int i = 0; i < 4; i++) k[i] = d[i];
    }
  }
  uint64_t c1[2], c2[1];
  round_quotient(k, kG1, c1);  // < b2 + 1 < 2^127
  round_quotient(k, kG2, c2);  // < -b1 + 1 < 2^64
  uint64_t v[3] = {k[0], k[1], k[2]}, t[3];  // k1 = k - c1 a1 - c2 a2
  mul_lo<3>(c1, kA1, t);
  sub_mod(v, t);
  mul_lo<3>(c2, kShort, t);
  sub_mod(v, t);
  neg1 = store_half(v, k1);
  mul_lo<3>(c1, kShort, v);  // k2 = c1 (-b1) - c2 b2
  mul_lo<3>(c2, kB2, t);
  sub_mod(v, t);
  neg2 = store_half(v, k2);
}

// One half of split: s -> |k1| (second = false) or |k2| (second = true), returning its sign.
__device__ __forceinline__ bool split_half(uint32_t s[8], bool second) {
  uint32_t h1[8], h2[8];
  bool n1, n2;
  split(s, h1, n1, h2, n2);
#pragma unroll
  for (int i = 0; i < 8; i++) s[i] = second ? h2[i] : h1[i];
  return second ? n2 : n1;
}
}  // namespace glv

// phi(P_i) = (beta x_i, y_i) for the n bases (affine, Montgomery form; infinity, (0, 0), stays
// (0, 0)): the bases of GLV entries n..2n-1. Entries 0..n-1 read P_i from the caller's bases, and
// every entry's half-scalar sign is in its digits.
__global__ void msm_glv_phi(const uint32_t* __restrict__ bases, size_t n, uint32_t* __restrict__ phi) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Fq beta;
#pragma unroll
  for (int k = 0; k < 8; k++) beta.w[k] = glv::kBetaMont[k];
  const uint4* src = reinterpret_cast<const uint4*>(bases + 16 * i);
  store_fe(phi + 16 * i, load_fe<Fq>(bases + 16 * i) * beta);
  uint4* dst = reinterpret_cast<uint4*>(phi + 16 * i);
  dst[2] = __ldg(src + 2);
  dst[3] = __ldg(src + 3);
}

// ------------------------------------------------------------------ ranked counting sort
//
// The same sort in two passes without scattered stores over the whole sorted array:
//   msm_rank  recodes each scalar once; the warp-aggregated atomic that counts a digit also
//             returns its rank within its slot; the digit (bucket | sign << 15, kRankZero for a
//             zero digit; 16 bits) and the rank (32 bits) go to window-major arrays (entry
//             w * n + i) with coalesced streaming stores.
//   msm_place after the scan, walks the entries window by window: sorted[slot_start + rank] =
//             point index | sign. A window's slots span ~4n bytes of the sorted array, so the
//             4-byte stores of the blocks in flight meet in L2 (the scalar-major scatter touches
//             all windows' ranges at once: 1 GiB at 2^24), and no pass needs a second atomic.
// For c <= 16 (15-bit buckets).
constexpr uint32_t kRankZero = 0x7fffu;  // a positive bucket 2^15 - 1 never occurs for c <= 16

// fixed (fixed-base tables: one set of buckets for all windows, see msm_place): the digit of
// window w counts in bucket slot |d| - 1 instead of w * 2^(c-1) + |d| - 1.
template <int AGG>
__global__ void msm_rank(const uint32_t* __restrict__ scalars, size_t n, uint32_t c, uint32_t windows, int fixed,
                         uint32_t* __restrict__ counts, uint16_t* __restrict__ digits,
                         uint32_t* __restrict__ ranks) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n;
  Recoder rc;
  if (live) load_scalar(scalars, i, rc.s);
  const uint32_t half = 1u << (c - 1);
  const unsigned lane = threadIdx.x & 31;
  // Windows four at a time: the four counting atomics (each returns the entry's rank) are in
  // flight together before any result is used.
  constexpr int kBatch = 4;
  for (uint32_t w0 = 0; w0 < windows; w0 += kBatch) {
    uint32_t slot[kBatch], base[kBatch];
    unsigned peers[kBatch];
    bool neg[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      const uint32_t w = w0 + k;
      slot[k] = kNoKey;
      neg[k] = false;
      if (w < windows) {  // uniform across the warp
        if (live) slot[k] = rc.next(w, c, half, &neg[k]);
        if (fixed && slot[k] != kNoKey) slot[k] -= w * half;
        peers[k] = slot_peers<AGG>(slot[k]);
        base[k] = 0;
        if (peers[k] && (int)lane == __ffs(peers[k]) - 1) base[k] = atomicAdd(&counts[slot[k]], (uint32_t)__popc(peers[k]));
      }
    }
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      const uint32_t w = w0 + k;
      if (w >= windows) break;
      const int leader = peers[k] ? __ffs(peers[k]) - 1 : (int)lane;
      const uint32_t b = __shfl_sync(0xffffffffu, base[k], leader);
      if (!live) continue;
      uint32_t code = kRankZero;
      const size_t e = (size_t)w * n + i;
      if (peers[k]) {
        code = (fixed ? slot[k] : slot[k] - w * half) | (neg[k] ? 0x8000u : 0u);
        __stcs(ranks + e, b + __popc(peers[k] & ((1u << lane) - 1)));  // streamed: read once by msm_place
      }
      __stcs(digits + e, (unsigned short)code);
    }
  }
}

// The GLV counting pass, one thread per scalar: thread i splits scalar i once (glv::split) and
// recodes both halves, point i (|k1|, base P_i) and point scalar_n + i (|k2|, base phi(P_i)),
// each half's sign folded into its digits. Entries are window-major with the two halves of a
// scalar side by side (column 2i + h): the placing pass then walks them in the order this pass
// ranked them (columns in point order put each slot's ranks of one half after the other half's
// and cost 0.6 ms more placement at 2^24). Two windows per batch: four counting atomics in
// flight.
template <int AGG>
__global__ void msm_rank_glv(const uint32_t* __restrict__ scalars, size_t scalar_n, uint32_t c, uint32_t windows,
                             uint32_t* __restrict__ counts, uint16_t* __restrict__ digits,
                             uint32_t* __restrict__ ranks) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < scalar_n;
  const size_t n = 2 * scalar_n;
  GlvRecoder rc[2];
  bool flip[2] = {false, false};
  if (live) {
    uint32_t s[8], h1[8], h2[8];
    load_scalar(scalars, i, s);
    glv::split(s, h1, flip[0], h2, flip[1]);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      rc[0].s[j] = h1[j];
      rc[1].s[j] = h2[j];
    }
  }
  const uint32_t half = 1u << (c - 1);
  const unsigned lane = threadIdx.x & 31;
  constexpr int kBatch = 2;
  for (uint32_t w0 = 0; w0 < windows; w0 += kBatch) {
    uint32_t slot[kBatch][2], base[kBatch][2];
    unsigned peers[kBatch][2];
    bool neg[kBatch][2];
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      const uint32_t w = w0 + k;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        slot[k][h] = kNoKey;
        neg[k][h] = false;
        peers[k][h] = 0;
        base[k][h] = 0;
        if (w < windows) {  // uniform across the warp
          if (live)
            slot[k][h] = rc[h].next_at(w, glv_window_pos(w, windows), glv_window_width(w, windows), half, flip[h],
                                       &neg[k][h]);
          peers[k][h] = slot_peers<AGG>(slot[k][h]);
          if (peers[k][h] && (int)lane == __ffs(peers[k][h]) - 1)
            base[k][h] = atomicAdd(&counts[slot[k][h]], (uint32_t)__popc(peers[k][h]));
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      const uint32_t w = w0 + k;
      if (w < windows) {
        uint32_t code[2], rank[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int leader = peers[k][h] ? __ffs(peers[k][h]) - 1 : (int)lane;
          const uint32_t b = __shfl_sync(0xffffffffu, base[k][h], leader);
          code[h] = peers[k][h] ? (slot[k][h] - w * half) | (neg[k][h] ? 0x8000u : 0u) : kRankZero;
          rank[h] = b + __popc(peers[k][h] & ((1u << lane) - 1));  // read only for a nonzero digit
        }
        if (live) {  // the halves side by side (msm_place), one store each for the pair
          const size_t e = (size_t)w * n + 2 * i;  // even (n = 2 scalar_n): 4- and 8-byte aligned stores
          __stcs(reinterpret_cast<uint32_t*>(digits + e), code[0] | code[1] << 16);
          __stcs(reinterpret_cast<uint2*>(ranks + e), make_uint2(rank[0], rank[1]));
        }
      }
    }
  }
}

// Grid (ceil(n / 256), windows): blockIdx.y is the window, so blocks run window by window.
// fixed: every window's digits share the buckets, and the entry names point w * n + i of a
// fixed-base table (2^(c w) P_i at row w). glv: column i holds half i & 1 of scalar i >> 1
// (msm_rank_glv), point (i >> 1) + (i & 1) n / 2.
// slot_start counts groups of 2^group_log places.
__global__ void msm_place(const uint16_t* __restrict__ digits, const uint32_t* __restrict__ ranks, size_t n,
                          uint32_t half, int fixed, int glv, const uint32_t* __restrict__ slot_start,
                          uint32_t group_log, uint32_t* __restrict__ sorted) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t w = blockIdx.y;
  const size_t e = (size_t)w * n + i;
  const uint32_t digit = __ldcs(digits + e);
  if (digit == kRankZero) return;
  const uint32_t slot = (fixed ? 0u : w * half) + (digit & 0x7fffu);
  const uint32_t point = fixed ? (uint32_t)e : glv ? (uint32_t)((i >> 1) + (i & 1) * (n >> 1)) : (uint32_t)i;
  sorted[(slot_start[slot] << group_log) + __ldcs(ranks + e)] = point | ((digit & 0x8000u) ? kNegBit : 0u);
}

// Fixed-base table: row w holds 2^(c w) P_i for every base i (affine, Montgomery form, infinity
// as zeros), rows 0..windows-1; an MSM over it needs no per-window buckets and no Horner
// combination. One thread per base: c doublings between rows, one inversion per row.
template <class F>
__global__ void msm_fixed_base_table(const uint32_t* __restrict__ bases, size_t n, uint32_t c, uint32_t windows,
                                     uint32_t* __restrict__ table) {
  constexpr int AW = PointWords<F>::affine;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Xyzz<F> acc = from_affine(load_affine<F>(bases + i * AW));
  for (uint32_t w = 0; w < windows; w++) {
    const Affine<F> a = to_affine(acc);
    uint32_t* o = table + ((size_t)w * n + i) * AW;
    store_elem(o, a.x);
    store_elem(o + AW / 2, a.y);
    if (w + 1 < windows)
      for (uint32_t k = 0; k < c; k++) acc = xyzz_double(acc);
  }
}

// ------------------------------------------------------------------ scan (3 phases)
//
// Over the slots' numbers of groups: a slot of k entries takes ceil(k / 2^group_log) groups of
// 2^group_log places in the sorted array (group_log = 0 without affine rounds: groups are entries).

__device__ __forceinline__ uint32_t groups_of(uint32_t entries, uint32_t group_log) {
  return (entries + (1u << group_log) - 1) >> group_log;
}

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total, uint32_t* warp_sums) {
  unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= (unsigned)d) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < blockDim.x / 32 ? warp_sums[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= (unsigned)d) s += y;
    }
    warp_sums[lane] = s;  // inclusive
  }
  __syncthreads();
  uint32_t before = warp ? warp_sums[warp - 1] : 0;
  *total = warp_sums[blockDim.x / 32 - 1];
  __syncthreads();
  return before + x - v;
}

// Also adds the entries themselves into *entries (zkg_msm_last_entries).
__global__ void __launch_bounds__(kScanBlock) scan_tile_sums(const uint32_t* __restrict__ in, size_t len,
                                                             uint32_t group_log, uint32_t* __restrict__ tile_sums,
                                                             uint32_t* __restrict__ entries) {
  __shared__ uint32_t warp_sums[32];
  size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t s = 0, raw = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++)
    if (base + k < len) {
      raw += in[base + k];
      s += groups_of(in[base + k], group_log);
    }
  raw = __reduce_add_sync(0xffffffffu, raw);
  if ((threadIdx.x & 31) == 0 && raw) atomicAdd(entries, raw);
  uint32_t total;
  block_exclusive_scan(s, &total, warp_sums);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Exclusive scan of the tile sums in place (tiles <= kScanTile), total into *grand.
__global__ void __launch_bounds__(kScanBlock) scan_tiles(uint32_t* __restrict__ tile_sums, uint32_t tiles,
                                                          uint32_t* __restrict__ grand) {
  __shared__ uint32_t warp_sums[32];
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    uint32_t idx = threadIdx.x * kScanItems + k;
    v[k] = idx < tiles ? tile_sums[idx] : 0;
    s += v[k];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(s, &total, warp_sums);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    uint32_t idx = threadIdx.x * kScanItems + k;
    if (idx < tiles) tile_sums[idx] = run;
    run += v[k];
  }
  if (threadIdx.x == 0) *grand = total;
}

// out[i] = exclusive prefix of the groups; also each slot's first place to out2 (the scatter cursor),
// and kPadEntry to the places of its last group that its entries leave free.
__global__ void __launch_bounds__(kScanBlock) scan_apply(const uint32_t* __restrict__ in, size_t len,
                                                         uint32_t group_log,
                                                         const uint32_t* __restrict__ tile_offsets,
                                                         uint32_t* __restrict__ out, uint32_t* __restrict__ out2,
                                                         uint32_t* __restrict__ sorted) {
  __shared__ uint32_t warp_sums[32];
  size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    v[k] = base + k < len ? in[base + k] : 0;
    s += groups_of(v[k], group_log);
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(s, &total, warp_sums) + tile_offsets[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const uint32_t next = run + groups_of(v[k], group_log);
    if (base + k < len) {
      out[base + k] = run;
      out2[base + k] = run << group_log;
      for (uint32_t e = (run << group_log) + v[k]; e < (next << group_log); e++) sorted[e] = kPadEntry;
    }
    run = next;
  }
}

// ------------------------------------------------------------------ accumulate

// Largest s in [lo, hi) with a[s] <= p, given a[lo] <= p < a[hi].
__device__ __forceinline__ uint32_t last_leq(const uint32_t* a, uint32_t lo, uint32_t hi, uint32_t p) {
  while (hi - lo > 1) {
    uint32_t mid = lo + (hi - lo) / 2;
    if (__ldg(&a[mid]) <= p) lo = mid;
    else hi = mid;
  }
  return lo;
}

// One thread per segment [t*L, t*L + L) of the sorted entries (all windows concatenated, slot
// order). slot_start has num_slots + 1 entries; slot_start[num_slots] = total entries.
// Points below `split` come from `bases`, the others from bases2 (point - split): the GLV
// entries' P_i and phi(P_i); plain plans pass split = 2^32 - 1. sorted = null: entry p is point p
// (the groups' sums that the affine rounds left, slot_start counting groups).
template <class F>
__global__ void __launch_bounds__(128) msm_accumulate(const uint32_t* __restrict__ bases,
                                                      const uint32_t* __restrict__ bases2, uint32_t split,
                                                      const uint32_t* __restrict__ sorted,
                                                      const uint32_t* __restrict__ slot_start, uint32_t num_slots,
                                                      uint32_t seg_len, uint32_t* __restrict__ buckets,
                                                      uint32_t* __restrict__ heads,
                                                      uint32_t* __restrict__ head_keys) {
  constexpr int XW = PointWords<F>::xyzz;
  const uint32_t total = __ldg(&slot_start[num_slots]);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t p0_64 = (uint64_t)t * seg_len;
  if (p0_64 >= total) return;
  const uint32_t p0 = (uint32_t)p0_64;
  const uint64_t e64 = p0_64 + seg_len;
  const uint32_t p1 = e64 < total ? (uint32_t)e64 : total;

  uint32_t s = last_leq(slot_start, 0, num_slots, p0);
  uint32_t end = __ldg(&slot_start[s + 1]);
  bool head = __ldg(&slot_start[s]) < p0;  // the slot began in an earlier segment
  uint32_t head_key = kNoKey;

  Xyzz<F> acc = xyzz_infinity<F>();
  // The next base is fetched into shared memory with cp.async while the current addition runs
  // (two slots per thread), so the prefetch holds no registers.
  constexpr int AW = PointWords<F>::affine;  // 16 (G1) or 32 (G2) words
  __shared__ __align__(16) uint32_t stage[2][128][AW];
  auto stage_base = [&](uint32_t slot, uint32_t e) {
    const uint32_t pt = e & ~kNegBit;
    const uint4* g = reinterpret_cast<const uint4*>(pt < split ? bases + (size_t)pt * AW
                                                               : bases2 + (size_t)(pt - split) * AW);
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(&stage[slot][threadIdx.x][0]);
#pragma unroll
    for (int k = 0; k < AW / 4; k++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa + 16 * k), "l"(g + k) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto entry_at = [&](uint32_t p) { return sorted ? __ldg(&sorted[p]) : p; };
  uint32_t entry = entry_at(p0);
  uint32_t cur_entry = entry, slot = 0;
  stage_base(0, entry);
  for (uint32_t p = p0; p < p1; p++) {
    if (p + 1 < p1) {
      entry = entry_at(p + 1);
      stage_base(slot ^ 1, entry);
      asm volatile("cp.async.wait_group 1;" ::: "memory");  // this point's copy has landed
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    Affine<F> cur = load_affine<F>(&stage[slot][threadIdx.x][0]);
    if (cur_entry & kNegBit) cur.y = neg(cur.y);
    cur_entry = entry;
    slot ^= 1;
    if (p == end) {  // slot s is complete; move to the slot that holds position p
      if (head) {
        store_xyzz(heads + (size_t)t * XW, acc);
        head_key = s;
        head = false;
      } else {
        store_xyzz(buckets + (size_t)s * XW, acc);
      }
      acc = xyzz_infinity<F>();
      uint32_t s2 = s + 1;
      if (__ldg(&slot_start[s2 + 1]) <= p) s2 = last_leq(slot_start, s2, num_slots, p);
      s = s2;
      end = __ldg(&slot_start[s + 1]);
    }
    acc = xyzz_add_affine(acc, cur);
  }
  if (head) {
    store_xyzz(heads + (size_t)t * XW, acc);
    head_key = s;
  } else {
    store_xyzz(buckets + (size_t)s * XW, acc);
  }
  head_keys[t] = head_key;
}

// ------------------------------------------------------------------ merge levels

// Heads of one block (a tile): 256 for G1, 128 for G2 (32 KiB of points).
template <class F>
struct MergeTile {
  static constexpr uint32_t value = PointWords<F>::xyzz == 32 ? 256 : 128;
};
constexpr uint32_t kMergeThreads = 128;

// Length of the head array at merge level `level` (level 0 = the accumulate output).
__device__ __forceinline__ uint32_t heads_len(uint32_t total, uint32_t seg_len, uint32_t tile, uint32_t level) {
  uint64_t len = ((uint64_t)total + seg_len - 1) / seg_len;
  for (uint32_t l = 0; l < level; l++) len = (len + tile - 1) / tile;
  return (uint32_t)len;
}

// One merge level: block u sums the runs of equal keys among heads [u T, u T + T). A run that starts
// there is added into its bucket; one that continues from the tile before becomes head u of the next
// level. One addition per bucket per level (only the tile where a run starts adds it), so a level
// needs no atomics.
//
// Within a run the sum is a tree: at step d the heads at offsets that are multiples of 2d take the one d
// further. Uniform scalars give runs of 4-5 heads, three steps; a bucket that fills the tile takes
// log2 T. A step's additions go a thread each when they are many (more than `few`), else a group of
// lanes each. Bound by the latency of the additions: the earlier levels of four heads per thread
// needed eight launches of four to five additions in a row for 49152 heads, this needs two.
template <class F>
__global__ void __launch_bounds__(kMergeThreads) msm_merge(const uint32_t* __restrict__ slot_start, uint32_t num_slots,
                                                           uint32_t seg_len, uint32_t level, uint32_t few,
                                                           const uint32_t* __restrict__ in_pts,
                                                           const uint32_t* __restrict__ in_keys,
                                                           uint32_t* __restrict__ out_pts,
                                                           uint32_t* __restrict__ out_keys,
                                                           uint32_t* __restrict__ buckets) {
  constexpr int XW = PointWords<F>::xyzz;
  constexpr uint32_t T = MergeTile<F>::value, kGroups = kMergeThreads / LaneGroup<F>::kLanes;
  extern __shared__ __align__(16) uint32_t merge_smem[];
  uint32_t* const pts = merge_smem;        // [T] points
  uint32_t* const keys = pts + T * XW;     // [T]
  uint32_t* const offset = keys + T;       // [T] offset within the run
  uint32_t* const work = offset + T;       // [T] the step's heads
  __shared__ uint32_t work_count;
  const uint32_t len = heads_len(__ldg(&slot_start[num_slots]), seg_len, T, level);
  const uint32_t u = blockIdx.x, base = u * T;
  if (len <= 1 || base >= len) return;  // the whole block
  const uint32_t n = min(T, len - base), group = threadIdx.x / LaneGroup<F>::kLanes;
  const uint32_t prev = base > 0 ? in_keys[base - 1] : kNoKey;
  for (uint32_t i = threadIdx.x; i < n; i += kMergeThreads) {
    const uint32_t k = in_keys[base + i];
    keys[i] = k;
    if (k != kNoKey) store_xyzz(pts + i * XW, load_xyzz<F>(in_pts + (size_t)(base + i) * XW));
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += kMergeThreads) {
    uint32_t o = 0;
    while (o < i && keys[i - o - 1] == keys[i]) o++;
    offset[i] = o;
  }
  // work[0 .. work_count) = the heads i < n that `pick` takes
  auto collect = [&](auto pick) {
    __syncthreads();
    if (threadIdx.x == 0) work_count = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kMergeThreads)
      if (keys[i] != kNoKey && pick(i)) work[atomicAdd(&work_count, 1u)] = i;
    __syncthreads();
    return work_count;
  };
  // target(i) += value(i) for the collected heads
  auto add_all = [&](uint32_t count, auto target, auto value) {
    if (count > few) {
      for (uint32_t j = threadIdx.x; j < count; j += kMergeThreads) {
        const uint32_t i = work[j];
        store_xyzz(target(i), xyzz_add(load_xyzz<F>(target(i)), load_xyzz<F>(value(i))));
      }
    } else {
      for (uint32_t j0 = 0; j0 < count; j0 += kGroups) {
        const bool active = j0 + group < count;
        const uint32_t i = work[active ? j0 + group : 0];
        lane_add<F>(active ? target(i) : pts + i * XW, active ? value(i) : pts + i * XW, target(i), active);
      }
    }
  };
  for (uint32_t d = 1; d < T; d <<= 1) {
    const uint32_t count = collect([&](uint32_t i) { return (offset[i] & (2 * d - 1)) == 0 && i + d < n && keys[i + d] == keys[i]; });
    if (count == 0) break;  // no run is longer than d
    add_all(count, [&](uint32_t i) { return pts + i * XW; }, [&](uint32_t i) { return pts + (i + d) * XW; });
  }
  const bool continued = keys[0] != kNoKey && keys[0] == prev;
  const uint32_t count = collect([&](uint32_t i) { return offset[i] == 0 && !(i == 0 && continued); });
  add_all(count, [&](uint32_t i) { return buckets + (size_t)keys[i] * XW; }, [&](uint32_t i) { return pts + i * XW; });
  if (continued && threadIdx.x < XW) out_pts[(size_t)u * XW + threadIdx.x] = pts[threadIdx.x];
  if (threadIdx.x == 0) out_keys[u] = continued ? keys[0] : kNoKey;
}

// ------------------------------------------------------------------ bucket reduction

// Sum of the n points (a power of two) in shared memory at sh, left in sh[0], by the whole block:
// halving levels, a thread per addition while there are at least kThreadAdds of them (G1; an Fq2
// addition takes a thread 18 us), a group of lanes per addition below (2 us, 2.6 us for G2, where a
// thread takes 6).
template <class F>
__device__ __forceinline__ void tree_sum(uint32_t* sh, uint32_t n) {
  constexpr int XW = PointWords<F>::xyzz;
  constexpr uint32_t kThreadAdds = XW == 32 ? 16 : 64;
  const uint32_t groups = blockDim.x / LaneGroup<F>::kLanes, group = threadIdx.x / LaneGroup<F>::kLanes;
  for (uint32_t h = n / 2; h >= 1; h >>= 1) {
    if (h >= kThreadAdds) {
      for (uint32_t i = threadIdx.x; i < h; i += blockDim.x)
        store_xyzz(sh + (size_t)i * XW, xyzz_add(load_xyzz<F>(sh + (size_t)i * XW), load_xyzz<F>(sh + (size_t)(i + h) * XW)));
    } else {
      for (uint32_t i0 = 0; i0 < h; i0 += groups) {
        const uint32_t i = i0 + group;
        const bool active = i < h;
        lane_add<F>(sh + (active ? i : 0) * XW, sh + (active ? i + h : 0) * XW, sh + (active ? i : 0) * XW, active);
      }
    }
    __syncthreads();
  }
}

// Level of the running-sum reduction. Per window w the input holds m values A_0..A_{m-1} at
// in + (w * in_stride + b) * XW; level 0 reads the buckets, where an empty slot (no entries)
// is the point at infinity. With chunk C = 2^chunk_log, chunk k of window w (b in [Ck, Ck + C)):
//   tot_k = sum_j (j+1) A_{Ck+j},  run_k = sum_j A_{Ck+j} -> run_out[w * run_stride + k - 1] (k >= 1).
// Block (w, j) covers chunks [jT, jT + T) of window w (T = kReduceThreads) and writes the sum of
// their tot_k to tot_out[w * tot_stride + j]: the window-sum stage then reads one point per
// block instead of one per chunk.
template <class F>
__global__ void __launch_bounds__(kReduceThreads) msm_reduce_level(const uint32_t* __restrict__ in, uint32_t in_stride,
                                                                   uint32_t m, uint32_t chunk_log,
                                                                   const uint32_t* __restrict__ slot_start,
                                                                   uint32_t* __restrict__ tot_out, uint32_t tot_stride,
                                                                   uint32_t* __restrict__ run_out, uint32_t run_stride) {
  constexpr int XW = PointWords<F>::xyzz;
  extern __shared__ __align__(16) uint32_t sh_words[];
  const uint32_t chunk = 1u << chunk_log;
  const uint32_t chunks = (m + chunk - 1) / chunk;
  const uint32_t w = blockIdx.y, j = blockIdx.x;
  const uint32_t k = j * kReduceThreads + threadIdx.x;
  Xyzz<F> run = xyzz_infinity<F>(), tot = xyzz_infinity<F>();
  if (k < chunks) {  // no early return: every thread takes part in the block sum below
    const uint32_t lo = k * chunk, hi = min(lo + chunk, m);
    for (uint32_t b = hi; b-- > lo;) {
      size_t slot = (size_t)w * in_stride + b;
      bool empty = slot_start && __ldg(&slot_start[slot]) == __ldg(&slot_start[slot + 1]);
      if (!empty) run = xyzz_add(run, load_xyzz<F>(in + slot * XW));
      tot = xyzz_add(tot, run);
    }
    if (k >= 1) store_xyzz(run_out + ((size_t)w * run_stride + k - 1) * XW, run);
  }
  store_xyzz(sh_words + threadIdx.x * XW, tot);
  __syncthreads();
  tree_sum<F>(sh_words, kReduceThreads);
  if (threadIdx.x < XW) tot_out[((size_t)w * tot_stride + j) * XW + threadIdx.x] = sh_words[threadIdx.x];
}


// The last level: S = sum_i (i + 1) A_i over m <= kMarginalMax values per window, by marginals. With i =
// l + 2^lo h, sum_i i A_i = sum_l l C_l + 2^lo sum_h h R_h, C_l the sum of column l and R_h of row h; and
// over the bits of l, sum_l l C_l = sum_k 2^k Z_k, Z_k the sum of the C_l whose l has bit k, likewise for
// h. So three launches: the columns and rows (each at most 64 values), the Z_k (at most 32 columns or
// rows each) and sum_l C_l (at most 64 columns), and the fold. All are trees, at most 2 log2(64) additions
// deep where running sums and a suffix scan over 256 threads made 26 additions, on one SM per window.
//
// A sum of points that a block forms: which values of a window's vector, and how many.
enum SubsetKind : uint32_t { kColumn, kRow, kBit, kAll };
struct Subset {
  SubsetKind kind;
  uint32_t arg, lo, m;  // column l, row h or bit k; columns = 2^lo; the vector's length
  __device__ __forceinline__ uint32_t size() const {
    const uint32_t cols = 1u << lo;
    switch (kind) {
      case kColumn: return arg < m ? (m - arg + cols - 1) >> lo : 0;
      case kRow: return min(cols, m - min(m, arg << lo));
      case kBit: {  // indices below m with bit arg set
        const uint32_t full = m >> (arg + 1), rest = m & ((2u << arg) - 1);
        return (full << arg) + (rest > (1u << arg) ? rest - (1u << arg) : 0);
      }
      default: return m;
    }
  }
  __device__ __forceinline__ uint32_t index(uint32_t e) const {
    switch (kind) {
      case kColumn: return arg + (e << lo);
      case kRow: return (arg << lo) + e;
      case kBit: return ((e >> arg) << (arg + 1)) | (1u << arg) | (e & ((1u << arg) - 1));
      default: return e;
    }
  }
};

// *out = the sum over the subset of the window's vector at `in`; a value whose slot is empty
// (slot_start, when given, has the window's slots) is the point at infinity. One block of at least
// PointWords<F>::xyzz threads.
template <class F>
__device__ __forceinline__ void subset_sum(const Subset& s, const uint32_t* __restrict__ in,
                                           const uint32_t* __restrict__ slot_start, uint32_t* __restrict__ out,
                                           uint32_t* sh) {
  constexpr int XW = PointWords<F>::xyzz;
  const uint32_t size = s.size();
  uint32_t n = 1;
  while (n < size && n < blockDim.x) n <<= 1;
  if (threadIdx.x < n) {
    Xyzz<F> v = xyzz_infinity<F>();
    for (uint32_t e = threadIdx.x; e < size; e += n) {
      const uint32_t i = s.index(e);
      if (slot_start && __ldg(&slot_start[i]) == __ldg(&slot_start[i + 1])) continue;
      v = xyzz_add(v, load_xyzz<F>(in + (size_t)i * XW));
    }
    store_xyzz(sh + (size_t)threadIdx.x * XW, v);
  }
  __syncthreads();
  tree_sum<F>(sh, n);
  if (threadIdx.x < XW) out[threadIdx.x] = sh[threadIdx.x];
}

// Threads of a subset's block: one warp for G1 (a window has at least 64 subsets), four for G2, whose
// additions take sixteen lanes.
template <class F>
struct SubsetThreads {
  static constexpr uint32_t value = PointWords<F>::xyzz == 32 ? 32 : 128;
};

// Grid (2^lo + rows + lv.count, windows): the columns and rows of the last level's vector, and each
// chunked level's block totals summed up; a window's results at marg + w * marg_stride points, columns
// first, then rows, then the levels.
template <class F>
__global__ void __launch_bounds__(SubsetThreads<F>::value)
    msm_marginals(const uint32_t* __restrict__ in, uint32_t in_stride, uint32_t m, uint32_t lo,
                  const uint32_t* __restrict__ slot_start, const uint32_t* __restrict__ tots, ReduceLevels lv,
                  uint32_t* __restrict__ marg, uint32_t marg_stride) {
  constexpr int XW = PointWords<F>::xyzz;
  __shared__ __align__(16) uint32_t sh[SubsetThreads<F>::value * XW];
  const uint32_t w = blockIdx.y, j = blockIdx.x, cols = 1u << lo, rows = (m + cols - 1) >> lo;
  uint32_t* const out = marg + ((size_t)w * marg_stride + j) * XW;
  if (j >= cols + rows) {
    const uint32_t l = j - cols - rows;
    subset_sum<F>(Subset{kAll, 0, 0, lv.tot_len[l]}, tots + ((size_t)lv.tot_offset[l] + (size_t)w * lv.tot_len[l]) * XW,
                  nullptr, out, sh);
    return;
  }
  subset_sum<F>(j < cols ? Subset{kColumn, j, lo, m} : Subset{kRow, j - cols, lo, m}, in + (size_t)w * in_stride * XW,
                slot_start ? slot_start + (size_t)w * in_stride : nullptr, out, sh);
}

// Grid (lo + hi + 1, windows): Z_k of the columns' bits, then of the rows', then the sum of all columns.
template <class F>
__global__ void __launch_bounds__(SubsetThreads<F>::value)
    msm_bit_sums(const uint32_t* __restrict__ marg, uint32_t marg_stride, uint32_t m, uint32_t lo, uint32_t hi,
                 uint32_t* __restrict__ bits) {
  constexpr int XW = PointWords<F>::xyzz;
  __shared__ __align__(16) uint32_t sh[SubsetThreads<F>::value * XW];
  const uint32_t w = blockIdx.y, k = blockIdx.x, cols = 1u << lo, rows = (m + cols - 1) >> lo;
  const uint32_t* const columns = marg + (size_t)w * marg_stride * XW;
  const bool high = k >= lo && k < lo + hi;
  const Subset s = k < lo ? Subset{kBit, k, 0, cols} : high ? Subset{kBit, k - lo, 0, rows} : Subset{kAll, 0, 0, cols};
  subset_sum<F>(s, high ? columns + (size_t)cols * XW : columns, nullptr, bits + ((size_t)w * (lo + hi + 1) + k) * XW, sh);
}

// part[0] <- sum_i 2^pos(i) part[i] over i < count, pos falling with i, by the whole block with one
// group of lanes (curve_lanes.cuh) a warp, at least count / 2 warps (all take part; a warp's other groups repeat
// its work). Neighbours meet pairwise, 2, 4, 8 .. values at a time from the top: the top value's
// doublings are the chain that any order has, but only log2 count additions lie on it.
template <class F, class Pos>
__device__ __forceinline__ void pairwise_horner(uint32_t (*part)[PointWords<F>::xyzz], uint32_t count, Pos pos) {
  const bool first = (threadIdx.x & 31) < LaneGroup<F, 2>::kLanes;
  const LaneRole<2> sm{lane_role<F, 2>()};
  for (uint32_t span = 1; span < count; span <<= 1) {
    __syncthreads();
    const uint32_t high = threadIdx.x / 32 * 2 * span, low = high + span;  // this warp's pair
    if (low >= count) continue;
    const uint32_t width = pos(low - 1) - pos(min(low + span, count) - 1);  // of the low part
    LaneChain<F> acc = lane_chain<F>(part[high], sm);
    for (uint32_t k = 0; k < width; k++) acc = lane_double(acc, sm);
    __syncwarp();
    lane_store<2>(part[high], acc, first);
    __syncwarp();
    lane_add<F, 2>(part[high], part[low], part[high], first);
  }
  __syncthreads();
}

// S_w from the Z_k and the sum of all values; then for each chunked level, from the last one down,
// S = 2^chunk_log S + its total. Four groups of lanes that ran Horner over a share of the bits each
// took six additions where four are left now: window sums of 12 G1 windows 0.097 ms, now 0.089, of 24 G2 windows
// 0.265, now 0.253.
constexpr uint32_t kFoldValues = 14;  // kMarginalMax has 12 bits
template <class F>
__global__ void __launch_bounds__(kFoldValues / 2 * 32)
    msm_window_fold(const uint32_t* __restrict__ bits, uint32_t bit_count, const uint32_t* __restrict__ totals,
                    uint32_t totals_stride, uint32_t levels, uint32_t chunk_log, uint32_t* __restrict__ window_sums) {
  constexpr int XW = PointWords<F>::xyzz;
  __shared__ __align__(16) uint32_t part[kFoldValues][XW];  // Z_k from the top bit down, the sum of all
  const uint32_t w = blockIdx.x;
  const uint32_t* const z = bits + (size_t)w * (bit_count + 1) * XW;
  for (uint32_t i = threadIdx.x; i < (bit_count + 1) * XW; i += blockDim.x) {
    const uint32_t k = i / XW;
    part[k == bit_count ? k : bit_count - 1 - k][i % XW] = z[i];
  }
  pairwise_horner<F>(part, bit_count + 1, [&](uint32_t i) { return i == bit_count ? 0 : bit_count - 1 - i; });
  if (threadIdx.x >= 32) return;
  const bool first = threadIdx.x < LaneGroup<F, 2>::kLanes;
  const LaneRole<2> role{lane_role<F, 2>()};
  for (uint32_t l = levels; l-- > 0;) {
    LaneChain<F> v = lane_chain<F>(part[0], role);
    for (uint32_t d = 0; d < chunk_log; d++) v = lane_double(v, role);
    __syncwarp();
    lane_store<2>(part[0], v, first);
    __syncwarp();
    lane_add<F, 2>(part[0], totals + ((size_t)w * totals_stride + l) * XW, part[0], first);
    __syncwarp();
  }
  for (uint32_t i = threadIdx.x; i < XW; i += 32) window_sums[(size_t)w * XW + i] = part[0][i];
}

// result = sum_w 2^(pos_w) S_w (msm_combine.wgsl:13-22), a warp for each pair of windows. Window w is `base`
// bits wide, or base + 1 for w < extra (pos_w is the sum of the widths below w): base = c, extra = 0
// for the plain windows, the glv_window_width split for GLV. Bound by the latency of the doublings'
// products; one chain (Horner) took W - 1 additions, 5.7 us each with their start of a chain (G2
// 8.9): G1 of 12 windows 0.169 ms, now 0.155, G2 of 24 0.495, now 0.440.
// WARPS bounds the block, and with it the registers. An Fq2 chain wants more than the 128 that 16 warps
// leave (192 bytes of spills stored, 76 loaded); bound to the 12 that the default windows take, it has 168
// and reloads nothing: G2 2^14 1076 us, 1080 before. G1 takes 88 of the 128, and bound to 12 its schedule is
// the slower (G1 of 1000 points 386 us against 383.4), so it keeps one form.
constexpr uint32_t kCombineWindows = 32;  // 255 bits in windows of 9, at most
template <class F>
struct CombineWarps {
  static constexpr uint32_t value = PointWords<F>::xyzz == 32 ? kCombineWindows / 2 : 12;
};
template <class F, uint32_t WARPS>
__global__ void __launch_bounds__(WARPS * 32)
    msm_combine_lanes(const uint32_t* __restrict__ window_sums, uint32_t windows, uint32_t base, uint32_t extra,
                      uint32_t* __restrict__ result) {
  constexpr int XW = PointWords<F>::xyzz;
  __shared__ __align__(16) uint32_t part[kCombineWindows][XW];  // from the top window down
  for (uint32_t i = threadIdx.x; i < windows * XW; i += blockDim.x) part[windows - 1 - i / XW][i % XW] = window_sums[i];
  pairwise_horner<F>(part, windows, [&](uint32_t i) { return (windows - 1 - i) * base + min(windows - 1 - i, extra); });
  for (uint32_t i = threadIdx.x; i < XW; i += blockDim.x) result[i] = part[0][i];
}

// result <- result + partial (XYZZ, one thread): the passes of a run over more points than one
// pass holds.
template <class F>
__global__ void msm_add_partial(uint32_t* __restrict__ result, const uint32_t* __restrict__ partial) {
  if (threadIdx.x != 0) return;
  store_xyzz(result, xyzz_add(load_xyzz<F>(result), load_xyzz<F>(partial)));
}

// ------------------------------------------------------------------ base upload

// x <- x * scale / 2^256 for every 8-word Fq coordinate (to_montgomery.wgsl:6-15). With
// scale = 2^512 mod q this maps plain coordinates to Montgomery form; (0,0) stays (0,0).
__global__ void fq_rescale(uint32_t* __restrict__ coords, size_t count, Fq scale) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  store_fe(coords + 8 * i, load_fe<Fq>(coords + 8 * i) * scale);
}

}  // namespace zkg
