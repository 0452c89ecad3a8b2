// BN254 base field Fq and scalar field Fr on sm_100a: 8 x 32-bit limbs, Montgomery radix
// R = 2^256, products on the integer multiply-add pipe (mad.wide.u32) with PTX carry chains
// (add.cc / addc) for the accumulation. No tensor cores: this is exact modular integer
// arithmetic.
//
// Replaces the reference's generated WGSL field code (src/field.rs:55-181: 20 x 13-bit limbs,
// R = 2^260, deferred carries). Memory format is unchanged: 8 little-endian u32 words per
// element (src/field.rs:63-93). Values in memory, and those that are compared, are fully reduced
// (< p), so equality and zero tests are word compares; operands that a function takes or leaves
// unreduced have their bounds stated at it.
#pragma once
#include <cstdint>

namespace zkg {

// Modulus parameters. INV = -p^-1 mod 2^32; ONE = 2^256 mod p (Montgomery one);
// R2 = 2^512 mod p (to_montgomery multiplier).
struct FqParams {
  static constexpr bool kCompact = false;
  static constexpr bool kPairs = false;
  static constexpr bool kLazy = false;
  static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u;
  static constexpr uint32_t P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xe4866389u;
  static constexpr uint32_t ONE0 = 0xc58f0d9du, ONE1 = 0xd35d438du, ONE2 = 0xf5c70b3du, ONE3 = 0x0a78eb28u;
  static constexpr uint32_t ONE4 = 0x7879462cu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
};

struct FrParams {
  static constexpr bool kCompact = false;
  static constexpr bool kPairs = false;
  static constexpr bool kLazy = false;
  static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u;
  static constexpr uint32_t P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xefffffffu;
  static constexpr uint32_t ONE0 = 0x4ffffffbu, ONE1 = 0xac96341cu, ONE2 = 0x9f60cd29u, ONE3 = 0x36fc7695u;
  static constexpr uint32_t ONE4 = 0x7879462eu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
};

// Same field, products through one out-of-line function instead of inlined copies. Kernels
// where few warps run long serial chains (merge, bucket reduction, window combination) use
// it: a fully inlined point addition is thousands of instructions, and a lone warp walking
// through straight-line code that size waits on instruction fetch rather than arithmetic.
struct FqCompactParams : FqParams {
  static constexpr bool kCompact = true;
};

// Compact, and independent products go two per call (mul2): shorter dependency waits for a
// lone thread, more registers per thread.
struct FqCompactPairParams : FqParams {
  static constexpr bool kCompact = true;
  static constexpr bool kPairs = true;
};

// Compact, and Fq2 products with one reduction per component (fq2_mul): the form of the G2 kernels
// where throughput counts.
struct FqLazyParams : FqParams {
  static constexpr bool kCompact = true;
  static constexpr bool kLazy = true;
};

template <class P>
struct Fp {
  static constexpr bool kLazy = P::kLazy;
  uint32_t w[8];

  __device__ __forceinline__ static Fp zero() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.w[i] = 0;
    return r;
  }
  __device__ __forceinline__ static Fp one() {
    Fp r;
    r.w[0] = P::ONE0; r.w[1] = P::ONE1; r.w[2] = P::ONE2; r.w[3] = P::ONE3;
    r.w[4] = P::ONE4; r.w[5] = P::ONE5; r.w[6] = P::ONE6; r.w[7] = P::ONE7;
    return r;
  }
  __device__ __forceinline__ bool is_zero() const {
    uint32_t x = w[0] | w[1] | w[2] | w[3] | w[4] | w[5] | w[6] | w[7];
    return x == 0;
  }
  __device__ __forceinline__ bool operator==(const Fp& o) const {
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) x |= w[i] ^ o.w[i];
    return x == 0;
  }
  __device__ __forceinline__ bool operator!=(const Fp& o) const { return !(*this == o); }
};

using Fq = Fp<FqParams>;
using Fr = Fp<FrParams>;
using FqC = Fp<FqCompactParams>;
using FqCP = Fp<FqCompactPairParams>;
using FqL = Fp<FqLazyParams>;

// ------------------------------------------------------------------ add / sub

// r = a + b mod p. Both < p < 2^254, so a + b < 2^255 never carries out of 8 words.
template <class P>
__device__ __forceinline__ Fp<P> operator+(const Fp<P>& a, const Fp<P>& b) {
  Fp<P> s, d;
  uint32_t borrow;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=&r"(s.w[0]), "=&r"(s.w[1]), "=&r"(s.w[2]), "=&r"(s.w[3]), "=&r"(s.w[4]), "=&r"(s.w[5]), "=&r"(s.w[6]),
        "=&r"(s.w[7])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
        "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]));
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=&r"(d.w[0]), "=&r"(d.w[1]), "=&r"(d.w[2]), "=&r"(d.w[3]), "=&r"(d.w[4]), "=&r"(d.w[5]), "=&r"(d.w[6]),
        "=&r"(d.w[7]), "=&r"(borrow)
      : "r"(s.w[0]), "r"(s.w[1]), "r"(s.w[2]), "r"(s.w[3]), "r"(s.w[4]), "r"(s.w[5]), "r"(s.w[6]), "r"(s.w[7]),
        "n"(P::P0), "n"(P::P1), "n"(P::P2), "n"(P::P3), "n"(P::P4), "n"(P::P5), "n"(P::P6), "n"(P::P7));
  // borrow = 0xffffffff when s < p: keep s; otherwise take s - p.
  Fp<P> r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.w[i] = (s.w[i] & borrow) | (d.w[i] & ~borrow);
  return r;
}

// r = a - b mod p: subtract, then add p back under the borrow mask.
template <class P>
__device__ __forceinline__ Fp<P> operator-(const Fp<P>& a, const Fp<P>& b) {
  Fp<P> d, r;
  uint32_t borrow;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=&r"(d.w[0]), "=&r"(d.w[1]), "=&r"(d.w[2]), "=&r"(d.w[3]), "=&r"(d.w[4]), "=&r"(d.w[5]), "=&r"(d.w[6]),
        "=&r"(d.w[7]), "=&r"(borrow)
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
        "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]));
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]),
        "=&r"(r.w[7])
      : "r"(d.w[0]), "r"(d.w[1]), "r"(d.w[2]), "r"(d.w[3]), "r"(d.w[4]), "r"(d.w[5]), "r"(d.w[6]), "r"(d.w[7]),
        "r"(P::P0 & borrow), "r"(P::P1 & borrow), "r"(P::P2 & borrow), "r"(P::P3 & borrow), "r"(P::P4 & borrow),
        "r"(P::P5 & borrow), "r"(P::P6 & borrow), "r"(P::P7 & borrow));
  return r;
}

template <class P>
__device__ __forceinline__ Fp<P> neg(const Fp<P>& a) {
  return Fp<P>::zero() - a;
}

template <class P>
__device__ __forceinline__ Fp<P> dbl(const Fp<P>& a) {
  return a + a;
}

// ------------------------------------------------------------------ Montgomery product
//
// Operand scanning (Koc, Acar and Kaliski, "Analyzing and comparing Montgomery multiplication
// algorithms", 1996) with 32x32 -> 64-bit products held as two interleaved accumulators: `e` sums
// the products whose low word falls on an even position and `o` those on an odd one, so every
// product is added to an aligned pair of words and consecutive products of one accumulator
// continue each other's carry chain. A mad.lo.cc / madc.hi.cc pair on such a pair of words is one
// wide multiply-add with carry in and out; the earlier forms (products first, then chains of
// add.cc over their halves) needed about 450 warp instructions per product, this one about 190:
// 128 wide multiply-adds, 8 multiples m = t_0 INV and the carries. The wide multiply-add issues at
// half rate, so 132 full-rate slots of that pipe bound it. Measured on B200: 68 G products/s (the
// pipe's limit) from two warps per scheduler on, 428 ns for a lone warp (422 before the last
// subtraction of p); before, 49.8 G/s and 518 ns.
//
// After the multiply row and the reduction row of word i, word 0 is zero and the value moves one
// word down: `o` becomes the even accumulator, and e[1] is added into its word 0 with the carry
// entering the odd chain, which starts at word 1. With a, b < 2^255 the running value stays below
// 2^288 (p < 2^254), so the odd chains never carry out of word 9.

// acc += (x0 + x1 2^64 + x2 2^128 + x3 2^192) y, the carry out added to cy.
__device__ __forceinline__ void mad4_carry(uint32_t (&c)[8], uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                           uint32_t y, uint32_t& cy) {
  asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32       %8, %8, 0;"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]), "+r"(cy)
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}

// acc += (x0 + x1 2^64 + x2 2^128 + x3 2^192) y where the sum fits.
__device__ __forceinline__ void mad4(uint32_t (&c)[8], uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                     uint32_t y) {
  asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32    %7, %11, %12, %7;"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7])
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}

// The word shifted out of the even accumulator joins the new even word e0, its carry entering the
// odd chain o += (x0 + ... + x3 2^192) y, whose top pair is fresh.
__device__ __forceinline__ void mad4_shift(uint32_t (&o)[8], uint32_t& e0, uint32_t out, uint32_t x0, uint32_t x1,
                                           uint32_t x2, uint32_t x3, uint32_t y) {
  asm("add.cc.u32     %8, %8, %14;\n\t"
      "madc.lo.cc.u32 %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, 0;\n\t"
      "madc.hi.u32    %7, %12, %13, 0;"
      : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "=&r"(o[6]), "=&r"(o[7]), "+r"(e0)
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y), "r"(out));
}

// (x0 + x1 2^64 + x2 2^128 + x3 2^192) y.
__device__ __forceinline__ void mul4(uint32_t (&c)[8], uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                     uint32_t y) {
  const uint32_t x[4] = {x0, x1, x2, x3};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint64_t t = (uint64_t)x[j] * y;
    c[2 * j] = (uint32_t)t;
    c[2 * j + 1] = (uint32_t)(t >> 32);
  }
}

// x - p when x >= p, else x (x < 2p).
template <class P>
__device__ __forceinline__ Fp<P> reduce_once(const Fp<P>& x) {
  Fp<P> d, r;
  uint32_t borrow;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=&r"(d.w[0]), "=&r"(d.w[1]), "=&r"(d.w[2]), "=&r"(d.w[3]), "=&r"(d.w[4]), "=&r"(d.w[5]), "=&r"(d.w[6]),
        "=&r"(d.w[7]), "=&r"(borrow)
      : "r"(x.w[0]), "r"(x.w[1]), "r"(x.w[2]), "r"(x.w[3]), "r"(x.w[4]), "r"(x.w[5]), "r"(x.w[6]), "r"(x.w[7]),
        "n"(P::P0), "n"(P::P1), "n"(P::P2), "n"(P::P3), "n"(P::P4), "n"(P::P5), "n"(P::P6), "n"(P::P7));
#pragma unroll
  for (int i = 0; i < 8; i++) r.w[i] = borrow ? x.w[i] : d.w[i];
  return r;
}

// The accumulators' value after the last row: o[k] at word k, e[k + 1] at word k (e[0] = 0).
template <class P>
__device__ __forceinline__ Fp<P> join(const uint32_t (&e)[8], const uint32_t (&o)[8]) {
  Fp<P> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, 0;"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]),
        "=&r"(r.w[7])
      : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(e[1]), "r"(e[2]),
        "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]));
  return r;
}

// a b 2^-256 mod p up to one p: below (a b + p 2^256) / 2^256, so below 2p for a, b < 2p.
template <class P>
__device__ __forceinline__ Fp<P> mont_mul_lazy(const Fp<P>& a, const Fp<P>& b) {
  constexpr uint32_t q[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  uint32_t acc[2][8];  // the even accumulator is acc[i & 1] in row i
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t(&e)[8] = acc[i & 1];
    uint32_t(&o)[8] = acc[(i & 1) ^ 1];
    if (i == 0) {
      mul4(e, a.w[0], a.w[2], a.w[4], a.w[6], b.w[0]);
      mul4(o, a.w[1], a.w[3], a.w[5], a.w[7], b.w[0]);
    } else {
      const uint32_t out = o[1];  // o was the even accumulator: drop its two low words
#pragma unroll
      for (int k = 0; k < 6; k++) o[k] = o[k + 2];
      mad4_shift(o, e[0], out, a.w[1], a.w[3], a.w[5], a.w[7], b.w[i]);
      mad4_carry(e, a.w[0], a.w[2], a.w[4], a.w[6], b.w[i], o[7]);
    }
    const uint32_t m = e[0] * P::INV;
    mad4_carry(e, q[0], q[2], q[4], q[6], m, o[7]);
    mad4(o, q[1], q[3], q[5], q[7], m);
  }
  return join<P>(acc[1], acc[0]);
}

// The reduction rows alone, of a value held in the two accumulators (e = acc[0], word k at e[k]; o =
// acc[1], word k + 1 at o[k], o[7] = 0): (value + m p) 2^-256 for the m < 2^256 that makes it whole.
template <class P>
__device__ __forceinline__ Fp<P> mont_rows(uint32_t (&acc)[2][8]) {
  constexpr uint32_t q[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t(&e)[8] = acc[i & 1];
    uint32_t(&o)[8] = acc[(i & 1) ^ 1];
    if (i == 0) {
      const uint32_t m = e[0] * P::INV;
      mad4_carry(e, q[0], q[2], q[4], q[6], m, o[7]);
      mad4(o, q[1], q[3], q[5], q[7], m);
    } else {
      const uint32_t out = o[1];
#pragma unroll
      for (int k = 0; k < 6; k++) o[k] = o[k + 2];
      const uint32_t m = (e[0] + out) * P::INV;
      mad4_shift(o, e[0], out, q[1], q[3], q[5], q[7], m);
      mad4_carry(e, q[0], q[2], q[4], q[6], m, o[7]);
    }
  }
  return join<P>(acc[1], acc[0]);
}

// c += (x[0] + x[1] 2^64 + ...) y over N pairs of words, a chain of one row of a square. The one word
// that the chain is the first to reach is written, not added to: the carry word past its last pair,
// or (top_fresh) the high word of the last pair, which the sum does not overflow.
template <int N>
__device__ __forceinline__ void sqr_chain(uint32_t* c, const uint32_t (&x)[N], uint32_t y, bool top_fresh) {
  static_assert(N >= 1 && N <= 4, "chain of one to four products");
  if constexpr (N == 1) {
    if (top_fresh)
      asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, 0;" : "+r"(c[0]), "=&r"(c[1]) : "r"(x[0]), "r"(y));
    else
      asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 %2, 0, 0;"
          : "+r"(c[0]), "+r"(c[1]), "=&r"(c[2]) : "r"(x[0]), "r"(y));
  } else if constexpr (N == 2) {
    if (top_fresh)
      asm("mad.lo.cc.u32 %0, %4, %6, %0;\n\tmadc.hi.cc.u32 %1, %4, %6, %1;\n\t"
          "madc.lo.cc.u32 %2, %5, %6, %2;\n\tmadc.hi.u32 %3, %5, %6, 0;"
          : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "=&r"(c[3]) : "r"(x[0]), "r"(x[1]), "r"(y));
    else
      asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\tmadc.hi.cc.u32 %1, %5, %7, %1;\n\t"
          "madc.lo.cc.u32 %2, %6, %7, %2;\n\tmadc.hi.cc.u32 %3, %6, %7, %3;\n\taddc.u32 %4, 0, 0;"
          : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "=&r"(c[4]) : "r"(x[0]), "r"(x[1]), "r"(y));
  } else if constexpr (N == 3) {
    if (top_fresh)
      asm("mad.lo.cc.u32 %0, %6, %9, %0;\n\tmadc.hi.cc.u32 %1, %6, %9, %1;\n\t"
          "madc.lo.cc.u32 %2, %7, %9, %2;\n\tmadc.hi.cc.u32 %3, %7, %9, %3;\n\t"
          "madc.lo.cc.u32 %4, %8, %9, %4;\n\tmadc.hi.u32 %5, %8, %9, 0;"
          : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "=&r"(c[5])
          : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(y));
    else
      asm("mad.lo.cc.u32 %0, %7, %10, %0;\n\tmadc.hi.cc.u32 %1, %7, %10, %1;\n\t"
          "madc.lo.cc.u32 %2, %8, %10, %2;\n\tmadc.hi.cc.u32 %3, %8, %10, %3;\n\t"
          "madc.lo.cc.u32 %4, %9, %10, %4;\n\tmadc.hi.cc.u32 %5, %9, %10, %5;\n\taddc.u32 %6, 0, 0;"
          : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "=&r"(c[6])
          : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(y));
  } else {  // both words of the longest chain's last pair are fresh
    asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\tmadc.hi.cc.u32 %1, %8, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %12, %2;\n\tmadc.hi.cc.u32 %3, %9, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %12, %4;\n\tmadc.hi.cc.u32 %5, %10, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %12, 0;\n\tmadc.hi.u32 %7, %11, %12, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "=&r"(c[6]), "=&r"(c[7])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y));
  }
}

// a^2 2^-256 mod p up to one p (a < 2^255): 36 products of words (each cross product once, with one
// factor doubled) and the reduction rows over the low half, 100 wide multiply-adds against 128:
// 78.6 G/s, 356 ns for a lone warp (product: 68.1 G/s, 422 ns).
template <class P>
__device__ __forceinline__ Fp<P> mont_sqr_lazy(const Fp<P>& a) {
  const uint32_t* w = a.w;
  // d = 2a; s_j = 2 a_j without the bit that a_{j-1} shifts in (the first cross product of row j - 1,
  // whose factor starts at word j)
  uint32_t d[8];
#pragma unroll
  for (int j = 1; j < 8; j++) d[j] = __funnelshift_l(w[j - 1], w[j], 1);
  uint32_t ev[16], od[16];
  mul4(reinterpret_cast<uint32_t(&)[8]>(ev[0]), w[0], d[2], d[4], d[6], w[0]);
  mul4(reinterpret_cast<uint32_t(&)[8]>(od[0]), w[1] << 1, d[3], d[5], d[7], w[0]);
  sqr_chain<4>(ev + 2, {w[1], d[3], d[5], d[7]}, w[1], true);
  sqr_chain<3>(od + 2, {w[2] << 1, d[4], d[6]}, w[1], false);
  sqr_chain<3>(ev + 4, {w[2], d[4], d[6]}, w[2], false);
  sqr_chain<3>(od + 4, {w[3] << 1, d[5], d[7]}, w[2], true);
  sqr_chain<3>(ev + 6, {w[3], d[5], d[7]}, w[3], true);
  sqr_chain<2>(od + 6, {w[4] << 1, d[6]}, w[3], false);
  sqr_chain<2>(ev + 8, {w[4], d[6]}, w[4], false);
  sqr_chain<2>(od + 8, {w[5] << 1, d[7]}, w[4], true);
  sqr_chain<2>(ev + 10, {w[5], d[7]}, w[5], true);
  sqr_chain<1>(od + 10, {w[6] << 1}, w[5], false);
  sqr_chain<1>(ev + 12, {w[6]}, w[6], false);
  sqr_chain<1>(od + 12, {w[7] << 1}, w[6], true);
  sqr_chain<1>(ev + 14, {w[7]}, w[7], true);
  // words 0..7 (ev[0..7], od[0..6]) through the rows, then words 8..15 (ev[8..15], od[7..13])
  uint32_t acc[2][8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    acc[0][k] = ev[k];
    acc[1][k] = k < 7 ? od[k] : 0;
  }
  const Fp<P> lo = mont_rows<P>(acc);
  Fp<P> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, 0;"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]),
        "=&r"(r.w[7])
      : "r"(ev[8]), "r"(ev[9]), "r"(ev[10]), "r"(ev[11]), "r"(ev[12]), "r"(ev[13]), "r"(ev[14]), "r"(ev[15]),
        "r"(od[7]), "r"(od[8]), "r"(od[9]), "r"(od[10]), "r"(od[11]), "r"(od[12]), "r"(od[13]));
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]), "+r"(r.w[6]), "+r"(r.w[7])
      : "r"(lo.w[0]), "r"(lo.w[1]), "r"(lo.w[2]), "r"(lo.w[3]), "r"(lo.w[4]), "r"(lo.w[5]), "r"(lo.w[6]), "r"(lo.w[7]));
  return r;
}

// p - a for a <= p (p for a = 0).
template <class P>
__device__ __forceinline__ Fp<P> complement(const Fp<P>& a) {
  Fp<P> r;
  asm("sub.cc.u32  %0, %16, %8;\n\t"
      "subc.cc.u32 %1, %17, %9;\n\t"
      "subc.cc.u32 %2, %18, %10;\n\t"
      "subc.cc.u32 %3, %19, %11;\n\t"
      "subc.cc.u32 %4, %20, %12;\n\t"
      "subc.cc.u32 %5, %21, %13;\n\t"
      "subc.cc.u32 %6, %22, %14;\n\t"
      "subc.u32    %7, %23, %15;"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]),
        "=&r"(r.w[7])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
        "r"(P::P0), "r"(P::P1), "r"(P::P2), "r"(P::P3), "r"(P::P4), "r"(P::P5), "r"(P::P6), "r"(P::P7));
  return r;
}

// (a b + c d) 2^-256 mod p up to one p, both products through one reduction (192 wide
// multiply-adds against 256; 45.7 G/s): below (a b + c d) 2^-256 + p, so below 2p for operands up
// to p.
template <class P>
__device__ __forceinline__ Fp<P> mont_mul_add_lazy(const Fp<P>& a, const Fp<P>& b, const Fp<P>& c, const Fp<P>& d) {
  constexpr uint32_t q[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  uint32_t acc[2][8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t(&e)[8] = acc[i & 1];
    uint32_t(&o)[8] = acc[(i & 1) ^ 1];
    if (i == 0) {
      mul4(e, a.w[0], a.w[2], a.w[4], a.w[6], b.w[0]);
      mul4(o, a.w[1], a.w[3], a.w[5], a.w[7], b.w[0]);
    } else {
      const uint32_t out = o[1];
#pragma unroll
      for (int k = 0; k < 6; k++) o[k] = o[k + 2];
      mad4_shift(o, e[0], out, a.w[1], a.w[3], a.w[5], a.w[7], b.w[i]);
      mad4_carry(e, a.w[0], a.w[2], a.w[4], a.w[6], b.w[i], o[7]);
    }
    mad4_carry(e, c.w[0], c.w[2], c.w[4], c.w[6], d.w[i], o[7]);
    mad4(o, c.w[1], c.w[3], c.w[5], c.w[7], d.w[i]);
    const uint32_t m = e[0] * P::INV;
    mad4_carry(e, q[0], q[2], q[4], q[6], m, o[7]);
    mad4(o, q[1], q[3], q[5], q[7], m);
  }
  return join<P>(acc[1], acc[0]);
}

// The product the library uses, fully reduced.
template <class P>
__device__ __forceinline__ Fp<P> mont_mul_prod(const Fp<P>& a, const Fp<P>& b) {
  return reduce_once(mont_mul_lazy(a, b));
}
template <class P>
__device__ __forceinline__ Fp<P> mont_sqr_prod(const Fp<P>& a) {
  return reduce_once(mont_sqr_lazy(a));
}
// a b - c d, fully reduced, for fully reduced operands.
template <class P>
__device__ __forceinline__ Fp<P> mont_mul_sub_prod(const Fp<P>& a, const Fp<P>& b, const Fp<P>& c, const Fp<P>& d) {
  return reduce_once(mont_mul_add_lazy(a, b, complement(c), d));
}

// ------------------------------------------------------------------ 512-bit products
//
// For Fq2, whose products have sums of products for components: three products of 64 wide
// multiply-adds (Karatsuba) and one reduction per component.

// acc += (x0 + ... + x3 2^192) y, the carry out to the fresh word c[8].
__device__ __forceinline__ void mad4_carry_fresh(uint32_t* c, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                                 uint32_t y) {
  asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32       %8, 0, 0;"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]), "=&r"(c[8])
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}
// The same with the last pair's high word c[7] fresh (the sum does not overflow it).
__device__ __forceinline__ void mad4_top_fresh(uint32_t* c, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                               uint32_t y) {
  asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32    %7, %11, %12, 0;"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "=&r"(c[7])
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}

struct Wide {
  uint32_t w[16];
};

// a +- b modulo 2^512, word chains in one piece each.
#define ZKG_WIDE_CHAIN(OP0, OP, a, b)                                                                       \
  asm(OP0 ".cc.u32 %0, %0, %16;\n\t" OP ".cc.u32 %1, %1, %17;\n\t" OP ".cc.u32 %2, %2, %18;\n\t"             \
      OP ".cc.u32 %3, %3, %19;\n\t" OP ".cc.u32 %4, %4, %20;\n\t" OP ".cc.u32 %5, %5, %21;\n\t"              \
      OP ".cc.u32 %6, %6, %22;\n\t" OP ".cc.u32 %7, %7, %23;\n\t" OP ".cc.u32 %8, %8, %24;\n\t"              \
      OP ".cc.u32 %9, %9, %25;\n\t" OP ".cc.u32 %10, %10, %26;\n\t" OP ".cc.u32 %11, %11, %27;\n\t"          \
      OP ".cc.u32 %12, %12, %28;\n\t" OP ".cc.u32 %13, %13, %29;\n\t" OP ".cc.u32 %14, %14, %30;\n\t"        \
      OP ".u32 %15, %15, %31;"                                                                                \
      : "+r"((a)[0]), "+r"((a)[1]), "+r"((a)[2]), "+r"((a)[3]), "+r"((a)[4]), "+r"((a)[5]), "+r"((a)[6]),      \
        "+r"((a)[7]), "+r"((a)[8]), "+r"((a)[9]), "+r"((a)[10]), "+r"((a)[11]), "+r"((a)[12]), "+r"((a)[13]), \
        "+r"((a)[14]), "+r"((a)[15])                                                                          \
      : "r"((b)[0]), "r"((b)[1]), "r"((b)[2]), "r"((b)[3]), "r"((b)[4]), "r"((b)[5]), "r"((b)[6]), "r"((b)[7]), \
        "r"((b)[8]), "r"((b)[9]), "r"((b)[10]), "r"((b)[11]), "r"((b)[12]), "r"((b)[13]), "r"((b)[14]),       \
        "r"((b)[15]))
__device__ __forceinline__ void wide_add(Wide& a, const Wide& b) { ZKG_WIDE_CHAIN("add", "addc", a.w, b.w); }
__device__ __forceinline__ void wide_sub(Wide& a, const Wide& b) { ZKG_WIDE_CHAIN("sub", "subc", a.w, b.w); }

// a b: even chains at even words in ev, odd chains one word up in od.
__device__ __forceinline__ Wide wide_mul(const uint32_t (&a)[8], const uint32_t (&b)[8]) {
  Wide ev, od;
  mul4(reinterpret_cast<uint32_t(&)[8]>(ev.w[0]), a[0], a[2], a[4], a[6], b[0]);
  mul4(reinterpret_cast<uint32_t(&)[8]>(od.w[1]), a[1], a[3], a[5], a[7], b[0]);
#pragma unroll
  for (int i = 1; i < 8; i++) {
    if (i & 1) {  // the odd words of a meet even words
      if (i == 1) sqr_chain<4>(ev.w + 2, {a[1], a[3], a[5], a[7]}, b[i], true);
      else mad4_top_fresh(ev.w + i + 1, a[1], a[3], a[5], a[7], b[i]);
      mad4_carry_fresh(od.w + i, a[0], a[2], a[4], a[6], b[i]);
    } else {
      mad4_carry_fresh(ev.w + i, a[0], a[2], a[4], a[6], b[i]);
      mad4_top_fresh(od.w + i + 1, a[1], a[3], a[5], a[7], b[i]);
    }
  }
  od.w[0] = 0;
  wide_add(ev, od);
  return ev;
}

// t 2^-256 mod p, fully reduced, for t = value + (0 or p 2^256 when its top bit says it is negative),
// |value| below p 2^256 / 2.
template <class P>
__device__ __forceinline__ Fp<P> wide_reduce(const Wide& t) {
  uint32_t acc[2][8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    acc[0][k] = t.w[k];
    acc[1][k] = 0;
  }
  Fp<P> r = mont_rows<P>(acc);  // at most p
  const uint32_t neg = (uint32_t)((int32_t)t.w[15] >> 31);
  const uint32_t p[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]), "+r"(r.w[6]), "+r"(r.w[7])
      : "r"(t.w[8]), "r"(t.w[9]), "r"(t.w[10]), "r"(t.w[11]), "r"(t.w[12]), "r"(t.w[13]), "r"(t.w[14]), "r"(t.w[15]));
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]), "+r"(r.w[6]), "+r"(r.w[7])
      : "r"(p[0] & neg), "r"(p[1] & neg), "r"(p[2] & neg), "r"(p[3] & neg), "r"(p[4] & neg), "r"(p[5] & neg),
        "r"(p[6] & neg), "r"(p[7] & neg));
  return reduce_once(r);
}

template <class P>
__device__ __noinline__ Fp<P> mont_mul_call(Fp<P> a, Fp<P> b) {
  return mont_mul_prod(a, b);
}

template <class P>
__device__ __forceinline__ Fp<P> operator*(const Fp<P>& a, const Fp<P>& b) {
  if constexpr (P::kCompact) return mont_mul_call<P>(a, b);
  else return mont_mul_prod(a, b);
}

template <class P>
__device__ __noinline__ Fp<P> mont_sqr_call(Fp<P> a) {
  return mont_sqr_prod(a);
}
template <class P>
__device__ __noinline__ Fp<P> mont_mul_sub_call(Fp<P> a, Fp<P> b, Fp<P> c, Fp<P> d) {
  return mont_mul_sub_prod(a, b, c, d);
}

template <class P>
__device__ __forceinline__ Fp<P> sqr(const Fp<P>& a) {
  if constexpr (P::kCompact) return mont_sqr_call<P>(a);
  else return mont_sqr_prod(a);
}

// a b - c d through one reduction.
template <class P>
__device__ __forceinline__ Fp<P> mul_sub(const Fp<P>& a, const Fp<P>& b, const Fp<P>& c, const Fp<P>& d) {
  if constexpr (P::kCompact) return mont_mul_sub_call<P>(a, b, c, d);
  else return mont_mul_sub_prod(a, b, c, d);
}

// Two independent products. In the compact form they share one out-of-line call, so the two
// dependency chains interleave (a lone thread, as in the window combination, otherwise waits
// on one product's chain at a time) and half the calls are made.
template <class P>
struct FpPair {
  Fp<P> x, y;
};

template <class P>
__device__ __noinline__ FpPair<P> mont_mul2_call(Fp<P> a, Fp<P> b, Fp<P> c, Fp<P> d) {
  return FpPair<P>{mont_mul_prod(a, b), mont_mul_prod(c, d)};
}

template <class P>
__device__ __forceinline__ void mul2(const Fp<P>& a, const Fp<P>& b, const Fp<P>& c, const Fp<P>& d, Fp<P>& r1,
                                     Fp<P>& r2) {
  if constexpr (P::kPairs) {
    FpPair<P> q = mont_mul2_call<P>(a, b, c, d);
    r1 = q.x;
    r2 = q.y;
  } else if constexpr (P::kCompact) {
    r1 = mont_mul_call<P>(a, b);
    r2 = mont_mul_call<P>(c, d);
  } else {
    r1 = mont_mul_prod(a, b);
    r2 = mont_mul_prod(c, d);
  }
}

// ------------------------------------------------------------------ memory helpers

// 32-byte element loads/stores as two 16-byte vector accesses (the address must be 16-byte
// aligned; every buffer and element offset in this library is).
template <class F>
__device__ __forceinline__ F load_fe(const void* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 lo = q[0], hi = q[1];
  F r;
  r.w[0] = lo.x; r.w[1] = lo.y; r.w[2] = lo.z; r.w[3] = lo.w;
  r.w[4] = hi.x; r.w[5] = hi.y; r.w[6] = hi.z; r.w[7] = hi.w;
  return r;
}

template <class F>
__device__ __forceinline__ F load_fe_cg(const void* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 lo = __ldcg(q), hi = __ldcg(q + 1);
  F r;
  r.w[0] = lo.x; r.w[1] = lo.y; r.w[2] = lo.z; r.w[3] = lo.w;
  r.w[4] = hi.x; r.w[5] = hi.y; r.w[6] = hi.z; r.w[7] = hi.w;
  return r;
}

template <class F>
__device__ __forceinline__ void store_fe(void* p, const F& a) {
  uint4* q = reinterpret_cast<uint4*>(p);
  q[0] = make_uint4(a.w[0], a.w[1], a.w[2], a.w[3]);
  q[1] = make_uint4(a.w[4], a.w[5], a.w[6], a.w[7]);
}

// ------------------------------------------------------------------ Fq2 = Fq[u] / (u^2 + 1)

// a + b*u. Karatsuba product in three Fq products, square in two (the reference's G2 prelude,
// src/group.rs:38-48). B is the base field type (Fq, or its compact form FqC).
template <class B>
struct Fq2T {
  B a, b;
  __device__ __forceinline__ static Fq2T zero() { return Fq2T{B::zero(), B::zero()}; }
  __device__ __forceinline__ static Fq2T one() { return Fq2T{B::one(), B::zero()}; }
  __device__ __forceinline__ bool is_zero() const { return a.is_zero() && b.is_zero(); }
  __device__ __forceinline__ bool operator==(const Fq2T& o) const { return a == o.a && b == o.b; }
};

template <class B>
__device__ __forceinline__ Fq2T<B> operator+(const Fq2T<B>& x, const Fq2T<B>& y) {
  return Fq2T<B>{x.a + y.a, x.b + y.b};
}
template <class B>
__device__ __forceinline__ Fq2T<B> operator-(const Fq2T<B>& x, const Fq2T<B>& y) {
  return Fq2T<B>{x.a - y.a, x.b - y.b};
}
template <class B>
__device__ __forceinline__ Fq2T<B> neg(const Fq2T<B>& x) {
  return Fq2T<B>{neg(x.a), neg(x.b)};
}
template <class B>
__device__ __forceinline__ Fq2T<B> dbl(const Fq2T<B>& x) {
  return Fq2T<B>{x.a + x.a, x.b + x.b};
}
// x y and x y - z w with one reduction per component: for each product ac, bd and (a + b)(c + d) as
// 512-bit values, re = ac - bd and im = (a + b)(c + d) - ac - bd (below 2 p^2 each, and 4 p^2 < p 2^256
// in magnitude for the difference). 328 and 520 slots of the multiply pipe, against 396 and 792
// for three reduced products each: 23.7 G Fq2 products/s against 20.4 inlined.
template <class P>
__device__ __forceinline__ Fp<P> sum_raw(const Fp<P>& a, const Fp<P>& b) {  // a + b, not reduced
  Fp<P> s;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=&r"(s.w[0]), "=&r"(s.w[1]), "=&r"(s.w[2]), "=&r"(s.w[3]), "=&r"(s.w[4]), "=&r"(s.w[5]), "=&r"(s.w[6]),
        "=&r"(s.w[7])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
        "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]));
  return s;
}
template <class P>
__device__ __forceinline__ Fq2T<Fp<P>> fq2_mul(const Fq2T<Fp<P>>& x, const Fq2T<Fp<P>>& y) {
  Wide re = wide_mul(x.a.w, y.a.w);
  const Wide bd = wide_mul(x.b.w, y.b.w);
  Wide im = wide_mul(sum_raw(x.a, x.b).w, sum_raw(y.a, y.b).w);
  wide_sub(im, re);
  wide_sub(im, bd);
  wide_sub(re, bd);
  return Fq2T<Fp<P>>{wide_reduce<P>(re), wide_reduce<P>(im)};
}
template <class P>
__device__ __forceinline__ Fq2T<Fp<P>> fq2_mul_sub(const Fq2T<Fp<P>>& x, const Fq2T<Fp<P>>& y, const Fq2T<Fp<P>>& z,
                                                   const Fq2T<Fp<P>>& w) {
  Wide re = wide_mul(x.a.w, y.a.w);
  Wide im = wide_mul(sum_raw(x.a, x.b).w, sum_raw(y.a, y.b).w);
  wide_sub(im, re);
  Wide t = wide_mul(x.b.w, y.b.w);
  wide_sub(re, t);
  wide_sub(im, t);
  t = wide_mul(z.a.w, w.a.w);
  wide_sub(re, t);
  wide_add(im, t);
  t = wide_mul(z.b.w, w.b.w);
  wide_add(re, t);
  wide_add(im, t);
  wide_sub(im, wide_mul(sum_raw(z.a, z.b).w, sum_raw(w.a, w.b).w));
  return Fq2T<Fp<P>>{wide_reduce<P>(re), wide_reduce<P>(im)};
}
template <class P>
__device__ __noinline__ Fq2T<Fp<P>> fq2_mul_call(Fq2T<Fp<P>> x, Fq2T<Fp<P>> y) {
  return fq2_mul(x, y);
}
template <class P>
__device__ __noinline__ Fq2T<Fp<P>> fq2_sqr_call(Fq2T<Fp<P>> x) {
  const Fp<P> ab = mont_mul_prod(x.a, x.b);
  return Fq2T<Fp<P>>{mont_mul_prod(sum_raw(x.a, x.b), x.a - x.b), ab + ab};
}

template <class B>
__device__ __forceinline__ Fq2T<B> operator*(const Fq2T<B>& x, const Fq2T<B>& y) {
  if constexpr (B::kLazy) return fq2_mul_call(x, y);
  B ac = x.a * y.a;
  B bd = x.b * y.b;
  B cross = (x.a + x.b) * (y.a + y.b);
  return Fq2T<B>{ac - bd, (cross - ac) - bd};
}
template <class B>
__device__ __forceinline__ Fq2T<B> sqr(const Fq2T<B>& x) {
  if constexpr (B::kLazy) return fq2_sqr_call(x);
  B ab = x.a * x.b;
  return Fq2T<B>{(x.a + x.b) * (x.a - x.b), ab + ab};
}

// Two independent Fq2 products: the three Karatsuba base products of each, paired.
template <class B>
__device__ __forceinline__ void mul2(const Fq2T<B>& x, const Fq2T<B>& y, const Fq2T<B>& z, const Fq2T<B>& w,
                                     Fq2T<B>& r1, Fq2T<B>& r2) {
  if constexpr (B::kLazy) {
    const Fq2T<B> p = fq2_mul_call(x, y);
    r2 = fq2_mul_call(z, w);
    r1 = p;
    return;
  }
  B ac1, ac2, bd1, bd2, cr1, cr2;
  mul2(x.a, y.a, z.a, w.a, ac1, ac2);
  mul2(x.b, y.b, z.b, w.b, bd1, bd2);
  mul2(x.a + x.b, y.a + y.b, z.a + z.b, w.a + w.b, cr1, cr2);
  r1 = Fq2T<B>{ac1 - bd1, (cr1 - ac1) - bd1};
  r2 = Fq2T<B>{ac2 - bd2, (cr2 - ac2) - bd2};
}

// a b - c d: one reduction per component, or two paired products and a difference.
template <class B>
__device__ __forceinline__ Fq2T<B> mul_sub(const Fq2T<B>& a, const Fq2T<B>& b, const Fq2T<B>& c, const Fq2T<B>& d) {
  if constexpr (B::kLazy) return fq2_mul_sub(a, b, c, d);
  Fq2T<B> ab, cd;
  mul2(a, b, c, d, ab, cd);
  return ab - cd;
}

// Two independent squarings. Fq2: (a+b)(a-b) and ab per element, two base products instead of
// three, paired across the two elements.
template <class P>
__device__ __noinline__ FpPair<P> mont_sqr2_call(Fp<P> a, Fp<P> b) {
  return FpPair<P>{mont_sqr_prod(a), mont_sqr_prod(b)};
}
template <class P>
__device__ __forceinline__ void sqr2(const Fp<P>& x, const Fp<P>& y, Fp<P>& rx, Fp<P>& ry) {
  if constexpr (P::kPairs) {
    FpPair<P> q = mont_sqr2_call<P>(x, y);
    rx = q.x;
    ry = q.y;
  } else {
    rx = sqr(x);
    ry = sqr(y);
  }
}
template <class B>
__device__ __forceinline__ void sqr2(const Fq2T<B>& x, const Fq2T<B>& y, Fq2T<B>& rx, Fq2T<B>& ry) {
  if constexpr (B::kLazy) {
    rx = fq2_sqr_call(x);
    ry = fq2_sqr_call(y);
    return;
  }
  B re_x, re_y, ab_x, ab_y;
  mul2(x.a + x.b, x.a - x.b, y.a + y.b, y.a - y.b, re_x, re_y);
  mul2(x.a, x.b, y.a, y.b, ab_x, ab_y);
  rx = Fq2T<B>{re_x, ab_x + ab_x};
  ry = Fq2T<B>{re_y, ab_y + ab_y};
}

using Fq2 = Fq2T<Fq>;
using Fq2C = Fq2T<FqC>;
using Fq2L = Fq2T<FqL>;

// The compact forms of a coordinate field (same memory layout): out-of-line products one at a
// time (CompactOf), or (PairedOf) two Fq products at a time and Fq2 products with one reduction per
// component.
template <class F>
struct CompactOf;
template <>
struct CompactOf<Fq> {
  using type = FqC;
};
template <>
struct CompactOf<Fq2> {
  using type = Fq2C;
};
template <class F>
struct PairedOf;
template <>
struct PairedOf<Fq> {
  using type = FqCP;
};
template <>
struct PairedOf<Fq2> {
  using type = Fq2L;
};

template <class F>
struct FieldWords;
template <>
struct FieldWords<Fq> {
  static constexpr int value = 8;
};
template <>
struct FieldWords<Fr> {
  static constexpr int value = 8;
};
template <>
struct FieldWords<FqC> {
  static constexpr int value = 8;
};
template <>
struct FieldWords<FqCP> {
  static constexpr int value = 8;
};
template <>
struct FieldWords<Fq2> {
  static constexpr int value = 16;
};
template <>
struct FieldWords<Fq2L> {
  static constexpr int value = 16;
};
template <>
struct FieldWords<Fq2C> {
  static constexpr int value = 16;
};

template <class F>
__device__ __forceinline__ F load_elem(const uint32_t* p);
template <>
__device__ __forceinline__ Fq load_elem<Fq>(const uint32_t* p) {
  return load_fe<Fq>(p);
}
template <>
__device__ __forceinline__ Fr load_elem<Fr>(const uint32_t* p) {
  return load_fe<Fr>(p);
}
template <>
__device__ __forceinline__ FqC load_elem<FqC>(const uint32_t* p) {
  return load_fe<FqC>(p);
}
template <>
__device__ __forceinline__ FqCP load_elem<FqCP>(const uint32_t* p) {
  return load_fe<FqCP>(p);
}
template <>
__device__ __forceinline__ Fq2L load_elem<Fq2L>(const uint32_t* p) {
  return Fq2L{load_fe<FqL>(p), load_fe<FqL>(p + 8)};
}
template <>
__device__ __forceinline__ Fq2 load_elem<Fq2>(const uint32_t* p) {
  return Fq2{load_fe<Fq>(p), load_fe<Fq>(p + 8)};
}
template <>
__device__ __forceinline__ Fq2C load_elem<Fq2C>(const uint32_t* p) {
  return Fq2C{load_fe<FqC>(p), load_fe<FqC>(p + 8)};
}

__device__ __forceinline__ void store_elem(uint32_t* p, const Fq& x) { store_fe(p, x); }
__device__ __forceinline__ void store_elem(uint32_t* p, const Fr& x) { store_fe(p, x); }
__device__ __forceinline__ void store_elem(uint32_t* p, const FqC& x) { store_fe(p, x); }
__device__ __forceinline__ void store_elem(uint32_t* p, const FqCP& x) { store_fe(p, x); }
template <class B>
__device__ __forceinline__ void store_elem(uint32_t* p, const Fq2T<B>& x) {
  store_fe(p, x.a);
  store_fe(p + 8, x.b);
}

}  // namespace zkg
