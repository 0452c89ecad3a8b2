// Products by constants of Fr with a precomputed quotient (Shoup's method): for a constant w < r and
// w' = floor(w 2^256 / r), q = floor(x w' / 2^256) makes x w - q r a residue of x w below 2r, and both
// products are needed modulo 2^256 alone.
//
// Of the 64 products of words in x w', the 21 below word 6 are left out: together they are under
// 2^-29 of a unit of q. The real number T that they leave is above x w / r - x / 2^256 - 2^-29 (w' is
// less than one below w 2^256 / r), and q = floor(T), so the residue is below r (1 + x / 2^256 + 2^-29):
// below 1.757r for x < 4r, below 2r for x < 2^256 (1 - 2^-29). 43 wide multiply-adds there, 28 and eight
// low halves for each of x w and q r, all on
// two interleaved accumulators as in field.cuh: 107 slots of the multiply pipe against the Montgomery
// product's 132, no chain of digits, and nothing to convert: x w stands in plain form. Measured on
// B200: 81.3 G products/s, 326 ns for a lone warp (Montgomery: 68.5 G/s, 422 ns).
#pragma once
#include "field.cuh"

namespace zkg {
namespace shoup {

// Chains of one row on an accumulator: c += (x[0] + x[1] 2^64 + ...) y over N pairs of words, then
//   mad_drop   nothing: the sum is taken modulo the last pair's end,
//   mad_low    c[2N] += low half of z y, and the carry,
//   mad_fresh  the last pair's high word is written, not added to (the sum does not overflow it),
//   mad_carry  the carry is written to c[2N].
template <int N>
__device__ __forceinline__ void mad_drop(uint32_t* c, const uint32_t (&x)[N], uint32_t y) {
  if constexpr (N == 1)
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32 %1, %2, %3, %1;"
        : "+r"(c[0]), "+r"(c[1])
        : "r"(x[0]), "r"(y));
  else if constexpr (N == 2)
    asm("mad.lo.cc.u32 %0, %4, %6, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
        "madc.hi.u32 %3, %5, %6, %3;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(x[0]), "r"(x[1]), "r"(y));
  else if constexpr (N == 3)
    asm("mad.lo.cc.u32 %0, %6, %9, %0;\n\t"
        "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
        "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
        "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
        "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
        "madc.hi.u32 %5, %8, %9, %5;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(y));
  else
    asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
        "madc.hi.u32 %7, %11, %12, %7;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y));
}
template <int N>
__device__ __forceinline__ void mad_low(uint32_t* c, const uint32_t (&x)[N], uint32_t z, uint32_t y) {
  if constexpr (N == 1)
    asm("mad.lo.cc.u32 %0, %3, %5, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %5, %1;\n\t"
        "madc.lo.u32 %2, %4, %5, %2;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2])
        : "r"(x[0]), "r"(z), "r"(y));
  else if constexpr (N == 2)
    asm("mad.lo.cc.u32 %0, %5, %8, %0;\n\t"
        "madc.hi.cc.u32 %1, %5, %8, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
        "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
        "madc.lo.u32 %4, %7, %8, %4;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4])
        : "r"(x[0]), "r"(x[1]), "r"(z), "r"(y));
  else
    asm("mad.lo.cc.u32 %0, %7, %11, %0;\n\t"
        "madc.hi.cc.u32 %1, %7, %11, %1;\n\t"
        "madc.lo.cc.u32 %2, %8, %11, %2;\n\t"
        "madc.hi.cc.u32 %3, %8, %11, %3;\n\t"
        "madc.lo.cc.u32 %4, %9, %11, %4;\n\t"
        "madc.hi.cc.u32 %5, %9, %11, %5;\n\t"
        "madc.lo.u32 %6, %10, %11, %6;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(z), "r"(y));
}
template <int N>
__device__ __forceinline__ void mad_fresh(uint32_t* c, const uint32_t (&x)[N], uint32_t y) {
  if constexpr (N == 1)
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32 %1, %2, %3, 0;"
        : "+r"(c[0]), "=&r"(c[1])
        : "r"(x[0]), "r"(y));
  else if constexpr (N == 2)
    asm("mad.lo.cc.u32 %0, %4, %6, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
        "madc.hi.u32 %3, %5, %6, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "=&r"(c[3])
        : "r"(x[0]), "r"(x[1]), "r"(y));
  else if constexpr (N == 3)
    asm("mad.lo.cc.u32 %0, %6, %9, %0;\n\t"
        "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
        "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
        "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
        "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
        "madc.hi.u32 %5, %8, %9, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "=&r"(c[5])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(y));
  else
    asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
        "madc.hi.u32 %7, %11, %12, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "=&r"(c[7])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y));
}
template <int N>
__device__ __forceinline__ void mad_carry(uint32_t* c, const uint32_t (&x)[N], uint32_t y) {
  if constexpr (N == 1)
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, 0, 0;"
        : "+r"(c[0]), "+r"(c[1]), "=&r"(c[2])
        : "r"(x[0]), "r"(y));
  else if constexpr (N == 2)
    asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\t"
        "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
        "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
        "addc.u32 %4, 0, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "=&r"(c[4])
        : "r"(x[0]), "r"(x[1]), "r"(y));
  else if constexpr (N == 3)
    asm("mad.lo.cc.u32 %0, %7, %10, %0;\n\t"
        "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
        "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
        "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
        "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
        "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
        "addc.u32 %6, 0, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "=&r"(c[6])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(y));
  else
    asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
        "addc.u32 %8, 0, 0;"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]), "=&r"(c[8])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y));
}

__device__ __forceinline__ void mul_pair(uint32_t* c, uint32_t x, uint32_t y) {
  const uint64_t t = (uint64_t)x * y;
  c[0] = (uint32_t)t;
  c[1] = (uint32_t)(t >> 32);
}

// (ev[0..7] at words 0..7, od[0..6] at words 1..7) += x w modulo 2^256; FRESH: they are written.
template <bool FRESH>
__device__ __forceinline__ void low_product(uint32_t (&ev)[8], uint32_t (&od)[7], const uint32_t (&x)[8],
                                            const uint32_t (&w)[8]) {
  if constexpr (FRESH) {
#pragma unroll
    for (int k = 0; k < 4; k++) mul_pair(ev + 2 * k, x[0], w[2 * k]);
#pragma unroll
    for (int k = 0; k < 3; k++) mul_pair(od + 2 * k, x[0], w[2 * k + 1]);
    od[6] = x[0] * w[7];
  } else {
    mad_drop<4>(ev, {w[0], w[2], w[4], w[6]}, x[0]);
    mad_low<3>(od, {w[1], w[3], w[5]}, w[7], x[0]);
  }
  mad_drop<3>(ev + 2, {w[1], w[3], w[5]}, x[1]);
  mad_low<3>(od, {w[0], w[2], w[4]}, w[6], x[1]);
  mad_drop<3>(ev + 2, {w[0], w[2], w[4]}, x[2]);
  mad_low<2>(od + 2, {w[1], w[3]}, w[5], x[2]);
  mad_drop<2>(ev + 4, {w[1], w[3]}, x[3]);
  mad_low<2>(od + 2, {w[0], w[2]}, w[4], x[3]);
  mad_drop<2>(ev + 4, {w[0], w[2]}, x[4]);
  mad_low<1>(od + 4, {w[1]}, w[3], x[4]);
  mad_drop<1>(ev + 6, {w[1]}, x[5]);
  mad_low<1>(od + 4, {w[0]}, w[2], x[5]);
  mad_drop<1>(ev + 6, {w[0]}, x[6]);
  od[6] += x[6] * w[1];
  od[6] += x[7] * w[0];
}

__device__ __forceinline__ Fr join_low(const uint32_t (&ev)[8], const uint32_t (&od)[7]) {
  Fr r;
  r.w[0] = ev[0];
  asm("add.cc.u32  %0, %7, %14;\n\t"
      "addc.cc.u32 %1, %8, %15;\n\t"
      "addc.cc.u32 %2, %9, %16;\n\t"
      "addc.cc.u32 %3, %10, %17;\n\t"
      "addc.cc.u32 %4, %11, %18;\n\t"
      "addc.cc.u32 %5, %12, %19;\n\t"
      "addc.u32    %6, %13, %20;"
      : "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]), "=&r"(r.w[7])
      : "r"(ev[1]), "r"(ev[2]), "r"(ev[3]), "r"(ev[4]), "r"(ev[5]), "r"(ev[6]), "r"(ev[7]), "r"(od[0]), "r"(od[1]),
        "r"(od[2]), "r"(od[3]), "r"(od[4]), "r"(od[5]), "r"(od[6]));
  return r;
}

// floor of a b / 2^256 less the products below word 6 (see above): that of a b / 2^256, or one less.
__device__ __forceinline__ void high_product(const uint32_t (&a)[8], const uint32_t (&b)[8], uint32_t (&q)[8]) {
  uint32_t e[10], o[8];  // words 6..15 and 7..14
  mul_pair(e, a[0], b[6]);
  mul_pair(o, a[0], b[7]);
  mad_carry<1>(e, {b[5]}, a[1]);
  mad_carry<1>(o, {b[6]}, a[1]);
  mad_fresh<1>(e + 2, {b[7]}, a[1]);
  mad_carry<2>(e, {b[4], b[6]}, a[2]);
  mad_fresh<2>(o, {b[5], b[7]}, a[2]);
  mad_fresh<3>(e, {b[3], b[5], b[7]}, a[3]);
  mad_carry<2>(o, {b[4], b[6]}, a[3]);
  mad_carry<3>(e, {b[2], b[4], b[6]}, a[4]);
  mad_fresh<3>(o, {b[3], b[5], b[7]}, a[4]);
  mad_fresh<4>(e, {b[1], b[3], b[5], b[7]}, a[5]);
  mad_carry<3>(o, {b[2], b[4], b[6]}, a[5]);
  mad_carry<4>(e, {b[0], b[2], b[4], b[6]}, a[6]);
  mad_fresh<4>(o, {b[1], b[3], b[5], b[7]}, a[6]);
  mad_fresh<4>(e + 2, {b[1], b[3], b[5], b[7]}, a[7]);
  uint32_t top[9] = {o[0], o[1], o[2], o[3], o[4], o[5], o[6], o[7], 0};
  mad_carry<4>(top, {b[0], b[2], b[4], b[6]}, a[7]);
  // words 8..15: e[2..9] + top[1..8], and the carry out of word 7 (e[1] + top[0])
  uint32_t word7;
  asm("add.cc.u32  %8, %9, %18;\n\t"
      "addc.cc.u32 %0, %10, %19;\n\t"
      "addc.cc.u32 %1, %11, %20;\n\t"
      "addc.cc.u32 %2, %12, %21;\n\t"
      "addc.cc.u32 %3, %13, %22;\n\t"
      "addc.cc.u32 %4, %14, %23;\n\t"
      "addc.cc.u32 %5, %15, %24;\n\t"
      "addc.cc.u32 %6, %16, %25;\n\t"
      "addc.u32    %7, %17, %26;"
      : "=&r"(q[0]), "=&r"(q[1]), "=&r"(q[2]), "=&r"(q[3]), "=&r"(q[4]), "=&r"(q[5]), "=&r"(q[6]), "=&r"(q[7]),
        "=&r"(word7)
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(top[0]),
        "r"(top[1]), "r"(top[2]), "r"(top[3]), "r"(top[4]), "r"(top[5]), "r"(top[6]), "r"(top[7]), "r"(top[8]));
}

// A constant: w < r and floor(w 2^256 / r), 16 words in memory.
struct Constant {
  Fr w, quotient;
};

// x c.w modulo r, below r (1 + x / 2^256 + 2^-29): below 1.757r for x < 4r.
__device__ __forceinline__ Fr mul(const Fr& x, const Constant& c) {
  constexpr uint32_t minus_r[8] = {0u - FrParams::P0, ~FrParams::P1, ~FrParams::P2, ~FrParams::P3,
                                   ~FrParams::P4,     ~FrParams::P5, ~FrParams::P6, ~FrParams::P7};
  uint32_t q[8], ev[8], od[7];
  high_product(x.w, c.quotient.w, q);
  low_product<true>(ev, od, x.w, c.w.w);
  low_product<false>(ev, od, q, minus_r);
  return join_low(ev, od);
}

// The constant of a Montgomery form m = w 2^256 mod r (reduced): w = m 2^-256 mod r, and w 2^256 =
// quotient r + m makes the quotient -m / r modulo 2^256.
__device__ __forceinline__ Constant constant(const Fr& m) {
  constexpr uint32_t minus_inverse[8] = {0xefffffffu, 0xc2e1f593u, 0x4c6911b3u, 0x6586864bu,
                                         0x99062391u, 0xe39a9828u, 0x0d8341b2u, 0x73f82f1du};  // -1 / r mod 2^256
  Fr one = Fr::zero();
  one.w[0] = 1;
  uint32_t ev[8], od[7];
  low_product<true>(ev, od, m.w, minus_inverse);
  return Constant{m * one, join_low(ev, od)};
}

}  // namespace shoup
}  // namespace zkg
