// Inverse of a field element by division steps (Bernstein and Yang, "Fast constant-time gcd
// computation and modular inversion", TCHES 2019), for a lone thread or a block's one inversion.
//
// (delta, f, g) starts at (1, p, x); a division step with g odd and delta > 0 makes it
// (1 - delta, g, (g - f) / 2), any other one (1 + delta, f, (g + (g mod 2) f) / 2). For 255-bit
// operands g is zero after at most 741 steps, and then f = +-1. Thirty steps at a time depend on the
// low 30 bits of f and g alone, so they run on single words and give a 2x2 matrix of integers with
// row sums at most 2^30 in magnitude; the matrix is then applied to f and g (exactly divisible by
// 2^30) and, modulo p, to (d, e), which keep d x = f and e x = g modulo p.
//
// About 18 rounds of ~1000 integer instructions: 14 us for a lone thread, against 254 squarings and
// ~80 products (120 us) for the power p - 2.
#pragma once
#include "field.cuh"

namespace zkg {

// 2^768 mod q: R^3 of the base field.
__device__ constexpr uint32_t kFqR3[8] = {0xda1530dfu, 0xb1cd6dafu, 0xa7283db6u, 0x62f210e6u,
                                          0x0ada0afbu, 0xef7f0b0cu, 0x2d592544u, 0x20fd6e90u};

namespace divsteps {

constexpr int kSteps = 30;
constexpr int kMaxRounds = 25;  // 750 steps

struct Matrix {
  int32_t u, v, q, r;
};

// Thirty division steps on the low words of f and g. (f, g) * 2^30 = matrix * (f, g).
__device__ __forceinline__ Matrix steps(uint32_t f, uint32_t g, int& delta) {
  uint32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 6
  for (int i = 0; i < kSteps; i++) {
    const bool odd = g & 1;
    const bool swap = odd && delta > 0;
    const uint32_t f0 = f, u0 = u, v0 = v;
    f = swap ? g : f;
    u = swap ? q : u;
    v = swap ? r : v;
    // the new g is g - f after a swap, g + f without one
    const uint32_t a = swap ? 0u - f0 : f0, b = swap ? 0u - u0 : u0, c = swap ? 0u - v0 : v0;
    delta = swap ? 1 - delta : 1 + delta;
    g = (odd ? g + a : g) >> 1;
    q = odd ? q + b : q;
    r = odd ? r + c : r;
    u <<= 1;
    v <<= 1;
  }
  return Matrix{(int32_t)u, (int32_t)v, (int32_t)q, (int32_t)r};
}

// t (9 words, modulo 2^288) += s * x, x a signed value of eight words and s a signed word.
__device__ __forceinline__ void add_scaled(uint32_t (&t)[9], int32_t s, const uint32_t (&x)[8]) {
  const uint32_t us = (uint32_t)s;
  const uint32_t sign = (uint32_t)((int32_t)x[7] >> 31);
  asm("mad.lo.cc.u32  %0, %9, %17, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %17, %1;\n\t"
      "madc.lo.cc.u32 %2, %11, %17, %2;\n\t"
      "madc.hi.cc.u32 %3, %11, %17, %3;\n\t"
      "madc.lo.cc.u32 %4, %13, %17, %4;\n\t"
      "madc.hi.cc.u32 %5, %13, %17, %5;\n\t"
      "madc.lo.cc.u32 %6, %15, %17, %6;\n\t"
      "madc.hi.cc.u32 %7, %15, %17, %7;\n\t"
      "madc.lo.u32    %8, %18, %17, %8;\n\t"
      "mad.lo.cc.u32  %1, %10, %17, %1;\n\t"
      "madc.hi.cc.u32 %2, %10, %17, %2;\n\t"
      "madc.lo.cc.u32 %3, %12, %17, %3;\n\t"
      "madc.hi.cc.u32 %4, %12, %17, %4;\n\t"
      "madc.lo.cc.u32 %5, %14, %17, %5;\n\t"
      "madc.hi.cc.u32 %6, %14, %17, %6;\n\t"
      "madc.lo.cc.u32 %7, %16, %17, %7;\n\t"
      "madc.hi.u32    %8, %16, %17, %8;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]), "+r"(t[8])
      : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(us), "r"(sign));
  // a negative s counted as s + 2^32: take x 2^32 off again
  const uint32_t m = (uint32_t)(s >> 31);
  asm("sub.cc.u32  %0, %0, %8;\n\t"
      "subc.cc.u32 %1, %1, %9;\n\t"
      "subc.cc.u32 %2, %2, %10;\n\t"
      "subc.cc.u32 %3, %3, %11;\n\t"
      "subc.cc.u32 %4, %4, %12;\n\t"
      "subc.cc.u32 %5, %5, %13;\n\t"
      "subc.cc.u32 %6, %6, %14;\n\t"
      "subc.u32    %7, %7, %15;"
      : "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]), "+r"(t[8])
      : "r"(x[0] & m), "r"(x[1] & m), "r"(x[2] & m), "r"(x[3] & m), "r"(x[4] & m), "r"(x[5] & m), "r"(x[6] & m),
        "r"(x[7] & m));
}

// t / 2^30 (t divisible by it), a signed value of eight words.
__device__ __forceinline__ void shift_down(const uint32_t (&t)[9], uint32_t (&x)[8]) {
#pragma unroll
  for (int i = 0; i < 8; i++) x[i] = __funnelshift_r(t[i], t[i + 1], kSteps);
}

// (s x + t y) / 2^30 modulo p, in [0, p), for x, y in [0, p) and |s| + |t| <= 2^30.
template <class P>
__device__ __forceinline__ void combine_mod(int32_t s, const uint32_t (&x)[8], int32_t t, const uint32_t (&y)[8],
                                            uint32_t (&out)[8]) {
  constexpr uint32_t p[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  uint32_t a[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  add_scaled(a, s, x);
  add_scaled(a, t, y);
  const uint32_t m = (a[0] * P::INV) & ((1u << kSteps) - 1);  // a + m p is divisible by 2^30
  add_scaled(a, (int32_t)m, p);
  shift_down(a, out);  // in (-p, 2p)
  const uint32_t neg = (uint32_t)((int32_t)out[7] >> 31);
  Fp<P> r;
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
      : "r"(out[0]), "r"(out[1]), "r"(out[2]), "r"(out[3]), "r"(out[4]), "r"(out[5]), "r"(out[6]), "r"(out[7]),
        "r"(p[0] & neg), "r"(p[1] & neg), "r"(p[2] & neg), "r"(p[3] & neg), "r"(p[4] & neg), "r"(p[5] & neg),
        "r"(p[6] & neg), "r"(p[7] & neg));
  r = reduce_once(r);
#pragma unroll
  for (int i = 0; i < 8; i++) out[i] = r.w[i];
}

}  // namespace divsteps

// 1/a in Montgomery form (a != 0; zero gives zero), a fully reduced: x = a R gives x^-1 = a^-1 R^-1,
// and one product by R^3 makes it a^-1 R. r3 = R^3 mod p.
template <class P>
__device__ __noinline__ Fp<P> mont_inverse(Fp<P> a, Fp<P> r3) {
  using namespace divsteps;
  uint32_t f[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  uint32_t g[8], d[8], e[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    g[i] = a.w[i];
    d[i] = 0;
    e[i] = i == 0;
  }
  int delta = 1;
#pragma unroll 1
  for (int round = 0; round < kMaxRounds; round++) {
    const Matrix m = steps(f[0], g[0], delta);
    uint32_t t[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, nf[8], ng[8];
    add_scaled(t, m.u, f);
    add_scaled(t, m.v, g);
    shift_down(t, nf);
#pragma unroll
    for (int i = 0; i < 9; i++) t[i] = 0;
    add_scaled(t, m.q, f);
    add_scaled(t, m.r, g);
    shift_down(t, ng);
    uint32_t nd[8], ne[8];
    combine_mod<P>(m.u, d, m.v, e, nd);
    combine_mod<P>(m.q, d, m.r, e, ne);
    uint32_t any = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      f[i] = nf[i];
      g[i] = ng[i];
      d[i] = nd[i];
      e[i] = ne[i];
      any |= ng[i];
    }
    if (any == 0) break;
  }
  Fp<P> r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.w[i] = d[i];
  if ((int32_t)f[7] < 0) r = neg(r);  // f = -1
  return mont_mul_prod(r, r3);
}

// 1/a in Montgomery form of the base field's forms (zero for zero).
template <class P>
__device__ __forceinline__ Fp<P> affine_inverse(const Fp<P>& a) {
  Fp<FqParams> x, r3;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    x.w[i] = a.w[i];
    r3.w[i] = kFqR3[i];
  }
  const Fp<FqParams> y = mont_inverse<FqParams>(x, r3);
  Fp<P> r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.w[i] = y.w[i];
  return r;
}
// 1 / (a + bu) = (a - bu) / (a^2 + b^2)
template <class B>
__device__ __forceinline__ Fq2T<B> affine_inverse(const Fq2T<B>& x) {
  const B inv = affine_inverse(sqr(x.a) + sqr(x.b));
  return Fq2T<B>{x.a * inv, neg(x.b * inv)};
}

}  // namespace zkg
