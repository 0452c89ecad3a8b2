// XYZZ doubling and addition by a group of lanes: the independent field products of each dependency
// level run on different lanes at once, so an operation takes its levels' latency (doubling 2,
// addition 4) instead of its products' (9 and 14).
//
// A group is eight roles, of one lane each for Fq and two or four for Fq2 (kLanes = 8, 16 or 32 lanes; a
// warp holds 4, 2 or 1 groups). In Fq2 the two lanes of a role compute one component of a product each,
// a0 b0 - a1 b1 and a0 b1 + a1 b0 through one reduction, and exchange them; with four lanes (SPLIT = 2)
// each computes one of the four products, for chains with nothing beside them to fill the warp. Values
// pass between roles by shuffles within the group; every lane of a warp takes part in every call.
//
// A lone warp's product takes 428 ns, a b - c d 611 ns; measured on B200 per doubling in the chain of
// the window combination (LaneChain), G1 1.1 us, G2 1.65 (dbl-2008-s-1, three products deep: 1.6 and
// 2.4; two lanes a role: G2 2.65). Every lane used to hold the whole point and to form every level's
// sums itself through shared memory: 1.9 and 5.4 us.
#pragma once
#include "curve.cuh"

namespace zkg {

template <class F, int SPLIT = 1>
struct LaneGroup;
template <class P, int SPLIT>
struct LaneGroup<Fp<P>, SPLIT> {  // a product of Fq is not split
  static constexpr unsigned kLanes = 8, kPerRole = 1;
};
template <class B, int SPLIT>
struct LaneGroup<Fq2T<B>, SPLIT> {
  static constexpr unsigned kLanes = 16 * SPLIT, kPerRole = 2 * SPLIT;
};
template <class F, int SPLIT = 1>
__device__ __forceinline__ unsigned lane_role() {
  return (threadIdx.x & (LaneGroup<F, SPLIT>::kLanes - 1)) / LaneGroup<F, SPLIT>::kPerRole;
}

// The value a role of this group holds (role: may differ between lanes).
template <int SPLIT = 1, class F>
__device__ __forceinline__ F lane_from(const F& v, unsigned role) {
  constexpr unsigned W = sizeof(F) / 4;
  const unsigned src = role * LaneGroup<F, SPLIT>::kPerRole;
  F r;
  const uint32_t* a = reinterpret_cast<const uint32_t*>(&v);
  uint32_t* b = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
  for (unsigned i = 0; i < W; i++) b[i] = __shfl_sync(0xffffffffu, a[i], src, LaneGroup<F, SPLIT>::kLanes);
  return r;
}
template <class F, int SPLIT = 1>
__device__ __forceinline__ bool lane_flag(bool v, unsigned role) {
  return __shfl_sync(0xffffffffu, (int)v, role * LaneGroup<F, SPLIT>::kPerRole, LaneGroup<F, SPLIT>::kLanes) != 0;
}

template <class P>
__device__ __forceinline__ Fp<P> lane_select(bool c, const Fp<P>& a, const Fp<P>& b) {
  Fp<P> r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.w[i] = c ? a.w[i] : b.w[i];
  return r;
}
template <class B>
__device__ __forceinline__ Fq2T<B> lane_select(bool c, const Fq2T<B>& a, const Fq2T<B>& b) {
  return Fq2T<B>{lane_select(c, a.a, b.a), lane_select(c, a.b, b.b)};
}

// A role's product and square: for Fq2 each lane its component, then both lanes both.
template <int SPLIT = 1, class P>
__device__ __forceinline__ Fp<P> lane_product(const Fp<P>& a, const Fp<P>& b) {
  return mont_mul_prod(a, b);
}
template <class P>
__device__ __forceinline__ Fp<P> lane_square(const Fp<P>& a) {
  return mont_sqr_prod(a);
}
template <class B>
__device__ __forceinline__ Fq2T<B> lane_exchange(const B& own) {
  B other;
#pragma unroll
  for (int i = 0; i < 8; i++) other.w[i] = __shfl_xor_sync(0xffffffffu, own.w[i], 1);
  const bool imaginary = threadIdx.x & 1;
  return Fq2T<B>{lane_select(imaginary, other, own), lane_select(imaginary, own, other)};
}
template <int SPLIT = 1, class B>
__device__ __forceinline__ Fq2T<B> lane_product(const Fq2T<B>& a, const Fq2T<B>& b) {
  const bool imaginary = threadIdx.x & 1;
  if constexpr (SPLIT == 2) {  // lanes 0, 2: a0 b0, a1 b1; 1, 3: a0 b1, a1 b0
    const bool second = threadIdx.x & 2;
    const B own = mont_mul_prod(lane_select(second, a.b, a.a), lane_select(second != imaginary, b.b, b.a));
    B other;
#pragma unroll
    for (int i = 0; i < 8; i++) other.w[i] = __shfl_xor_sync(0xffffffffu, own.w[i], 2);
    const B difference = lane_select(second, other, own) - lane_select(second, own, other);
    return lane_exchange(lane_select(imaginary, own + other, difference));
  }
  return lane_exchange(reduce_once(mont_mul_add_lazy(a.a, lane_select(imaginary, b.b, b.a),
                                                     lane_select(imaginary, a.b, complement(a.b)),
                                                     lane_select(imaginary, b.a, b.b))));
}
template <class B>
__device__ __forceinline__ Fq2T<B> lane_square(const Fq2T<B>& a) {  // (a0 + a1)(a0 - a1), 2 a0 a1
  const bool imaginary = threadIdx.x & 1;
  return lane_exchange(mont_mul_prod(lane_select(imaginary, dbl(a.a), a.a + a.b),
                                     lane_select(imaginary, a.b, a.a - a.b)));
}

// A lane's role in a group of SPLIT lanes a component.
template <int SPLIT>
struct LaneRole {
  unsigned role;
};

// Sums left between p and 2^256 for a product's operand (a p + p stays below 2^256 for a <= 4).
template <class P>
__device__ __forceinline__ Fp<P> lane_sum(const Fp<P>& a, const Fp<P>& b) {
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
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
        "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]));
  return r;
}
template <int BITS, class P>
__device__ __forceinline__ Fp<P> lane_shift(const Fp<P>& a) {  // 2^BITS a
  Fp<P> r;
  r.w[0] = a.w[0] << BITS;
#pragma unroll
  for (int i = 1; i < 8; i++) r.w[i] = __funnelshift_l(a.w[i - 1], a.w[i], BITS);
  return r;
}
template <class P>
__device__ __forceinline__ Fp<P> lane_complement(const Fp<P>& a) {
  return complement(a);
}
template <class P>
__device__ __forceinline__ Fp<P> lane_halve(const Fp<P>& a) {
  constexpr uint32_t q[8] = {P::P0, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
  Fp<P> p, r;
#pragma unroll
  for (int i = 0; i < 8; i++) p.w[i] = (a.w[0] & 1) ? q[i] : 0;
  const Fp<P> s = lane_sum(a, p);
#pragma unroll
  for (int i = 0; i < 7; i++) r.w[i] = __funnelshift_r(s.w[i], s.w[i + 1], 1);
  r.w[7] = s.w[7] >> 1;
  return r;
}
template <class B>
__device__ __forceinline__ Fq2T<B> lane_sum(const Fq2T<B>& a, const Fq2T<B>& b) {
  return Fq2T<B>{lane_sum(a.a, b.a), lane_sum(a.b, b.b)};
}
template <int BITS, class B>
__device__ __forceinline__ Fq2T<B> lane_shift(const Fq2T<B>& a) {
  return Fq2T<B>{lane_shift<BITS>(a.a), lane_shift<BITS>(a.b)};
}
template <class B>
__device__ __forceinline__ Fq2T<B> lane_complement(const Fq2T<B>& a) {
  return Fq2T<B>{complement(a.a), complement(a.b)};
}
template <class B>
__device__ __forceinline__ Fq2T<B> lane_halve(const Fq2T<B>& a) {
  return Fq2T<B>{lane_halve(a.a), lane_halve(a.b)};
}

// A point through repeated doublings, two products deep each instead of dbl-2008-s-1's three. With
// D = Y^2 - X^3 (which doubling multiplies by (2Y)^6, whatever curve y^2 = x^3 + b the point is on) and A = Y^2,
//   X' = X (A - 9D),  Y' = (A + 9D)^2 - 108 D^2,  D' = 64 D A^3,  ZZ' = 4A ZZ,  ZZZ' = 8 Y A ZZZ,
// the same values. Kept: V = 9D and T = 12D, so that 108 D^2 = V T. A doubling forms A, V, T, 2Y ZZZ/2
// from the last one's products, then its own, one a role:
//   0: (A + V)^2   1: V T   2: X'   3: V 4A   4: T 4A   5: A 4A   6: ZZ'   7: ZZZ'/2
// V' = 4 (V 4A) (A 4A), T' likewise. Operands are left up to 4p, or 2p by 2p: products come out below 2p
// before their one subtraction.
template <class F>
struct LaneChain {
  F v;  // the role's
};

template <class F, int SPLIT>
__device__ __forceinline__ LaneChain<F> lane_chain(const uint32_t* p, LaneRole<SPLIT> lane) {
  constexpr int W = FieldWords<F>::value;
  const unsigned role = lane.role;
  const F x = load_elem<F>(p), y = load_elem<F>(p + W);
  const F own = load_elem<F>(p + (role == 6 ? 2 : role == 7 ? 3 : role & 1) * W);  // X or Y, ZZ, ZZZ
  const F sq = lane_square(lane_select(role == 1, y, x));
  const F d = lane_from<SPLIT>(sq, 1) - lane_product<SPLIT>(lane_from<SPLIT>(sq, 0), x);
  const F d3 = dbl(d) + d, d6 = dbl(d3);
  const F quarter = lane_halve(lane_halve(F::one()));  // for role 5: V = 4 (9D) / 4
  F v = lane_select(role == 0, y, own);
  v = lane_select(role == 1, F::zero(), lane_select(role == 2, x, v));
  v = lane_select(role == 3, d6 + d3, lane_select(role == 4, dbl(d6), v));
  v = lane_select(role == 5, quarter, lane_select(role == 7, lane_halve(own), v));
  return LaneChain<F>{v};
}
template <int SPLIT, class F>
__device__ __forceinline__ LaneChain<F> lane_double(const LaneChain<F>& c, LaneRole<SPLIT> lane) {
  const unsigned role = lane.role;
  const bool vt = role == 1 || role == 3 || role == 4;  // 3: V', 1 and 4: T'; the others: Y'
  const F s = lane_from<SPLIT>(c.v, vt ? 5u : 0u), t = lane_from<SPLIT>(c.v, !vt ? 1u : role == 3 ? 3u : 4u);
  const F y = s - t;
  const F l1 = lane_product<SPLIT>(lane_select(vt, lane_shift<2>(t), y),
                                   lane_select(vt, s, lane_select(role == 7, lane_shift<1>(c.v), y)));
  const F a = lane_from<SPLIT>(l1, 0), v = lane_from<SPLIT>(l1, 3);
  const F sum = lane_sum(a, lane_select(role == 2, lane_complement(v), v));
  const F left = lane_select(role == 0 || role == 2, sum, lane_select(role == 1, v, lane_shift<2>(a)));
  const F kept = lane_select(role == 2 || role == 6, c.v, l1);  // X, ZZ; T, V, 2Y ZZZ/2; A in role 5
  return LaneChain<F>{lane_product<SPLIT>(left, lane_select(role == 0, sum, kept))};
}

// A group's values to memory that it may write.
template <class P>
__device__ __forceinline__ void lane_store_elem(uint32_t* p, const Fp<P>& v) {
  store_fe(p, v);
}
template <class B>
__device__ __forceinline__ void lane_store_elem(uint32_t* p, const Fq2T<B>& v) {  // each lane its component
  const bool imaginary = threadIdx.x & 1;
  store_fe(p + (imaginary ? 8 : 0), lane_select(imaginary, v.b, v.a));
}
template <int SPLIT, class F>
__device__ __forceinline__ void lane_store(uint32_t* out, const LaneChain<F>& c, bool active) {
  constexpr int W = FieldWords<F>::value;
  const unsigned role = lane_role<F, SPLIT>();
  const F y = c.v - lane_from<SPLIT>(c.v, 1);  // in role 0
  if (!active) return;
  if (role == 0) lane_store_elem(out + W, y);
  if (role == 2) lane_store_elem(out, c.v);
  if (role == 6) lane_store_elem(out + 2 * W, c.v);
  if (role == 7) lane_store_elem(out + 3 * W, dbl(c.v));
}

// *out = *p + *q (add-2008-s), as xyzz_add, for points in memory that the group may read; out may be p
// or q. A group with active = false takes part and writes nothing (p and q: any readable points).
template <class F, int SPLIT = 1>
__device__ __forceinline__ void lane_add(const uint32_t* p, const uint32_t* q, uint32_t* out, bool active) {
  constexpr int W = FieldWords<F>::value;
  const unsigned role = lane_role<F, SPLIT>();
  // roles 0..5: X1 ZZ2, X2 ZZ1, Y1 ZZZ2, Y2 ZZZ1, ZZ1 ZZ2, ZZZ1 ZZZ2
  const bool second = role == 1 || role == 3;
  const uint32_t* const pa = second ? q : p;
  const uint32_t* const pb = second ? p : q;
  const int ca = role < 2 ? 0 : role < 4 ? 1 : (role & 1) ? 3 : 2;
  const int cb = role < 2 ? 2 : role < 4 ? 3 : ca;
  const F a = load_elem<F>(pa + ca * W), b = load_elem<F>(pb + cb * W);
  const bool inf_p = lane_flag<F, SPLIT>(a.is_zero(), 4), inf_q = lane_flag<F, SPLIT>(b.is_zero(), 4);
  const F l1 = lane_product<SPLIT>(a, b);
  const F other = lane_from<SPLIT>(l1, role ^ 1);
  const F d = lane_select(role & 1, l1 - other, other - l1);  // roles 0, 1: P; 2, 3: R
  const bool p_zero = lane_flag<F, SPLIT>(d.is_zero(), 0), r_zero = lane_flag<F, SPLIT>(d.is_zero(), 2);
  const F sq = lane_square(d);                                  // PP; RR
  const F l3 = lane_product<SPLIT>(lane_select(role == 1, d, l1), lane_from<SPLIT>(sq, 0));  // Q, PPP, -, -, ZZ3
  const F qq = lane_from<SPLIT>(l3, 0), ppp = lane_from<SPLIT>(l3, 1);
  const F x3 = (sq - ppp) - dbl(qq);
  // 2: S1 PPP, 3: R (Q - X3), 5: ZZZ3
  const F l4 = lane_product<SPLIT>(lane_select(role == 3, d, l1), lane_select(role == 3, qq - x3, ppp));
  const F y3 = l4 - lane_from<SPLIT>(l4, 2);
  __syncwarp();
  if (!active) return;
  if (inf_p || inf_q) {
    const uint32_t* const src = inf_p ? q : p;
    if (src != out && role < 4) lane_store_elem(out + role * W, load_elem<F>(src + role * W));
  } else if (p_zero) {
    if ((threadIdx.x & (LaneGroup<F, SPLIT>::kLanes - 1)) == 0)
      store_xyzz(out, r_zero ? xyzz_double_call(load_xyzz<F>(p)) : xyzz_infinity<F>());
  } else if (role == 3) {
    lane_store_elem(out, x3);
    lane_store_elem(out + W, y3);
  } else if (role == 4) {
    lane_store_elem(out + 2 * W, l3);
  } else if (role == 5) {
    lane_store_elem(out + 3 * W, l4);
  }
}

}  // namespace zkg
