// NTT passes on 32-bit words: radix-4 butterflies in registers, products by twiddles with a
// precomputed quotient (field_shoup.cuh), unreduced sums.
//
// A pass of s stages works on tiles of 2^tl elements, 2^(tl - s) columns of 2^s rows. A thread
// holds four rows of one column and runs two stages on them per step; between steps the tile goes
// through shared memory (16-byte pieces, one array per half element, so that neighbouring lanes
// never share a bank), the first step reads global memory and the last one writes it. What bounds
// the pass is the wide multiply-add pipe: four products (428 of its slots) per four elements and
// step beside ~400 add-pipe instructions; a butterfly takes about 240 instructions, where the
// double-precision form of the same butterfly took about 570. At 2^22 the pipe is 60-76% busy in a
// pass; the rest goes to the tiles' loads and stores, which other blocks' products cover in part.
//
// Bounds: r < 0.19 2^256, so 5r < 2^256. Elements between steps are below 2r; a sum of two is
// brought below 2r again by one conditional subtraction of 2r; a difference gets 2r added and is a
// product's operand (below 4r), and the product by a twiddle is below 1.757r (field_shoup.cuh): the
// conditional subtraction that follows it too (`times`) finds nothing to take off.
#pragma once
#include "field_shoup.cuh"

namespace zkg {
namespace words {

__device__ __forceinline__ Fr add_raw(const Fr& a, const Fr& b) {
  Fr s;
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

// Word j of 2r.
__host__ __device__ constexpr uint32_t two_r(int j) {
  constexpr uint32_t p[8] = {FrParams::P0, FrParams::P1, FrParams::P2, FrParams::P3,
                             FrParams::P4, FrParams::P5, FrParams::P6, FrParams::P7};
  return j == 0 ? p[0] << 1 : p[j] << 1 | p[j - 1] >> 31;
}

// a - b + 2r (b <= a + 2r).
__device__ __forceinline__ Fr sub_raw(const Fr& a, const Fr& b) {
  Fr d;
  asm("sub.cc.u32  %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32    %7, %15, %23;"
      : "=&r"(d.w[0]), "=&r"(d.w[1]), "=&r"(d.w[2]), "=&r"(d.w[3]), "=&r"(d.w[4]), "=&r"(d.w[5]), "=&r"(d.w[6]),
        "=&r"(d.w[7])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
        "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]));
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(d.w[0]), "+r"(d.w[1]), "+r"(d.w[2]), "+r"(d.w[3]), "+r"(d.w[4]), "+r"(d.w[5]), "+r"(d.w[6]), "+r"(d.w[7])
      : "n"(two_r(0)), "n"(two_r(1)), "n"(two_r(2)), "n"(two_r(3)), "n"(two_r(4)), "n"(two_r(5)), "n"(two_r(6)),
        "n"(two_r(7)));
  return d;
}

// x - 2r when x >= 2r, else x: below 2r for x below 4r.
__device__ __forceinline__ Fr reduce_2r(const Fr& x) {
  Fr d, r;
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
        "n"(two_r(0)), "n"(two_r(1)), "n"(two_r(2)), "n"(two_r(3)), "n"(two_r(4)), "n"(two_r(5)), "n"(two_r(6)),
        "n"(two_r(7)));
#pragma unroll
  for (int i = 0; i < 8; i++) r.w[i] = borrow ? x.w[i] : d.w[i];
  return r;
}

// A thread's place in step st of a pass: column and first of its four rows, `gap` rows apart.
struct Rows {
  uint32_t col, row, gap;
};
__device__ __forceinline__ Rows rows_of(uint32_t u, uint32_t lg, uint32_t gap_log) {
  const uint32_t q = u >> lg;
  return Rows{u & ((1u << lg) - 1), ((q >> gap_log) << (gap_log + 2)) + (q & ((1u << gap_log) - 1)), 1u << gap_log};
}

}  // namespace words

// The pass table for tiles of 2^tl elements (ntt_stage_twiddles' order, a shoup::Constant of 64 bytes
// per entry): a block of 2^tl entries per distinct tile, stage st's 2^(tl - st - 1) twiddles from entry
// 2^tl - 2^(tl - st) on, butterfly b's at b mod their number.
__global__ void ntt_words_twiddles(const uint32_t* __restrict__ hi, const uint32_t* __restrict__ lo, uint32_t lo_bits,
                                   uint32_t log_n, uint32_t tl, uint32_t lm, uint32_t s, size_t entries,
                                   uint32_t* __restrict__ out) {
  const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= entries) return;
  const uint32_t elems = 1u << tl, lg = tl - s;
  const uint32_t block = (uint32_t)(id >> tl), off = (uint32_t)(id & (elems - 1));
  const uint32_t left = elems - 1 - off;  // stage st holds left in [2^(tl-st-1), 2^(tl-st) - 1]
  const uint32_t st = left == 0 ? tl : tl - 1 - (31 - __clz(left));
  if (st >= s) return;  // the block's last 2^lg entries are not used
  const uint32_t e = off - (elems - (elems >> st));
  const uint32_t j0 = ((block << lg) + (e & ((1u << lg) - 1))) & ((1u << lm) - 1);
  const uint32_t idx = (((e >> lg) << lm) + j0) << (log_n - lm - s + st);  // < n / 2
  const shoup::Constant c = shoup::constant(load_fe<Fr>(hi + 8 * (size_t)(idx >> lo_bits)) *
                                            load_fe<Fr>(lo + 8 * (size_t)(idx & ((1u << lo_bits) - 1))));
  store_fe(out + 16 * id, c.w);
  store_fe(out + 16 * id + 8, c.quotient);
}

// One pass: stages [log_n - lm - s, log_n - lm), 2 <= s <= tl, with 2^(tl - 2) threads. LAST writes
// canonical words in natural order, with the 1/n scaling of an inverse, the fused coset shift
// (sh_hi != null) or the fused quotient (qa != null).
template <bool LAST, uint32_t THREADS, uint32_t BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS)
    ntt_pass_words(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, const uint32_t* __restrict__ tw,
                   uint32_t tw_mask, uint32_t log_n, uint32_t tl, uint32_t lm, uint32_t s, int scale_flag, Fr scale,
                   const uint32_t* __restrict__ sh_hi, const uint32_t* __restrict__ sh_lo, uint32_t sh_bits,
                   const uint32_t* __restrict__ qa, const uint32_t* __restrict__ qb, Fr qz2) {
  using namespace words;
  extern __shared__ __align__(16) uint4 pieces[];  // low halves of the tile's elements, then high halves
  const uint32_t lg = tl - s, tile = blockIdx.x, elems = 1u << tl;
  const uint32_t* const table = tw + 16 * ((size_t)(tile & tw_mask) << tl);
  // x times twiddle e of stage st, below 2r
  auto times = [&](const Fr& x, uint32_t st, uint32_t e) {
    const uint4* p = reinterpret_cast<const uint4*>(table + 16 * (size_t)(elems - (elems >> st) + e));
    const uint4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3);
    return reduce_2r(shoup::mul(x, shoup::Constant{Fr{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}},
                                                   Fr{{c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w}}}));
  };
  Fr v[4];
  for (uint32_t st = 0; st < s; st += 2) {
    const bool pair = st + 1 < s;  // the last step of an odd pass has one stage
    const Rows at = rows_of(threadIdx.x, lg, pair ? s - 2 - st : 0);
    const uint32_t slot = (at.row << lg) + at.col, gap = at.gap << lg;
    if (st == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++)
        v[k] = load_fe_cg<Fr>(src + 8 * (size_t)tile_global_index(tile, slot + k * gap, lg, lm, s));
    } else {
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint4 lo = pieces[slot + k * gap], hi = pieces[elems + slot + k * gap];
        v[k] = Fr{{lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w}};
      }
      __syncthreads();
    }
    const bool unit = LAST && lm == 0 && st + (pair ? 2 : 1) == s;  // the transform's last stages: twiddles 1 and w^(n/4)
    if (pair) {
      const uint32_t e0 = ((at.row & (at.gap - 1)) << lg) + at.col;
      const Fr y0 = reduce_2r(add_raw(v[0], v[2])), y1 = reduce_2r(add_raw(v[1], v[3]));
      Fr y2 = sub_raw(v[0], v[2]);
      y2 = unit ? reduce_2r(y2) : times(y2, st, e0);
      const Fr y3 = times(sub_raw(v[1], v[3]), st, e0 + gap);
      v[0] = reduce_2r(add_raw(y0, y1));
      v[2] = reduce_2r(add_raw(y2, y3));
      if (unit) {
        v[1] = reduce_2r(sub_raw(y0, y1));
        v[3] = reduce_2r(sub_raw(y2, y3));
      } else {
        v[1] = times(sub_raw(y0, y1), st + 1, e0);
        v[3] = times(sub_raw(y2, y3), st + 1, e0);
      }
    } else {  // rows (0, 1) and (2, 3)
      Fr d0 = sub_raw(v[0], v[1]), d1 = sub_raw(v[2], v[3]);
      v[0] = reduce_2r(add_raw(v[0], v[1]));
      v[2] = reduce_2r(add_raw(v[2], v[3]));
      if (unit) {
        v[1] = reduce_2r(d0);
        v[3] = reduce_2r(d1);
      } else {
        v[1] = times(d0, st, at.col);
        v[3] = times(d1, st, at.col);
      }
    }
    if (st + 2 < s) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        pieces[slot + k * gap] = make_uint4(v[k].w[0], v[k].w[1], v[k].w[2], v[k].w[3]);
        pieces[elems + slot + k * gap] = make_uint4(v[k].w[4], v[k].w[5], v[k].w[6], v[k].w[7]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        uint32_t g = tile_global_index(tile, slot + k * gap, lg, lm, s);
        Fr out = v[k];
        if (LAST) {
          g = __brev(g) >> (32 - log_n);
          if (sh_hi != nullptr)
            out = out * (load_fe<Fr>(sh_hi + 8 * (size_t)(g >> sh_bits)) *
                         load_fe<Fr>(sh_lo + 8 * (size_t)(g & ((1u << sh_bits) - 1))));
          else if (scale_flag)
            out = out * scale;
          else
            out = reduce_once(out);
          if (qa != nullptr)
            out = quotient_element(load_fe<Fr>(qa + 8 * (size_t)g), load_fe<Fr>(qb + 8 * (size_t)g), out, qz2);
        }
        store_fe(dst + 8 * (size_t)g, out);
      }
    }
  }
}

}  // namespace zkg
