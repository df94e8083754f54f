// field.cuh — BN254 Fr / Fq arithmetic for sm_100a on 8 x 32-bit limbs.
//
// Elements are 256-bit little-endian integers in Montgomery form with
// R = 2^256 — bit-identical to the reference's BigNum (cuda/bn256.h:10-13,
// 4 x u64 LE) and to halo2curves' Fr / Fq repr, so device buffers are the
// host buffers reinterpreted.  The moduli (cuda/bn256.h:37, :54) are both
// < 2^254, so 4p < R, which allows "lazy" forms:
//   mul_lazy : a, b < 2p  ->  a*b*R^-1 mod p  in [0, 2p)   (no final subtract)
//   add_lazy : a, b < 2p  ->  a + b           in [0, 2p)
//   sub_lazy : a, b < 2p  ->  a - b           in [0, 2p)
// and canonical forms (inputs < p, outputs < p) used where values are
// compared.  Every carry chain lives inside ONE asm statement: the carry
// flag is never assumed to survive between statements (the reference's
// gpu_math.h:31-77 macros rely on that; this file does not).
//
// The Montgomery product (mul_lazy) is described where it is defined.
#pragma once
#include <cstdint>

namespace zk {

struct fe {
  uint32_t w[8];
};

// ---- moduli (cuda/bn256.h:37-56) ----------------------------------------
struct FrP {
  static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xefffffffu;  // -p^-1 mod 2^32
  // R mod p (Montgomery one)
  static constexpr uint32_t O0 = 0x4ffffffbu, O1 = 0xac96341cu, O2 = 0x9f60cd29u, O3 = 0x36fc7695u,
                            O4 = 0x7879462eu, O5 = 0x666ea36fu, O6 = 0x9a07df2fu, O7 = 0x0e0a77c1u;
};
struct FqP {
  static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xe4866389u;
  static constexpr uint32_t O0 = 0xc58f0d9du, O1 = 0xd35d438du, O2 = 0xf5c70b3du, O3 = 0x0a78eb28u,
                            O4 = 0x7879462cu, O5 = 0x666ea36fu, O6 = 0x9a07df2fu, O7 = 0x0e0a77c1u;
};

#define ZK_A_OPS(a) "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7])

// ---- Montgomery product ----------------------------------------------------
// r = a b 2^-256 mod p on 32-bit words: Montgomery's product with the reduction
// interleaved row by row, the sums of even and odd columns in carry chains of
// their own, a published arrangement of wide products on multiply-add pairs
// that other GPU libraries use too.  The running sum T is kept as two
// column chains: E holds word pairs at even positions, O at odd ones, so each
// 32 x 32-bit product lands in one aligned pair and a row of four products is
// one lo/hi multiply-add chain whose carries run from pair to pair.  A row
// multiplies a by one word of b, then adds m p (m = T_0 (-p^-1) mod 2^32) and
// drops T_0: the chains change places, and the shift by one word rides on the
// next row's odd chain, which takes E two words up as its addend.
//
// What bounds it (B200, cycles per warp instruction on one of an SM's four
// schedulers, measured with independent chains): a lo/hi multiply-add pair
// 4.2, an FP64 multiply-add 2.0, an add 1.0, an add with carry or a logic or
// shift instruction 2.0; a pair and an FP64 multiply-add do not overlap (6.6
// for one of each).  The 128 pairs of a product are 534 cycles of its 555
// (66-68 G products/s in a loop, 40 registers).  The same product on the FP64
// pipe (five 52-bit limbs, two multiply-adds and a subtraction per exact
// partial product) took 600-635 cycles (59-62 G/s) at 80 registers there, and
// 840 in the NTT passes, whose other values leave it fewer registers.
//
// Bounds: every row keeps T < (a + p) 2^32 (1 + 2^-32), below 2^288 for
// a < 4p, so the chains never carry out of word 8; r < a b / 2^256 + p, which
// is < 2p for a, b < 2p and for a < 4p, b < p.
// A += (x0, x1, x2, x3) * b over the four word pairs of A
#define ZK_ROW_CHAIN                \
  "mad.lo.cc.u32  %0, %8, %12, %0;\n\t"  \
  "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"  \
  "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"  \
  "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"  \
  "madc.lo.cc.u32 %4, %10, %12, %4;\n\t" \
  "madc.hi.cc.u32 %5, %10, %12, %5;\n\t" \
  "madc.lo.cc.u32 %6, %11, %12, %6;\n\t" \
  "madc.hi.u32    %7, %11, %12, %7;"
#define ZK_ROW_CHAIN_C              \
  "mad.lo.cc.u32  %0, %9, %13, %0;\n\t"  \
  "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"  \
  "madc.lo.cc.u32 %2, %10, %13, %2;\n\t" \
  "madc.hi.cc.u32 %3, %10, %13, %3;\n\t" \
  "madc.lo.cc.u32 %4, %11, %13, %4;\n\t" \
  "madc.hi.cc.u32 %5, %11, %13, %5;\n\t" \
  "madc.lo.cc.u32 %6, %12, %13, %6;\n\t" \
  "madc.hi.cc.u32 %7, %12, %13, %7;\n\t" \
  "addc.u32       %8, %8, 0;"
#define ZK_A8(A) "+r"(A[0]), "+r"(A[1]), "+r"(A[2]), "+r"(A[3]), "+r"(A[4]), "+r"(A[5]), "+r"(A[6]), "+r"(A[7])

__device__ __forceinline__ void row_mad(uint32_t A[8], uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t b) {
  asm(ZK_ROW_CHAIN : ZK_A8(A) : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b));
}
// the same with the carry out of the top pair added to `top`
__device__ __forceinline__ void row_mad_c(uint32_t A[8], uint32_t& top, uint32_t x0, uint32_t x1, uint32_t x2,
                                          uint32_t x3, uint32_t b) {
  asm(ZK_ROW_CHAIN_C : ZK_A8(A), "+r"(top) : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b));
}
__device__ __forceinline__ void row_mul(uint32_t A[8], uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t b) {
  const uint64_t p0 = (uint64_t)x0 * b, p1 = (uint64_t)x1 * b, p2 = (uint64_t)x2 * b, p3 = (uint64_t)x3 * b;
  A[0] = (uint32_t)p0; A[1] = (uint32_t)(p0 >> 32); A[2] = (uint32_t)p1; A[3] = (uint32_t)(p1 >> 32);
  A[4] = (uint32_t)p2; A[5] = (uint32_t)(p2 >> 32); A[6] = (uint32_t)p3; A[7] = (uint32_t)(p3 >> 32);
}
// N = (E >> 64) + (x0..x3) * b with the carry of o0 += E[1] coming in below
__device__ __forceinline__ void row_mad_shift(uint32_t N[8], const uint32_t E[8], uint32_t& o0, uint32_t x0,
                                              uint32_t x1, uint32_t x2, uint32_t x3, uint32_t b) {
  asm("add.cc.u32     %8, %8, %9;\n\t"
      "madc.lo.cc.u32 %0, %16, %20, %10;\n\t"
      "madc.hi.cc.u32 %1, %16, %20, %11;\n\t"
      "madc.lo.cc.u32 %2, %17, %20, %12;\n\t"
      "madc.hi.cc.u32 %3, %17, %20, %13;\n\t"
      "madc.lo.cc.u32 %4, %18, %20, %14;\n\t"
      "madc.hi.cc.u32 %5, %18, %20, %15;\n\t"
      "madc.lo.cc.u32 %6, %19, %20, 0;\n\t"
      "madc.hi.u32    %7, %19, %20, 0;"
      : "=&r"(N[0]), "=&r"(N[1]), "=&r"(N[2]), "=&r"(N[3]), "=&r"(N[4]), "=&r"(N[5]), "=&r"(N[6]), "=&r"(N[7]),
        "+r"(o0)
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(x0), "r"(x1), "r"(x2),
        "r"(x3), "r"(b));
}
// r = (E >> 32) + O
__device__ __forceinline__ void merge_chains(uint32_t r[8], const uint32_t E[8], const uint32_t O[8]) {
  asm("add.cc.u32  %0, %8, %15;\n\t"
      "addc.cc.u32 %1, %9, %16;\n\t"
      "addc.cc.u32 %2, %10, %17;\n\t"
      "addc.cc.u32 %3, %11, %18;\n\t"
      "addc.cc.u32 %4, %12, %19;\n\t"
      "addc.cc.u32 %5, %13, %20;\n\t"
      "addc.cc.u32 %6, %14, %21;\n\t"
      "addc.u32    %7, %22, 0;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(O[0]), "r"(O[1]), "r"(O[2]),
        "r"(O[3]), "r"(O[4]), "r"(O[5]), "r"(O[6]), "r"(O[7]));
}

template <class P>
__device__ __forceinline__ void mul_lazy(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t E[8], O[8];
  row_mul(E, a[0], a[2], a[4], a[6], b[0]);
  row_mul(O, a[1], a[3], a[5], a[7], b[0]);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if (i > 0) {
      uint32_t N[8];
      row_mad_shift(N, E, O[0], a[1], a[3], a[5], a[7], b[i]);
#pragma unroll
      for (int j = 0; j < 8; j++) E[j] = O[j], O[j] = N[j];
      row_mad_c(E, O[7], a[0], a[2], a[4], a[6], b[i]);
    }
    const uint32_t m = E[0] * P::INV;
    row_mad(O, P::P1, P::P3, P::P5, P::P7, m);
    row_mad_c(E, O[7], P::P0, P::P2, P::P4, P::P6, m);
  }
  merge_chains(r, E, O);
}

// The same product as a call of one out-of-line function: operands and
// result pass by value (in registers), so a kernel that runs many products
// keeps one copy of the product's code in the instruction cache instead of
// one inlined copy per call site.
struct Fe8 {
  uint32_t w[8];
};
template <class P>
__device__ __noinline__ Fe8 mul_call(const Fe8 a, const Fe8 b) {
  Fe8 r;
  mul_lazy<P>(r.w, a.w, b.w);
  return r;
}
template <class P>
__device__ __forceinline__ void mul_out(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  Fe8 av, bv;
#pragma unroll
  for (int k = 0; k < 8; k++) av.w[k] = a[k], bv.w[k] = b[k];
  const Fe8 rv = mul_call<P>(av, bv);
#pragma unroll
  for (int k = 0; k < 8; k++) r[k] = rv.w[k];
}

// ---- products by tabulated multiplicands -----------------------------------
// Half of a Montgomery product's 128 multiply-add pairs go into its reduction.
// For a multiplicand w that is known beforehand (a root of unity, a twist),
// tables of w 2^(32 s) mod p let rows of a that lie 32 s bits apart share one
// reduction, so that only a few words are left to reduce:
//   mul_w4: w^(k) = w 2^(64 k + 96) mod p, k < 4 (128 B): a = sum_k A_k 2^(64 k),
//     V = sum_k A_k w^(k) < 4 2^64 p, three words reduced: 64 + 24 pairs;
//   mul_w2: w^(k) = w 2^(128 k + 160) mod p, k < 2 (64 B): four words and one
//     more reduced: 64 + 40 pairs.
// Both take any a < 2^256 (5.29 p) and return a w mod p below p (1 + 2^-29),
// in the form (Montgomery or not) a has; the last reduced word is there for
// that bound, which lets a radix-8 butterfly add eight such values without
// conditional subtractions in between.  Cycles per warp on one scheduler
// (B200): 555 mul_lazy, 440 mul_w2, 390 mul_w4.

// A += x b over the four pairs of A[0..7], the carry into the two words above
__device__ __forceinline__ void row_mad_cc(uint32_t A[10], uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                           uint32_t b) {
  asm("mad.lo.cc.u32  %0, %10, %14, %0;\n\t"
      "madc.hi.cc.u32 %1, %10, %14, %1;\n\t"
      "madc.lo.cc.u32 %2, %11, %14, %2;\n\t"
      "madc.hi.cc.u32 %3, %11, %14, %3;\n\t"
      "madc.lo.cc.u32 %4, %12, %14, %4;\n\t"
      "madc.hi.cc.u32 %5, %12, %14, %5;\n\t"
      "madc.lo.cc.u32 %6, %13, %14, %6;\n\t"
      "madc.hi.cc.u32 %7, %13, %14, %7;\n\t"
      "addc.cc.u32    %8, %8, 0;\n\t"
      "addc.u32       %9, %9, 0;"
      : ZK_A8(A), "+r"(A[8]), "+r"(A[9])
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(b));
}
// One reduced word on the chains E (E[0] = 0 already dropped into E[1..7] and
// E89 = words 8, 9 of E) and O: afterwards E is the old O plus m p's even
// words, O the old E >> 64 plus its odd ones.
template <class P>
__device__ __forceinline__ void reduce_word(uint32_t E[8], uint32_t O[8], uint32_t e8, uint32_t e9) {
  uint32_t N[8], m;
  asm("add.cc.u32     %8, %8, %10;\n\t"
      "mul.lo.u32     %9, %8, %19;\n\t"
      "madc.lo.cc.u32 %0, %9, %20, %11;\n\t"
      "madc.hi.cc.u32 %1, %9, %20, %12;\n\t"
      "madc.lo.cc.u32 %2, %9, %21, %13;\n\t"
      "madc.hi.cc.u32 %3, %9, %21, %14;\n\t"
      "madc.lo.cc.u32 %4, %9, %22, %15;\n\t"
      "madc.hi.cc.u32 %5, %9, %22, %16;\n\t"
      "madc.lo.cc.u32 %6, %9, %23, %17;\n\t"
      "madc.hi.u32    %7, %9, %23, %18;"
      : "=&r"(N[0]), "=&r"(N[1]), "=&r"(N[2]), "=&r"(N[3]), "=&r"(N[4]), "=&r"(N[5]), "=&r"(N[6]), "=&r"(N[7]),
        "+r"(O[0]), "=&r"(m)
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(e8), "r"(e9), "n"(P::INV),
        "n"(P::P1), "n"(P::P3), "n"(P::P5), "n"(P::P7));
  row_mad_c(O, N[7], P::P0, P::P2, P::P4, P::P6, m);
#pragma unroll
  for (int j = 0; j < 8; j++) E[j] = O[j], O[j] = N[j];
}

// Table words through a loader: w(k, v) puts the eight words of w^(k) in v.
template <class P, class W>
__device__ __forceinline__ void mul_w4(uint32_t r[8], const uint32_t a[8], W w) {
  uint32_t E[10], O[8], o8 = 0, v[8];
  w(0, v);
  row_mul(E, v[0], v[2], v[4], v[6], a[0]);
  E[8] = E[9] = 0;
  row_mul(O, v[1], v[3], v[5], v[7], a[0]);
  row_mad_c(O, o8, v[0], v[2], v[4], v[6], a[1]);
  row_mad(E + 2, v[1], v[3], v[5], v[7], a[1]);
#pragma unroll
  for (int k = 1; k < 4; k++) {
    w(k, v);
    row_mad_cc(E, v[0], v[2], v[4], v[6], a[2 * k]);
    row_mad_c(O, o8, v[1], v[3], v[5], v[7], a[2 * k]);
    row_mad_c(O, o8, v[0], v[2], v[4], v[6], a[2 * k + 1]);
    row_mad(E + 2, v[1], v[3], v[5], v[7], a[2 * k + 1]);
  }
  const uint32_t m = E[0] * P::INV;
  row_mad_cc(E, P::P0, P::P2, P::P4, P::P6, m);
  row_mad_c(O, o8, P::P1, P::P3, P::P5, P::P7, m);
  reduce_word<P>(E, O, E[8], E[9] + o8);
  reduce_word<P>(E, O, 0u, 0u);
  merge_chains(r, E, O);
}
template <class P>
__device__ __forceinline__ void mul_w2(uint32_t r[8], const uint32_t a[8], const uint32_t v[8], const uint32_t w[8]) {
  uint32_t E[8], O[8];
  row_mul(E, v[0], v[2], v[4], v[6], a[0]);
  row_mul(O, v[1], v[3], v[5], v[7], a[0]);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (i > 0) {
      uint32_t N[8];
      row_mad_shift(N, E, O[0], v[1], v[3], v[5], v[7], a[i]);
#pragma unroll
      for (int j = 0; j < 8; j++) E[j] = O[j], O[j] = N[j];
      row_mad_c(E, O[7], v[0], v[2], v[4], v[6], a[i]);
    }
    row_mad(O, w[1], w[3], w[5], w[7], a[i + 4]);
    row_mad_c(E, O[7], w[0], w[2], w[4], w[6], a[i + 4]);
    const uint32_t m = E[0] * P::INV;
    row_mad(O, P::P1, P::P3, P::P5, P::P7, m);
    row_mad_c(E, O[7], P::P0, P::P2, P::P4, P::P6, m);
  }
  reduce_word<P>(E, O, 0u, 0u);
  merge_chains(r, E, O);
}

// mul_w8: w^(k) = w 2^(32 k + 64) mod p, k < 8 (256 B), V < 8 2^32 p, two words
// reduced: 64 + 16 pairs; the result is below p (1 + 2^-28).
template <class P, class W>
__device__ __forceinline__ void mul_w8(uint32_t r[8], const uint32_t a[8], W w) {
  uint32_t E[8], O[8], e8 = 0, o8 = 0, v[8];
  w(0, v);
  row_mul(E, v[0], v[2], v[4], v[6], a[0]);
  row_mul(O, v[1], v[3], v[5], v[7], a[0]);
#pragma unroll
  for (int k = 1; k < 8; k++) {
    w(k, v);
    row_mad_c(E, e8, v[0], v[2], v[4], v[6], a[k]);
    row_mad_c(O, o8, v[1], v[3], v[5], v[7], a[k]);
  }
  const uint32_t m = E[0] * P::INV;
  row_mad_c(E, e8, P::P0, P::P2, P::P4, P::P6, m);
  row_mad_c(O, o8, P::P1, P::P3, P::P5, P::P7, m);
  reduce_word<P>(E, O, e8, o8);
  merge_chains(r, E, O);
}

// word j of K p (K p < 2^256: K <= 5)
template <class P, uint32_t K>
__host__ __device__ constexpr uint32_t kp(int j) {
  uint64_t c = 0;
  for (int i = 0; i <= j; i++) {
    const uint32_t w = i == 0   ? P::P0
                       : i == 1 ? P::P1
                       : i == 2 ? P::P2
                       : i == 3 ? P::P3
                       : i == 4 ? P::P4
                       : i == 5 ? P::P5
                       : i == 6 ? P::P6
                                : P::P7;
    c = (c >> 32) + (uint64_t)w * K;
  }
  return (uint32_t)c;
}
#define ZK_KP_OPS(P, K)                                                                                      \
  "n"(kp<P, K>(0)), "n"(kp<P, K>(1)), "n"(kp<P, K>(2)), "n"(kp<P, K>(3)), "n"(kp<P, K>(4)), "n"(kp<P, K>(5)), \
      "n"(kp<P, K>(6)), "n"(kp<P, K>(7))

// r = a + b (no reduction)
__device__ __forceinline__ void add_raw(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : ZK_A_OPS(a), ZK_A_OPS(b));
}
// r = a + K p - b (the caller keeps it within [0, 2^256))
template <class P, uint32_t K>
__device__ __forceinline__ void sub_off(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t t[8];
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
      : ZK_A_OPS(a), ZK_KP_OPS(P, K));
  asm("sub.cc.u32  %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32    %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : ZK_A_OPS(t), ZK_A_OPS(b));
}
// x -= K p if x >= K p
template <class P, uint32_t K>
__device__ __forceinline__ void cond_sub(uint32_t x[8]) {
  uint32_t t[8], borrow;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(borrow)
      : ZK_A_OPS(x), ZK_KP_OPS(P, K));
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = borrow ? x[j] : t[j];
}

// r = a + b - 2p if that does not borrow, else a + b.  Inputs < 2p.
template <class P>
__device__ __forceinline__ void add_lazy(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t s[8], t[8], borrow;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
      : ZK_A_OPS(a), ZK_A_OPS(b));
  // t = s - 2p
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(borrow)
      : ZK_A_OPS(s), "n"((uint32_t)(P::P0 << 1)), "n"((P::P1 << 1) | (P::P0 >> 31)), "n"((P::P2 << 1) | (P::P1 >> 31)),
        "n"((P::P3 << 1) | (P::P2 >> 31)), "n"((P::P4 << 1) | (P::P3 >> 31)), "n"((P::P5 << 1) | (P::P4 >> 31)),
        "n"((P::P6 << 1) | (P::P5 >> 31)), "n"((P::P7 << 1) | (P::P6 >> 31)));
#pragma unroll
  for (int j = 0; j < 8; j++) r[j] = borrow ? s[j] : t[j];
}

// r = a - b, plus 2p if that borrowed.  Inputs < 2p.
template <class P>
__device__ __forceinline__ void sub_lazy(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t d[8], borrow;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(borrow)
      : ZK_A_OPS(a), ZK_A_OPS(b));
  // conditional + 2p (mask form keeps it branch-free)
  const uint32_t mk = borrow;  // 0 or 0xffffffff
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7])
      : "r"(mk & (uint32_t)(P::P0 << 1)), "r"(mk & ((P::P1 << 1) | (P::P0 >> 31))), "r"(mk & ((P::P2 << 1) | (P::P1 >> 31))),
        "r"(mk & ((P::P3 << 1) | (P::P2 >> 31))), "r"(mk & ((P::P4 << 1) | (P::P3 >> 31))),
        "r"(mk & ((P::P5 << 1) | (P::P4 >> 31))), "r"(mk & ((P::P6 << 1) | (P::P5 >> 31))),
        "r"(mk & ((P::P7 << 1) | (P::P6 >> 31))));
#pragma unroll
  for (int j = 0; j < 8; j++) r[j] = d[j];
}

// Reduce a value < 2p to canonical [0, p).
template <class P>
__device__ __forceinline__ void reduce_once(uint32_t r[8], const uint32_t a[8]) {
  uint32_t t[8], borrow;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(borrow)
      : ZK_A_OPS(a), "n"(P::P0), "n"(P::P1), "n"(P::P2), "n"(P::P3), "n"(P::P4), "n"(P::P5), "n"(P::P6), "n"(P::P7));
#pragma unroll
  for (int j = 0; j < 8; j++) r[j] = borrow ? a[j] : t[j];
}

// ---- canonical forms (inputs < p, outputs < p) ---------------------------
template <class P>
__device__ __forceinline__ void mul(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t t[8];
  mul_lazy<P>(t, a, b);
  reduce_once<P>(r, t);
}
template <class P>
__device__ __forceinline__ void sqr(uint32_t r[8], const uint32_t a[8]) {
  mul<P>(r, a, a);
}
template <class P>
__device__ __forceinline__ void add(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t s[8];
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
      : ZK_A_OPS(a), ZK_A_OPS(b));
  reduce_once<P>(r, s);
}
template <class P>
__device__ __forceinline__ void sub(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  uint32_t d[8], borrow;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(borrow)
      : ZK_A_OPS(a), ZK_A_OPS(b));
  const uint32_t mk = borrow;
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7])
      : "r"(mk & P::P0), "r"(mk & P::P1), "r"(mk & P::P2), "r"(mk & P::P3), "r"(mk & P::P4), "r"(mk & P::P5),
        "r"(mk & P::P6), "r"(mk & P::P7));
#pragma unroll
  for (int j = 0; j < 8; j++) r[j] = d[j];
}
template <class P>
__device__ __forceinline__ void dbl(uint32_t r[8], const uint32_t a[8]) {
  add<P>(r, a, a);
}

__device__ __forceinline__ bool is_zero(const uint32_t a[8]) {
  return (a[0] | a[1] | a[2] | a[3] | a[4] | a[5] | a[6] | a[7]) == 0;
}
__device__ __forceinline__ bool eq(const uint32_t a[8], const uint32_t b[8]) {
  return ((a[0] ^ b[0]) | (a[1] ^ b[1]) | (a[2] ^ b[2]) | (a[3] ^ b[3]) | (a[4] ^ b[4]) | (a[5] ^ b[5]) |
          (a[6] ^ b[6]) | (a[7] ^ b[7])) == 0;
}
template <class P>
__device__ __forceinline__ void set_one(uint32_t r[8]) {
  r[0] = P::O0; r[1] = P::O1; r[2] = P::O2; r[3] = P::O3;
  r[4] = P::O4; r[5] = P::O5; r[6] = P::O6; r[7] = P::O7;
}
__device__ __forceinline__ void set_zero(uint32_t r[8]) {
#pragma unroll
  for (int j = 0; j < 8; j++) r[j] = 0;
}
__device__ __forceinline__ void cpy(uint32_t r[8], const uint32_t a[8]) {
#pragma unroll
  for (int j = 0; j < 8; j++) r[j] = a[j];
}

// a^e for a small exponent (canonical inputs), square-and-multiply
template <class P>
__device__ __forceinline__ void pow_u64(uint32_t r[8], const uint32_t a[8], uint64_t e) {
  uint32_t acc[8], base[8];
  set_one<P>(acc);
  cpy(base, a);
  while (e) {
    if (e & 1) mul<P>(acc, acc, base);
    e >>= 1;
    if (e) sqr<P>(base, base);
  }
  cpy(r, acc);
}

// ---- global memory element access (32 B = one sector, two 16 B vectors) --
__device__ __forceinline__ void ld_fe(uint32_t r[8], const fe* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 x = q[0], y = q[1];
  r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w;
  r[4] = y.x; r[5] = y.y; r[6] = y.z; r[7] = y.w;
}
__device__ __forceinline__ void ld_fe_nc(uint32_t r[8], const fe* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 x = __ldg(q), y = __ldg(q + 1);
  r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w;
  r[4] = y.x; r[5] = y.y; r[6] = y.z; r[7] = y.w;
}
// through L2 only: data another CTA of the same launch may have written
__device__ __forceinline__ void ld_fe_cg(uint32_t r[8], const fe* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 x = __ldcg(q), y = __ldcg(q + 1);
  r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w;
  r[4] = y.x; r[5] = y.y; r[6] = y.z; r[7] = y.w;
}
__device__ __forceinline__ void st_fe(fe* p, const uint32_t r[8]) {
  uint4* q = reinterpret_cast<uint4*>(p);
  q[0] = make_uint4(r[0], r[1], r[2], r[3]);
  q[1] = make_uint4(r[4], r[5], r[6], r[7]);
}

}  // namespace zk
