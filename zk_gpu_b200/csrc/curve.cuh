// curve.cuh — BN254 G1 (y^2 = x^3 + 3 over Fq) on device, XYZZ coordinates.
//
// A point (X, Y, ZZ, ZZZ) represents x = X/ZZ, y = Y/ZZZ with ZZ^3 = ZZZ^2;
// the identity is ZZ = 0.  Formulas are the EFD's "xyzz" set for a = 0:
// dbl-2008-s-1 (6M + 3S), mdbl-2008-s-1, madd-2008-s (8M + 2S) and
// add-2008-s (12M + 2S), with the degenerate cases (P == Q -> doubling,
// P == -Q -> identity) handled explicitly, which the reference's Jacobian
// code gets wrong (cuda/curve.cuh:13-20, 170-179: its "identity" (0,0,R) is
// not recognised as zero afterwards).  Affine inputs use (0, 0) for the
// identity (cuda/bn256.h:15-20).
//
// Arithmetic form: coordinates are in the R = 2^256 Montgomery form the API
// holds in memory (bit-identical to halo2curves), lazily reduced in [0, 2q);
// values are made canonical only where they are compared with zero.
#pragma once
#include "field.cuh"

namespace zk {

using P_q = FqP;

struct xyzz_t {
  uint32_t x[8], y[8], zz[8], zzz[8];
};
struct aff_t {
  uint32_t x[8], y[8];
};

// ---- lazy Fq helpers ------------------------------------------------------
// Products are calls of the one out-of-line product, except where a kernel's
// hot loop asks for them inline.  The reduction's kernels are short chains of
// large point operations: with inlined products they would miss the
// instruction cache (MSM of 2^14 points on B200: 745 us called, 801 us inline).
template <bool INLINE = false>
__device__ __forceinline__ void qmul(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  if constexpr (INLINE)
    mul_lazy<P_q>(r, a, b);
  else
    mul_out<P_q>(r, a, b);
}
template <bool INLINE = false>
__device__ __forceinline__ void qsqr(uint32_t r[8], const uint32_t a[8]) {
  qmul<INLINE>(r, a, a);
}
__device__ __forceinline__ void qadd(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) { add_lazy<P_q>(r, a, b); }
__device__ __forceinline__ void qsub(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) { sub_lazy<P_q>(r, a, b); }
__device__ __forceinline__ void qdbl(uint32_t r[8], const uint32_t a[8]) { add_lazy<P_q>(r, a, a); }
__device__ __forceinline__ bool qzero(const uint32_t a[8]) {
  uint32_t c[8];
  reduce_once<P_q>(c, a);
  return is_zero(c);
}
__device__ __forceinline__ void xyzz_set_inf(xyzz_t& p) {
  set_zero(p.x);
  set_zero(p.y);
  set_zero(p.zz);
  set_zero(p.zzz);
}
__device__ __forceinline__ bool xyzz_is_inf(const xyzz_t& p) { return qzero(p.zz); }
__device__ __forceinline__ bool aff_is_inf(const aff_t& p) { return is_zero(p.x) && is_zero(p.y); }

__device__ __forceinline__ void xyzz_from_aff(xyzz_t& r, const aff_t& q) {
  if (aff_is_inf(q)) {
    xyzz_set_inf(r);
    return;
  }
  cpy(r.x, q.x);
  cpy(r.y, q.y);
  set_one<P_q>(r.zz);
  set_one<P_q>(r.zzz);
}

// r = 2p  (dbl-2008-s-1, a = 0).  The identity doubles to itself (ZZ stays 0).
__device__ __forceinline__ void xyzz_dbl(xyzz_t& r, const xyzz_t& p) {
  uint32_t U[8], V[8], W[8], S[8], M[8], t[8];
  qdbl(U, p.y);
  qsqr(V, U);
  qmul(W, U, V);
  qmul(S, p.x, V);
  qsqr(M, p.x);
  qdbl(t, M);
  qadd(M, M, t);  // M = 3 X^2
  uint32_t X3[8], Y3[8];
  qsqr(X3, M);
  qdbl(t, S);
  qsub(X3, X3, t);
  qsub(t, S, X3);
  qmul(Y3, M, t);
  qmul(t, W, p.y);
  qsub(Y3, Y3, t);
  qmul(r.zz, V, p.zz);
  qmul(r.zzz, W, p.zzz);
  cpy(r.x, X3);
  cpy(r.y, Y3);
}

// r = 2q for an affine q (mdbl-2008-s-1)
__device__ __forceinline__ void xyzz_mdbl(xyzz_t& r, const aff_t& q) {
  if (aff_is_inf(q)) {
    xyzz_set_inf(r);
    return;
  }
  uint32_t U[8], V[8], W[8], S[8], M[8], t[8];
  qdbl(U, q.y);
  qsqr(V, U);
  qmul(W, U, V);
  qmul(S, q.x, V);
  qsqr(M, q.x);
  qdbl(t, M);
  qadd(M, M, t);
  qsqr(r.x, M);
  qdbl(t, S);
  qsub(r.x, r.x, t);
  qsub(t, S, r.x);
  qmul(r.y, M, t);
  qmul(t, W, q.y);
  qsub(r.y, r.y, t);
  cpy(r.zz, V);
  cpy(r.zzz, W);
}

// p += q (affine), madd-2008-s with all special cases
template <bool INLINE = false>
__device__ __forceinline__ void xyzz_madd(xyzz_t& p, const aff_t& q) {
  if (aff_is_inf(q)) return;
  if (xyzz_is_inf(p)) {
    xyzz_from_aff(p, q);
    return;
  }
  uint32_t U2[8], S2[8], P[8], R[8];
  qmul<INLINE>(U2, q.x, p.zz);
  qmul<INLINE>(S2, q.y, p.zzz);
  qsub(P, U2, p.x);
  qsub(R, S2, p.y);
  if (qzero(P)) {
    if (qzero(R))
      xyzz_mdbl(p, q);
    else
      xyzz_set_inf(p);
    return;
  }
  uint32_t PP[8], PPP[8], Q[8], t[8];
  qsqr<INLINE>(PP, P);
  qmul<INLINE>(PPP, P, PP);
  qmul<INLINE>(Q, p.x, PP);
  qsqr<INLINE>(t, R);
  qsub(t, t, PPP);
  uint32_t X3[8];
  qdbl(X3, Q);
  qsub(X3, t, X3);
  qsub(t, Q, X3);
  qmul<INLINE>(t, R, t);
  uint32_t u[8];
  qmul<INLINE>(u, p.y, PPP);
  qsub(p.y, t, u);
  cpy(p.x, X3);
  qmul<INLINE>(p.zz, p.zz, PP);
  qmul<INLINE>(p.zzz, p.zzz, PPP);
}

// p += q (both XYZZ), add-2008-s with all special cases
__device__ __forceinline__ void xyzz_add(xyzz_t& p, const xyzz_t& q) {
  if (xyzz_is_inf(q)) return;
  if (xyzz_is_inf(p)) {
    p = q;
    return;
  }
  uint32_t U1[8], U2[8], S1[8], S2[8], P[8], R[8];
  qmul(U1, p.x, q.zz);
  qmul(U2, q.x, p.zz);
  qmul(S1, p.y, q.zzz);
  qmul(S2, q.y, p.zzz);
  qsub(P, U2, U1);
  qsub(R, S2, S1);
  if (qzero(P)) {
    if (qzero(R))
      xyzz_dbl(p, p);
    else
      xyzz_set_inf(p);
    return;
  }
  uint32_t PP[8], PPP[8], Q[8], t[8], X3[8];
  qsqr(PP, P);
  qmul(PPP, P, PP);
  qmul(Q, U1, PP);
  qsqr(t, R);
  qsub(t, t, PPP);
  qdbl(X3, Q);
  qsub(X3, t, X3);
  qsub(t, Q, X3);
  qmul(t, R, t);
  qmul(S1, S1, PPP);
  qsub(p.y, t, S1);
  cpy(p.x, X3);
  qmul(p.zz, p.zz, q.zz);
  qmul(p.zz, p.zz, PP);
  qmul(p.zzz, p.zzz, q.zzz);
  qmul(p.zzz, p.zzz, PPP);
}

__device__ __forceinline__ void ld_aff(aff_t& q, const fe* p) {
  ld_fe(q.x, p);
  ld_fe(q.y, p + 1);
}
__device__ __forceinline__ void ld_xyzz(xyzz_t& q, const fe* p) {
  ld_fe(q.x, p);
  ld_fe(q.y, p + 1);
  ld_fe(q.zz, p + 2);
  ld_fe(q.zzz, p + 3);
}
__device__ __forceinline__ void st_xyzz(fe* p, const xyzz_t& q) {
  st_fe(p, q.x);
  st_fe(p + 1, q.y);
  st_fe(p + 2, q.zz);
  st_fe(p + 3, q.zzz);
}

}  // namespace zk
