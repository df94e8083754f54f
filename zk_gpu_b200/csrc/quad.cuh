// quad.cuh — XYZZ additions and doublings by four lanes at once.
//
// The bucket reduction is short of points, not of lanes: its kernels run
// chains of dependent point operations, and one lane needs 14 dependent
// products (about 7 us on B200) for an addition.  Here the four lanes of a
// quad hold the coordinates (X, Y, ZZ, ZZZ) of a point, one each, and run the
// products of add-2008-s in four steps and those of dbl-2008-s-1 in three,
// exchanging operands by shuffles: 2.2 us for an addition.  A point in memory
// (four elements in that order) is one 128-B line of which each lane loads its
// own element.
//
// All four lanes of a quad call these functions together and agree on every
// branch; different quads of a warp may diverge.  Values are lazily reduced
// (< 2q), the identity is ZZ = 0, as in curve.cuh.
#pragma once
#include "curve.cuh"

namespace zk {

struct Quad {
  uint32_t j;     // coordinate held by this lane
  unsigned mask;  // lanes of the quad
  __device__ __forceinline__ Quad() {
    const uint32_t lane = threadIdx.x & 31u;
    j = lane & 3u;
    mask = 0xfu << (lane & ~3u);
  }
  // a of the quad's lane `src`
  __device__ __forceinline__ void from(uint32_t r[8], const uint32_t a[8], uint32_t src) const {
#pragma unroll
    for (int k = 0; k < 8; k++) r[k] = __shfl_sync(mask, a[k], (int)src, 4);
  }
  __device__ __forceinline__ bool flag(bool f, uint32_t src) const {
    return __shfl_sync(mask, f ? 1 : 0, (int)src, 4) != 0;
  }
};
__device__ __forceinline__ void sel(uint32_t r[8], bool c, const uint32_t a[8], const uint32_t b[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) r[k] = c ? a[k] : b[k];
}

// p = 2 p (the identity stays: ZZ = 0)
__device__ __forceinline__ void quad_dbl(const Quad& z, uint32_t p[8]) {
  uint32_t a[8], b[8], m[8], u[8], v[8], s[8], t[8];
  qdbl(t, p);                 // lane 1: U = 2 Y
  sel(a, z.j == 1, t, p);
  qmul(m, a, a);              // lane 0: X^2, lane 1: V = U^2
  z.from(u, t, 1);
  z.from(v, m, 1);
  z.from(s, p, 0);            // X
  qdbl(t, m);
  qadd(t, t, m);              // lane 0: M = 3 X^2
  sel(a, z.j == 0, t, v);
  sel(b, z.j == 1, u, p);     // lane 1: W = V U, lane 2: V ZZ
  sel(b, z.j == 3, s, b);     // lane 3: S = V X
  sel(b, z.j == 0, t, b);     // lane 0: M^2
  qmul(m, a, b);
  z.from(s, m, 3);
  z.from(v, m, 1);            // W
  uint32_t x3[8];
  qdbl(u, s);
  qsub(x3, m, u);             // lane 0: X3 = M^2 - 2 S
  qsub(u, s, x3);
  sel(a, z.j == 0, t, v);     // lane 0: M (S - X3), lane 1: W Y, lane 3: W ZZZ
  sel(b, z.j == 0, u, p);
  qmul(t, a, b);
  z.from(u, t, 0);
  qsub(u, u, t);              // lane 1: Y3
  sel(p, z.j == 0, x3, u);
  sel(p, z.j == 2, m, p);
  sel(p, z.j == 3, t, p);
}

// p += q
__device__ __forceinline__ void quad_add(const Quad& z, uint32_t p[8], const uint32_t q[8]) {
  // an identity's ZZ is the zero it was set to: products keep it (0 x = 0)
  if (z.flag(is_zero(q), 2)) return;
  if (z.flag(is_zero(p), 2)) {
    cpy(p, q);
    return;
  }
  uint32_t a[8], b[8], m1[8], m2[8], m3[8], d[8];
  const bool low = z.j < 2;
  z.from(b, q, z.j ^ 2u);
  qmul(m1, p, b);             // U1, S1, U2, S2
  z.from(b, m1, z.j ^ 2u);
  sel(a, low, b, m1);
  sel(b, low, m1, b);
  qsub(d, a, b);              // lanes 0, 2: P = U2 - U1, lanes 1, 3: R = S2 - S1
  const bool zero = qzero(d);
  if (z.flag(zero, 0)) {
    if (z.flag(zero, 1))
      quad_dbl(z, p);
    else
      set_zero(p);
    return;
  }
  sel(a, low, d, p);
  sel(b, low, d, q);
  qmul(m2, a, b);             // P^2, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
  z.from(b, m2, 0);
  z.from(a, d, 0);
  sel(a, z.j == 0, m1, a);
  sel(a, z.j == 2, m2, a);
  qmul(m3, a, b);             // Q = U1 P^2, P^3, ZZ3, P^3
  uint32_t x3[8], t[8];
  z.from(t, m3, 0);
  qsub(x3, m2, m3);
  qdbl(a, t);
  qsub(x3, x3, a);            // lane 1: X3 = R^2 - P^3 - 2 Q
  qsub(t, t, x3);
  z.from(a, m1, 1);           // S1
  z.from(b, m3, 1);           // P^3
  sel(a, z.j == 1, d, a);
  sel(b, z.j == 1, t, b);     // lane 0: S1 P^3, lane 1: R (Q - X3)
  sel(a, z.j == 3, m2, a);    // lane 3: ZZZ3
  qmul(m1, a, b);
  z.from(t, m1, 0);
  z.from(a, x3, 1);
  qsub(t, m1, t);             // lane 1: Y3
  sel(p, z.j == 0, a, t);
  sel(p, z.j == 2, m3, p);
  sel(p, z.j == 3, m1, p);
}

}  // namespace zk
