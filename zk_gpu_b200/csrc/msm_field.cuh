// msm_field.cuh — Fq inversion in Montgomery form for the MSM kernels.
#pragma once
#include "curve.cuh"
#include "fq_inv.cuh"

namespace zk {

// a^-1 for a != 0 in Montgomery form, lazy in, canonical out: the divstep
// inversion (fq_inv.cuh) of the representative a 2^256 gives a^-1 2^-256,
// and one product with 2^768 mod q returns it to Montgomery form.
__device__ __forceinline__ void fq_inv_mont(uint32_t r[8], const uint32_t a[8]) {
  const uint32_t k768[8] = {0xda1530dfu, 0xb1cd6dafu, 0xa7283db6u, 0x62f210e6u, 0x0ada0afbu, 0xef7f0b0cu, 0x2d592544u, 0x20fd6e90u};
  uint32_t c[8], t[8];
  reduce_once<FqP>(c, a);
  fq_inv_divsteps(t, c);
  qmul(r, t, k768);
  reduce_once<FqP>(r, r);
}

}  // namespace zk
