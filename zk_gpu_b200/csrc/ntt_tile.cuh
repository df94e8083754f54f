// ntt_tile.cuh — the device side of one NTT pass (a CTA tile of radix-2^B
// DIF columns with the twist or the final digit-reversed store), shared by
// the per-pass kernels, the persistent batch kernel and their launchers.
//
// The launchers of the passes B = 7..11 live in their own translation unit,
// ntt_pass_wide.cu, which compiles in parallel with ntt.cu.
#pragma once
#include <cuda_runtime.h>

#include "field.cuh"
#include "ntt.cuh"

namespace zk {

using P_r = FrP;

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
// Shared-memory word of element i of column g.  Columns are adjacent, so a
// warp whose lanes hold 32 columns reads and writes 32 consecutive words (and
// reads one twiddle for all lanes).  With fewer columns the lanes differ in
// low bits of the thread's column position q, which are element bits 0.. in
// all rounds but the last and bits 3.. there; the XOR puts both on distinct
// banks.
__device__ __forceinline__ uint32_t word_of(uint32_t i, uint32_t g, uint32_t log_G) {
  return ((i << log_G) + g) ^ (((i >> 3) << log_G) & 31u);
}

template <int LO>
__device__ __forceinline__ uint32_t ins3(uint32_t q, uint32_t r) {
  return (q & ((1u << LO) - 1u)) | (r << LO) | ((q >> LO) << (LO + 3));
}

__device__ __forceinline__ void ld_smem_fe(uint32_t r[8], const uint32_t* plane0, uint32_t plane_stride, uint32_t a) {
#pragma unroll
  for (int k = 0; k < 8; k++) r[k] = plane0[k * plane_stride + a];
}
__device__ __forceinline__ void st_smem_fe(uint32_t* plane0, uint32_t plane_stride, uint32_t a, const uint32_t r[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) plane0[k * plane_stride + a] = r[k];
}

// ---------------------------------------------------------------------------
// Rounds of the passes of up to 2^8 points.
//
// A round runs 8-point DFTs on the elements a thread holds, then multiplies
// output f of the DFT by the round's twiddle w^(f low).  What bounds a pass is
// its field products, so the round is arranged for few and cheap ones:
//  * the DFT takes four products instead of five.  With t_i = x_i - x_(i+4)
//    and w = w_8, the odd outputs need w t_1 + w^3 t_3 and
//    i (w t_1 - w^3 t_3) = w^3 t_1 + w t_3, which are E_1 + E_2 and E_1 - E_2
//    for E_1 = (w + w^3) / 2 (t_1 + t_3), E_2 = (w - w^3) / 2 (t_1 - t_3);
//  * eight twiddle-free stages and seven products by f, low instead of twelve
//    butterflies with a product each: 11 products per 8 elements and 3 bits;
//  * the bits that do not make up a round of three come first, as a radix-2 or
//    radix-4 round (4 or 8 products per 8 elements), so that the last round,
//    which has no twiddles, is always a whole one: B = 7 takes 19 products,
//    with the short round last 22 (2^21 as 7+7+7: 354 -> 338 us, 2^24 as 8+8+8:
//    2674 -> 2586);
//  * every multiplicand is known beforehand, so each product is a mul_w4 over
//    a table in shared memory (about 390 cycles against mul_lazy's 555).
//  * the DFT's three constants are the same for the whole pass: the per-pass
//    kernels take them as kernel parameters in the form of mul_w8 (350 cycles,
//    no loads).
// Forward NTT of 2^24 (8+8+8) on B200: 4320 us with a mul_lazy in each radix-2
// butterfly, 2685 us in this form; the multiply pipe is then busy for 73 % of a
// pass (ncu, sm__pipe_fmaheavy_cycles_active).  Every product is inlined; the
// batch kernel, which holds all pass widths, orders its work by width so that
// the blocks of an SM run the same code (512 transforms of 2^10..2^20: 20.0 ms
// with one product called out of line, 18.0 ms inlined).
//
// Ranges, with 1 for p (1 + 2^-29), the bound of a mul_w4 result: inputs <= 1;
// a difference gets the multiple of p that keeps it positive, and a sum that
// would leave [0, 5.29] (2^256 = 5.29 p) loses 2p first if it is at least 2p.
// ---------------------------------------------------------------------------
constexpr int kNarrowMax = 8;  // widest pass of this form: its tables take 32 KiB of shared memory

// Twiddle table of a pass: I = w_4, (w_8 + w_8^3) / 2, (w_8 - w_8^3) / 2; then
// the short first round's, if there is one (B mod 3 = F bits): the roots
// w_m^(f low), 1 <= f < 2^F, low < 2^(B - F), at [(f - 1) 2^(B - F) + low]; then
// per later round with LO > 0 w_(8 2^LO)^(f low) at [(f - 1) 2^LO + low].
__host__ __device__ constexpr int tw_first(int B) { return ((1 << B % 3) - 1) << (B - B % 3); }
__host__ __device__ constexpr int tw_entries(int B) {
  int n = 3 + tw_first(B);
  for (int lo = B - B % 3 - 3; lo > 0; lo -= 3) n += 7 << lo;
  return n;
}
__host__ __device__ constexpr int tw_offset(int B, int LO) {
  int n = 3 + tw_first(B);
  for (int lo = B - B % 3 - 3; lo > LO; lo -= 3) n += 7 << lo;
  return n;
}

// shared memory of a pass's root table
__host__ __device__ constexpr size_t tw_smem_bytes(int B) {
  return B <= kNarrowMax ? (size_t)tw_entries(B) * 128 : (size_t)16 << B;
}

__device__ __forceinline__ void lds_v4(uint32_t v[4], uint32_t addr) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
struct SmemW4 {  // entry at `addr` of a table stored as eight planes of 16 bytes
  uint32_t addr, plane;
  __device__ __forceinline__ void operator()(int k, uint32_t v[8]) const {
    lds_v4(v, addr + 2 * k * plane);
    lds_v4(v + 4, addr + (2 * k + 1) * plane);
  }
};
// r = a times table entry e
template <int B>
__device__ __forceinline__ void tw_mul(uint32_t r[8], const uint32_t a[8], uint32_t tab, uint32_t e) {
  mul_w4<P_r>(r, a, SmemW4{tab + 16 * e, 16 * tw_entries(B)});
}

struct ParamC8 {
  const DftConsts& d;
  __device__ __forceinline__ void mul(uint32_t r[8], const uint32_t a[8], int e) const {
    const uint32_t* t = d.w[e];
    mul_w8<P_r>(r, a, [t](int k, uint32_t v[8]) {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = t[8 * k + j];
    });
  }
};
template <int B>
struct SmemC4 {
  uint32_t tab;
  __device__ __forceinline__ void mul(uint32_t r[8], const uint32_t a[8], int e) const { tw_mul<B>(r, a, tab, e); }
};
// 8-point DFT in place, position r <- output rev3(r); inputs <= 1, outputs <= 5
template <class C>
__device__ __forceinline__ void dft8(uint32_t x[8][8], const C& c) {
  uint32_t s0[8], s1[8], s2[8], s3[8], u[8], v[8], e[8], f[8];
  // products first: their operands die here
  add_raw(s1, x[1], x[5]);
  add_raw(s3, x[3], x[7]);
  add_raw(u, x[1], x[3]);
  add_raw(e, x[5], x[7]);
  sub_off<P_r, 3>(u, u, e);       // t1 + t3, 1 .. 5
  add_raw(v, x[1], x[7]);
  add_raw(e, x[3], x[5]);
  sub_off<P_r, 3>(v, v, e);       // t1 - t3, 1 .. 5
  c.mul(u, u, 1);        // E1
  c.mul(v, v, 2);        // E2
  sub_off<P_r, 2>(e, x[2], x[6]);
  c.mul(e, e, 0);        // i t2
  add_raw(s0, x[0], x[4]);
  add_raw(s2, x[2], x[6]);
  // odd outputs
  add_raw(x[5], x[4], e);
  sub_off<P_r, 3>(x[7], x[0], x[5]);  // t0 - i t2, 1 .. 4
  cond_sub<P_r, 2>(x[7]);
  sub_off<P_r, 2>(x[0], x[0], x[4]);
  add_raw(x[0], x[0], e);             // t0 + i t2, 1 .. 4
  cond_sub<P_r, 2>(x[0]);
  add_raw(e, u, v);
  sub_off<P_r, 2>(u, u, v);           // E1 - E2 + 2, 1 .. 3
  add_raw(x[4], x[0], e);             // 0 .. 4
  sub_off<P_r, 3>(x[5], x[0], e);     // 1 .. 5
  add_raw(x[6], x[7], u);             // 1 .. 5
  sub_off<P_r, 4>(x[7], x[7], u);     // 1 .. 5: E2 - E1 + 2 added
  // even outputs
  add_raw(e, s0, s2);
  cond_sub<P_r, 2>(e);
  add_raw(f, s1, s3);
  cond_sub<P_r, 2>(f);
  add_raw(x[0], e, f);                // 0 .. 4
  sub_off<P_r, 3>(x[1], e, f);        // 1 .. 5
  sub_off<P_r, 3>(s0, s0, s2);        // 1 .. 5
  cond_sub<P_r, 2>(s0);               // 0 .. 3
  sub_off<P_r, 3>(s1, s1, s3);        // 1 .. 5
  c.mul(s1, s1, 0);
  add_raw(x[2], s0, s1);              // 0 .. 4
  sub_off<P_r, 2>(x[3], s0, s1);      // 1 .. 5
}
// 4-point DFT of a, b, c, d (positions 0..3), position r <- output rev2(r);
// inputs <= 1, outputs <= 5, the first <= 4
template <class C>
__device__ __forceinline__ void dft4(uint32_t x0[8], uint32_t x1[8], uint32_t x2[8], uint32_t x3[8], const C& c) {
  uint32_t s0[8], s1[8], d[8];
  sub_off<P_r, 2>(d, x1, x3);
  c.mul(d, d, 0);
  add_raw(s0, x0, x2);
  add_raw(s1, x1, x3);
  sub_off<P_r, 2>(x0, x0, x2);
  add_raw(x2, x0, d);             // 1 .. 4
  sub_off<P_r, 2>(x3, x0, d);     // 2 .. 5
  add_raw(x0, s0, s1);
  sub_off<P_r, 3>(x1, s0, s1);    // 1 .. 5
}

// The short first round (F = 1 or 2 bits): the thread holds the column's top
// three bits, x[r] at r 2^(B - 3) + q.
template <int B, class C>
__device__ __forceinline__ void short_round(uint32_t x[8][8], uint32_t q, uint32_t tab, const C& c) {
  constexpr int F = B % 3;
  if constexpr (F == 1) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
      uint32_t t[8];
      sub_off<P_r, 2>(t, x[r], x[r + 4]);
      add_raw(x[r], x[r], x[r + 4]);
      cond_sub<P_r, 1>(x[r]);
      tw_mul<B>(x[r + 4], t, tab, 3 + (r << (B - 3)) + q);
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; h++) {  // elements h, h + 2, h + 4, h + 6
      dft4(x[h], x[h + 2], x[h + 4], x[h + 6], c);
      cond_sub<P_r, 2>(x[h]);
      cond_sub<P_r, 1>(x[h]);
      const uint32_t low = (h << (B - 3)) + q;
#pragma unroll
      for (int r = 1; r < 4; r++) {  // position r <- output rev2(r)
        const uint32_t f = (uint32_t)((r & 1) << 1 | r >> 1);
        tw_mul<B>(x[h + 2 * r], x[h + 2 * r], tab, 3 + ((f - 1) << (B - 2)) + low);
      }
    }
  }
}

template <int B, int LO, class C>
__device__ __forceinline__ void narrow_round(uint32_t x[8][8], uint32_t q, uint32_t tab, const C& c) {
  dft8(x, c);
  if constexpr (LO > 0) {
    const uint32_t low = q & ((1u << LO) - 1u);
    cond_sub<P_r, 2>(x[0]);
    cond_sub<P_r, 1>(x[0]);
#pragma unroll
    for (int r = 1; r < 8; r++) {
      const uint32_t f = (uint32_t)((r & 1) << 2 | (r & 2) | r >> 2);
      tw_mul<B>(x[r], x[r], tab, tw_offset(B, LO) + ((f - 1) << LO) + low);
    }
  }
}

// ---------------------------------------------------------------------------
// Rounds of the wider passes (B = 9..11), which only plans asked for by name
// or by the autotuner use: their root tables would not leave room for two
// blocks per SM in the form above.  Radix-2 butterflies on values below 2p,
// each with a Montgomery product by a root w_m^e, e < m / 2.
// ---------------------------------------------------------------------------
// a twiddle: its low and high 16 bytes in two planes
__device__ __forceinline__ void ld_smem_tw(uint32_t r[8], const uint4* plane0, uint32_t plane_stride, uint32_t a) {
  const uint4 x = plane0[a], y = plane0[plane_stride + a];
  r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w;
  r[4] = y.x; r[5] = y.y; r[6] = y.z; r[7] = y.w;
}
// One round: registers hold i(r) = ins3<LO>(q, r); perform the DIF stages
// with butterfly bits HI-1 .. LO.  tws: inner roots w_m^e (e < m/2), 2 planes.
template <int B, int LO, int HI>
__device__ __forceinline__ void ntt_round(uint32_t x[8][8], uint32_t q, const uint4* tws) {
  constexpr uint32_t HALF = 1u << (B - 1);
#pragma unroll
  for (int b = HI - 1; b >= LO; b--) {
    const int rb = b - LO;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      if (r & (1 << rb)) continue;
      const int r2 = r | (1 << rb);
      uint32_t t[8];
      sub_lazy<P_r>(t, x[r], x[r2]);
      add_lazy<P_r>(x[r], x[r], x[r2]);
      if constexpr (LO == 0) {
        // exponent is a compile-time constant: (r mod 2^b) << (B-1-b)
        const uint32_t e = (uint32_t)(r & ((1 << b) - 1)) << (B - 1 - b);
        if (e == 0) {
#pragma unroll
          for (int k = 0; k < 8; k++) x[r2][k] = t[k];
        } else {
          uint32_t w[8];
          ld_smem_tw(w, tws, HALF, e);
          mul_out<P_r>(x[r2], t, w);
        }
      } else {
        const uint32_t e = ((q & ((1u << LO) - 1u)) | ((uint32_t)(r & ((1 << rb) - 1)) << LO)) << (B - 1 - b);
        uint32_t w[8];
        ld_smem_tw(w, tws, HALF, e);
        mul_out<P_r>(x[r2], t, w);
      }
    }
  }
}

// A block runs up to two tiles that share its root table and nothing else, so
// that each waits at its own barriers: with 256 threads at one barrier the
// pass is in the same phase (loads, products, exchange) in half of an SM's
// warps at a time, and its products overlap less with the rest.
struct TilePos {
  uint32_t q, g;  // position in the column, column
  uint32_t log_G;
  uint32_t t, nt;   // thread of the tile, its threads
  uint32_t barrier, barrier_threads;
  bool active;
};
// Barriers 1 and 2; barrier 0 stays with __syncthreads, which one tile's threads
// may already wait at (the batch kernel's end of a work item) while the other's
// still meet here: one barrier must not be met with two thread counts at once.
__device__ __forceinline__ void tile_sync(const TilePos& pos) {
  asm volatile("bar.sync %0, %1;" ::"r"(pos.barrier), "r"(pos.barrier_threads) : "memory");
}

template <int B, int LO_CUR, int LO_NEXT>
__device__ __forceinline__ void ntt_exchange(uint32_t x[8][8], const TilePos& pos, uint32_t* sm,
                                             uint32_t plane_stride) {
  // q is made opaque so that the eight addresses are computed here again and
  // not kept in registers through the round before (spills at 128 registers)
  uint32_t q = pos.q;
  asm volatile("" : "+r"(q));
  if (pos.active) {
#pragma unroll
    for (int r = 0; r < 8; r++) st_smem_fe(sm, plane_stride, word_of(ins3<LO_CUR>(q, r), pos.g, pos.log_G), x[r]);
  }
  tile_sync(pos);
  asm volatile("" : "+r"(q));
  if (pos.active) {
#pragma unroll
    for (int r = 0; r < 8; r++) ld_smem_fe(x[r], sm, plane_stride, word_of(ins3<LO_NEXT>(q, r), pos.g, pos.log_G));
  }
  tile_sync(pos);
}

// The twists of a thread's eight outputs (64 B each) come through four slots
// of the data area, free once the last exchange is over: cp.async fills them
// while the last round computes, and refills each after its product, so the
// products do not wait for the table (measured without: 2.6-3.3 stalled warps
// per issue on it).  A thread reads only what it copied itself.
__device__ __forceinline__ uint32_t twist_index(const PassParams& p, int B, uint32_t q, uint32_t col, int r) {
  return (__brev(8 * q + r) >> (32 - B) << p.log_J) + col;
}
__device__ __forceinline__ void twist_fetch(const PassParams& p, int B, const TilePos& pos, uint32_t col, uint32_t sm,
                                            int r) {
  if (pos.active) {
    const char* src = reinterpret_cast<const char*>(p.twist + 2 * (size_t)twist_index(p, B, pos.q, col, r));
    const uint32_t dst = sm + 16 * (4 * (r & 3) * pos.nt + pos.t);
#pragma unroll
    for (int c = 0; c < 4; c++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * c * pos.nt), "l"(src + 16 * c)
                   : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// The first output index of the last pass's column o, its mixed-radix digits
// reversed: o = k_1 2^(b_2+..) + ... + k_(p-1) gives k_1 + 2^b_1 k_2 + ...;
// total = their bits
__device__ __forceinline__ uint32_t rev_digits(const PassParams& p, uint32_t o, uint32_t& total) {
  uint32_t rev = 0, low_bits = 0;
  total = 0;
#pragma unroll
  for (int t = 0; t < NTT_MAX_PASS; t++)
    if (t < (int)p.nprev) total += p.prev_bits[t];
  uint32_t above = total;
#pragma unroll
  for (int t = 0; t < NTT_MAX_PASS; t++) {
    if (t < (int)p.nprev) {
      above -= p.prev_bits[t];
      const uint32_t digit = o >> above;
      o &= (1u << above) - 1u;
      rev |= digit << low_bits;
      low_bits += p.prev_bits[t];
    }
  }
  return rev;
}
// input element xi of the first pass, scaled by its coset power or, as the
// caller gave it (taken up to 2p), below p
__device__ __forceinline__ void prepare_first(const PassParams& p, uint32_t x[8], uint32_t xi) {
  if (p.pre_lo) {
    uint32_t a[8], b[8];
    ld_fe_nc(a, p.pre_lo + (xi & ((1u << p.pre_shift) - 1u)));
    ld_fe_nc(b, p.pre_hi + (xi >> p.pre_shift));
    mul_out<P_r>(a, a, b);
    mul_out<P_r>(x, a, x);  // < 3p for any input
    cond_sub<P_r, 2>(x);
  }
  cond_sub<P_r, 1>(x);
}
// output kout, scaled and made canonical; WIDE_RANGE: x is below 5p, else 2p.
// The batch kernel has the product by the output scale inline and tabulated
// (post; 512 jobs 17870 -> 17660 us); the pass kernels call it, as inline it
// takes registers from the rest of the pass (2^24 without any scaling: 2670 us
// against 2576).
template <bool WIDE_RANGE, bool BATCH>
__device__ __forceinline__ void store_final(const PassParams& p, const fe* post, const uint32_t x[8], uint32_t kout) {
  uint32_t v[8];
  if (p.post_lo) {
    if (kout >= p.out_count) return;
    uint32_t a[8], b[8];
    ld_fe_nc(a, p.post_lo + (kout & ((1u << p.post_shift) - 1u)));
    ld_fe_nc(b, p.post_hi + (kout >> p.post_shift));
    mul_out<P_r>(a, a, b);
    mul_out<P_r>(v, a, x);  // < 3p
    cond_sub<P_r, 2>(v);
  } else if (p.has_post && BATCH) {
    mul_w2<P_r>(v, x, post[0].w, post[1].w);
  } else if (p.has_post) {
    mul_out<P_r>(v, p.post.w, x);  // < 2p
  } else {
    cpy(v, x);
    if (WIDE_RANGE) {
      cond_sub<P_r, 4>(v);
      cond_sub<P_r, 2>(v);
    }
  }
  cond_sub<P_r, 1>(v);
  st_fe(p.out + kout, v);
}

// Rounds from index bit HI down.  Narrow passes: a short round if HI = B is no
// multiple of three, then rounds of three bits; wide ones: rounds of three bits
// from the top, the last taking what is left.
template <int B, int HI, bool BATCH>
__device__ __forceinline__ void ntt_rounds(const PassParams& p, const DftConsts* dft, uint32_t x[8][8],
                                           TilePos pos, uint32_t col,
                                           uint32_t* sm, uint32_t plane_stride, const uint4* tws) {
  constexpr bool NARROW = B <= kNarrowMax, SHORT = NARROW && HI % 3 != 0;
  constexpr int LO = SHORT ? B - B % 3 : HI - 3 > 0 ? HI - 3 : 0;  // lowest bit of this round
  constexpr int MAP = SHORT ? B - 3 : LO;                          // lowest bit the thread holds
  if constexpr (LO == 0) {
    if (!p.is_final) {
#pragma unroll
      for (int r = 0; r < 4; r++) twist_fetch(p, B, pos, col, (uint32_t)__cvta_generic_to_shared(sm), r);
    }
  }
  if constexpr (NARROW) {
    const uint32_t tab = (uint32_t)__cvta_generic_to_shared(tws);
    auto round = [&](const auto& c) {
      if constexpr (SHORT)
        short_round<B>(x, pos.q, tab, c);
      else
        narrow_round<B, LO>(x, pos.q, tab, c);
    };
    if constexpr (BATCH)
      round(SmemC4<B>{tab});
    else
      round(ParamC8{*dft});
  } else {
    ntt_round<B, LO, HI>(x, pos.q, tws);
  }
  if constexpr (LO > 0) {
    constexpr int LO_N = LO - 3 > 0 ? LO - 3 : 0;
    ntt_exchange<B, MAP, LO_N>(x, pos, sm, plane_stride);
    // what follows depends on the thread's position through this copy: the
    // addresses of later phases are not computed ahead and kept (spills)
    asm volatile("" : "+r"(pos.q), "+r"(col));
    ntt_rounds<B, LO, BATCH>(p, dft, x, pos, col, sm, plane_stride, tws);
  }
}

template <int B, bool BATCH>
__device__ __forceinline__ void ntt_pass_tile(const PassParams& p, const DftConsts* dft, const fe* post, uint64_t tile,
                                              uint32_t* smem, bool have_roots = false) {
  constexpr uint32_t M = 1u << B;
  constexpr uint32_t T = M / 8;  // threads per column
  const uint32_t G = p.G;
  const uint32_t plane_stride = G * M;
  uint4* tws = reinterpret_cast<uint4*>(smem + 8 * plane_stride * p.ntile);  // 32 G M bytes per tile in

  const uint32_t tid = threadIdx.x;
  const uint32_t log_G = __ffs(G) - 1, log_nt = log_G + (B - 3);
  const uint32_t sub = p.ntile > 1 ? tid >> log_nt : 0u;
  const uint32_t t = tid - (sub << log_nt);
  const uint32_t g = t & (G - 1), q = t >> log_G;
  const bool active = !BATCH || (sub < p.ntile && q < T);
  const TilePos pos{q, g, log_G, t, G * T, 1 + sub, p.ntile > 1 ? G * T : (blockDim.x + 31u) & ~31u, active};

  if constexpr (B <= kNarrowMax) {
    constexpr uint32_t N = tw_entries(B);
    const uint4* src = reinterpret_cast<const uint4*>(p.inner);
    if (!have_roots)
      for (uint32_t e = tid; e < 8 * N; e += blockDim.x) tws[(e & 7) * N + (e >> 3)] = __ldg(src + e);
  } else {
    for (uint32_t e = tid; e < M / 2; e += blockDim.x) {
      uint32_t w[8];
      ld_fe_nc(w, p.inner + e);
      tws[e] = make_uint4(w[0], w[1], w[2], w[3]);
      tws[M / 2 + e] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }

  // element indices are < 2^28: 32-bit arithmetic, powers of two as shifts
  const uint32_t t32 = (uint32_t)tile * p.ntile + sub;
  smem += 8 * plane_stride * sub;
  const uint32_t J = 1u << p.log_J;
  uint32_t o, col = 0, base, stride;
  if (!p.is_final) {
    const uint32_t log_cpo = p.log_J - log_G;  // columns per outer block = J / G
    o = t32 >> log_cpo;
    col = ((t32 & ((1u << log_cpo) - 1u)) << log_G) + g;
    base = ((o << B) << p.log_J) + col;
    stride = J;
  } else {
    const uint32_t log_rest = p.log_O - p.log_m1;  // rest_count = O / m_1
    const uint32_t rest = t32 & ((1u << log_rest) - 1u);
    const uint32_t k1 = ((t32 >> log_rest) << log_G) + g;
    o = (k1 << log_rest) + rest;
    base = o << B;
    stride = 1;
  }

  uint32_t x[8][8];
  if (active) {
    const uint32_t rows = p.in_rows ? p.in_rows : M;  // rows past in_rows are zero padding
#pragma unroll
    for (int r = 0; r < 8; r++) {
      if (q + T * r >= rows)
        set_zero(x[r]);
      else if (BATCH)
        ld_fe_cg(x[r], p.in + (base + (q + T * r) * stride));
      else
        ld_fe(x[r], p.in + (base + (q + T * r) * stride));
    }
  } else {
#pragma unroll
    for (int r = 0; r < 8; r++) set_zero(x[r]);
  }

  if (p.is_first && active) {
#pragma unroll
    for (int r = 0; r < 8; r++) prepare_first(p, x[r], base + (q + T * r) * stride);
  }
  __syncthreads();

  ntt_rounds<B, B, BATCH>(p, dft, x, pos, col, smem, plane_stride, tws);
  if (!active) return;

  // element r now holds output k = bitrev_B(8q + r)
  if (!p.is_final) {
    const uint32_t sm = (uint32_t)__cvta_generic_to_shared(smem);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      asm volatile("cp.async.wait_group 3;" ::: "memory");
      uint32_t v[8], w[8];
      const uint32_t slot = sm + 16 * (4 * (r & 3) * pos.nt + t);
      lds_v4(v, slot);
      lds_v4(v + 4, slot + 16 * pos.nt);
      lds_v4(w, slot + 32 * pos.nt);
      lds_v4(w + 4, slot + 48 * pos.nt);
      mul_w2<P_r>(x[r], x[r], v, w);
      if (r < 4)
        twist_fetch(p, B, pos, col, sm, r + 4);
      else
        asm volatile("cp.async.commit_group;" ::: "memory");
      st_fe(p.out + ((o << B << p.log_J) + twist_index(p, B, q, col, r)), x[r]);
    }
  } else {
    uint32_t total;
    const uint32_t rev = rev_digits(p, o, total);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const uint32_t k = __brev(8 * q + r) >> (32 - B);
      store_final<(B <= kNarrowMax), BATCH>(p, post, x[r], rev + (k << total));
    }
  }
}

template <int B>
__global__ void __launch_bounds__(256, 2) ntt_pass_kernel(const PassParams p, const DftParam<B> dft) {
  extern __shared__ __align__(16) uint32_t smem[];
  ntt_pass_tile<B, false>(p, &dft.c, nullptr, blockIdx.x, smem);
}

// ---------------------------------------------------------------------------
// Passes of small transforms.  A tile's thread runs the products of its eight
// elements one after the other (some 20 per pass, 0.3 us each when the SM has
// nothing else), and a small transform leaves most SMs without a tile.  Here a
// thread holds two elements: a radix-2 stage costs it one product, stages
// exchange one element between the lanes of a warp by shuffles (between warps
// through shared memory where a column has more than 64 elements), and the
// next stage's root is loaded while the product runs.  That is as much work in
// all (B - 1 products per two elements) on four times the threads, with
// 4 to 7 us per pass (2^10, 2^13) instead of 9 to 17.  Roots: w_m^e, e < m / 2, after the
// entries of the tile kernel's rounds.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int roots_entries(int B) { return tw_entries(B) + (1 << (B - 1)); }

struct W4Regs {
  uint32_t w[4][8];
  __device__ __forceinline__ void load(const fe* entry) {
#pragma unroll
    for (int k = 0; k < 4; k++) ld_fe_nc(w[k], entry + k);
  }
  __device__ __forceinline__ void operator()(int k, uint32_t v[8]) const { cpy(v, w[k]); }
};

// stages b .. 0 of a column: thread q of 2^(B - 1) holds the elements whose
// index has bit b clear and set and its other bits from q
template <int B, int b>
__device__ __forceinline__ void pair_stages(uint32_t x0[8], uint32_t x1[8], uint32_t q, const fe* roots,
                                            const W4Regs& w, uint32_t* sm, unsigned mask) {
  uint32_t d[8];
  sub_off<P_r, 2>(d, x0, x1);
  add_raw(x0, x0, x1);
  if constexpr (b == 0) {
    cpy(x1, d);  // <= 2 and <= 3
  } else {
    W4Regs next;
    if constexpr (b > 1) next.load(roots + 4 * ((q & ((1u << (b - 1)) - 1u)) << (B - b)));
    cond_sub<P_r, 1>(x0);
    mul_w4<P_r>(x1, d, w);
    // the lane whose bit b - 1 is clear keeps x0 and gets the other's x0
    const bool up = (q >> (b - 1)) & 1u;
    uint32_t s[8];
#pragma unroll
    for (int k = 0; k < 8; k++) s[k] = up ? x0[k] : x1[k];
    if constexpr (b - 1 < 5) {
#pragma unroll
      for (int k = 0; k < 8; k++) s[k] = __shfl_xor_sync(mask, s[k], 1 << (b - 1));
    } else {
      constexpr uint32_t T = 1u << (B - 1);
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 8; k++) sm[k * T + q] = s[k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 8; k++) s[k] = sm[k * T + (q ^ (1u << (b - 1)))];
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      x0[k] = up ? s[k] : x0[k];
      x1[k] = up ? x1[k] : s[k];
    }
    pair_stages<B, b - 1>(x0, x1, q, roots, next, sm, mask);
  }
}

// One column per 2^(B - 1) threads; a block of more than 32 threads is one column.
template <int B>
__global__ void __launch_bounds__(B > 6 ? 1 << (B - 1) : 32) ntt_pair_kernel(const PassParams p) {
  constexpr uint32_t T = 1u << (B - 1), M = 1u << B;
  __shared__ uint32_t sm[B > 6 ? 8 * T : 1];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t c = t >> (B - 1), q = t & (T - 1);
  const unsigned mask = blockDim.x < 32 ? (1u << blockDim.x) - 1u : 0xffffffffu;
  uint32_t o = c, col = 0, base = c << B, stride = 1;
  if (!p.is_final) {
    o = c >> p.log_J;
    col = c & ((1u << p.log_J) - 1u);
    base = (o << B << p.log_J) + col;
    stride = 1u << p.log_J;
  }
  const fe* roots = p.inner + 4 * tw_entries(B);
  W4Regs w;
  w.load(roots + 4 * q);
  uint32_t x0[8], x1[8];
  const uint32_t rows = p.in_rows ? p.in_rows : M;
  set_zero(x0);
  set_zero(x1);
  if (q < rows) ld_fe(x0, p.in + (base + q * stride));
  if (q + T < rows) ld_fe(x1, p.in + (base + (q + T) * stride));
  if (p.is_first) {
    prepare_first(p, x0, base + q * stride);
    prepare_first(p, x1, base + (q + T) * stride);
  }
  // where the outputs go: positions 2 q and 2 q + 1 hold outputs bitrev
  const uint32_t k0 = __brev(2 * q) >> (32 - B), k1 = k0 + M / 2;
  uint32_t v[2][2][8];
  if (!p.is_final) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const fe* tw = p.twist + 2 * (size_t)(((h ? k1 : k0) << p.log_J) + col);
      ld_fe_nc(v[h][0], tw);
      ld_fe_nc(v[h][1], tw + 1);
    }
  }
  pair_stages<B, B - 1>(x0, x1, q, roots, w, sm, mask);
  if (!p.is_final) {
    mul_w2<P_r>(x0, x0, v[0][0], v[0][1]);
    mul_w2<P_r>(x1, x1, v[1][0], v[1][1]);
    fe* out = p.out + (o << B << p.log_J) + col;
    st_fe(out + (k0 << p.log_J), x0);
    st_fe(out + (k1 << p.log_J), x1);
  } else {
    uint32_t total;
    const uint32_t rev = rev_digits(p, o, total);
    store_final<true, false>(p, nullptr, x0, rev + (k0 << total));
    store_final<true, false>(p, nullptr, x1, rev + (k1 << total));
  }
}
template <int B>
inline cudaError_t launch_pair(const PassParams& pp, int log_n, cudaStream_t s) {
  const unsigned threads = 1u << (log_n - 1);
  const unsigned block = threads < 32 ? threads : (B > 6 ? 1u << (B - 1) : 32u);
  ntt_pair_kernel<B><<<threads / block, block, 0, s>>>(pp);
  return cudaGetLastError();
}

template <int B>
inline cudaError_t launch_pass(const PassParams& pp, const DftConsts& dft, uint64_t ncta, cudaStream_t s) {
  constexpr uint32_t M = 1u << B;
  const uint32_t threads = pp.ntile * pp.G * (M / 8);
  const size_t smem = (size_t)8 * pp.ntile * pp.G * M * 4 + tw_smem_bytes(B);
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaFuncSetAttribute(ntt_pass_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    attr_set[dev & 63] = true;
  }
  ntt_pass_kernel<B><<<(unsigned)ncta, threads, smem, s>>>(pp, DftParam<B>{{}, dft});
  return cudaGetLastError();
}

// B = 7..11 (ntt_pass_wide.cu)
cudaError_t launch_pass_wide(int B, const PassParams& pp, const DftConsts& dft, uint64_t ncta, cudaStream_t s);

}  // namespace zk
