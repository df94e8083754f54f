// ntt.cu — Fr NTT pass kernels and host orchestration (see ntt.cuh).
//
// Per pass, one CTA owns G columns of one outer block (or, in the last pass,
// G groups whose outputs are adjacent).  Each thread holds 8 elements of one
// column and runs the m-point DIF DFT as "rounds" (ntt_tile.cuh): a round
// covers three index bits [lo, lo+3) that the thread holds in registers.
// Between rounds the columns are exchanged through shared memory, stored as
// 8 u32 planes.  Values stay below 2^256 between rounds (lazy reduction) and
// are made canonical on the final store.
#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "ntt.cuh"
#include "ntt_tile.cuh"
#include "prof.cuh"
#include "runtime.cuh"

namespace zk {

static fe to_fe(const host::Fr& a) {
  fe r;
  std::memcpy(r.w, a.v, 32);
  return r;
}

NttPlan make_ntt_plan(int log_n) {
  NttPlan p;
  p.log_n = log_n;
  if (log_n <= 2) {  // direct DFT kernel
    p.npass = 0;
    return p;
  }
  // Balanced passes of at most kNarrowMax bits; from 2^25, where four are
  // needed, passes of 6 bits (the fewest products per bit) with what is left
  // over in the last pass, which has no twists, and then the first: 2^26 as
  // 6+6+6+8 takes 10.7 ms, as 7+7+6+6 12.2 ms (B200).
  const int np = (log_n + kNarrowMax - 1) / kNarrowMax;
  p.npass = np;
  if (np == NTT_MAX_PASS) {
    const int last = std::min(log_n - 18, kNarrowMax);
    p.bits[0] = log_n - 12 - last;
    p.bits[1] = p.bits[2] = 6;
    p.bits[3] = last;
    return p;
  }
  // Three passes as 6, 7 or 8, 8 bits where that adds up: a pass of 7 takes a
  // short round of one bit first and is the slowest per bit, and the last pass,
  // which has no twists, is the cheapest place for 8.  Against balanced widths
  // (B200, us): 2^21 327.6 / 329.2 (7+7+7), 2^22 619.4 / 660.0 (8+7+7).  Left
  // balanced: 2^17 and 2^18, where that is fastest; 2^19, 94.6 at best against
  // 96.6; 2^20, 185.0 as 6+6+8 against 197.1, whose plan of 7+7+6 the tuner's
  // test knows as the built-in one, as it does 8+8+8 for 2^24 (2557, 2519 as
  // 6+6+6+6); 2^23, 1262 as 6+6+6+5 against 1291.
  const int middle = log_n - 6 - kNarrowMax;
  if (np == 3 && middle >= 7 && middle <= kNarrowMax) {
    p.bits[0] = 6;
    p.bits[1] = middle;
    p.bits[2] = kNarrowMax;
    return p;
  }
  const int base = log_n / np, extra = log_n % np;
  for (int t = 0; t < np; t++) p.bits[t] = base + (t < extra ? 1 : 0);
  return p;
}


// ---------------------------------------------------------------------------
// persistent batch kernel: the passes of many transforms in one launch
// ---------------------------------------------------------------------------
// Work items are CTA tiles ordered by pass level (every first pass before any
// second pass, ...).  A CTA takes the next item with one atomic; before a
// tile of pass t it waits for all tiles of pass t-1 of the same transform.
// Those were handed out earlier to CTAs that are already running and never
// wait on later items, so the waits always end; each is still bounded by a
// clock budget after which the kernel records an error and stops.
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

//
// A block takes its next item while it still works on the current one, so the
// atomic's latency is hidden; it waits for nothing but items before its own,
// so the argument above holds with it (the first unfinished item is always
// one being worked on).  Warp 0 finds the item's pass by a 32-way search (two
// or three dependent loads among the passes of 512 transforms; a binary search
// by one thread took eleven), and the roots stay in shared memory while items
// of the same pass width and table follow one another.
__global__ void __launch_bounds__(256, 2) ntt_batch_kernel(const BatchPass* passes, uint32_t npass,
                                                          uint32_t total_tiles, uint32_t* next, uint32_t* done,
                                                          uint32_t* err, uint64_t spin_cycles) {
  extern __shared__ __align__(16) uint32_t smem[];
  __shared__ uint32_t s_w, s_k, s_stop;
  uint32_t taken = 0;  // thread 0: the item taken ahead
  if (threadIdx.x == 0) taken = atomicAdd(next, 1u);
  const fe* roots = nullptr;  // table in shared memory, its pass width and place
  uint32_t roots_b = 0, roots_at = 0;
  for (;;) {
    if (threadIdx.x < 32) {
      const uint32_t w = __shfl_sync(0xffffffffu, taken, 0);
      uint32_t lo = 0;
      if (w < total_tiles) {
        // last pass whose first tile index is <= w
        uint32_t n = npass;  // it is among [lo, lo + n)
        while (n > 1) {
          const uint32_t step = (n + 31) / 32, at = lo + threadIdx.x * step;
          const bool le = threadIdx.x * step < n && passes[at].tile_base <= w;
          const uint32_t k = 31 - __clz(__ballot_sync(0xffffffffu, le));  // lane 0 always holds
          n = min(step, n - k * step);
          lo += k * step;
        }
      }
      if (threadIdx.x == 0) {
        s_stop = (w >= total_tiles || ld_acquire_u32(err) != 0) ? 1u : 0u;
        if (!s_stop) {
          const BatchPass& bp = passes[lo];
          if (bp.dep != 0xffffffffu) {
            const uint64_t t0 = clock64();
            while (ld_acquire_u32(done + bp.dep) < bp.dep_tiles) {
              if (clock64() - t0 > spin_cycles) {
                atomicExch(err, 1u);
                s_stop = 1;
                break;
              }
              __nanosleep(64);
            }
          }
          s_w = w;
          s_k = lo;
        }
      }
    }
    __syncthreads();
    if (s_stop) return;
    if (threadIdx.x == 0) taken = atomicAdd(next, 1u);
    const BatchPass& bp = passes[s_k];
    const uint64_t tile = s_w - bp.tile_base;
    const uint32_t at = bp.p.ntile * bp.p.G;
    const bool have = bp.p.inner == roots && bp.B == roots_b && at == roots_at;
    roots = bp.p.inner;
    roots_b = bp.B;
    roots_at = at;
    switch (bp.B) {
      case 3: ntt_pass_tile<3, true>(bp.p, nullptr, bp.post, tile, smem, have); break;
      case 4: ntt_pass_tile<4, true>(bp.p, nullptr, bp.post, tile, smem, have); break;
      case 5: ntt_pass_tile<5, true>(bp.p, nullptr, bp.post, tile, smem, have); break;
      case 6: ntt_pass_tile<6, true>(bp.p, nullptr, bp.post, tile, smem, have); break;
      case 7: ntt_pass_tile<7, true>(bp.p, nullptr, bp.post, tile, smem, have); break;
      case 8: ntt_pass_tile<8, true>(bp.p, nullptr, bp.post, tile, smem, have); break;
      case 9: ntt_pass_tile<9, true>(bp.p, nullptr, bp.post, tile, smem); break;
      case 10: ntt_pass_tile<10, true>(bp.p, nullptr, bp.post, tile, smem); break;
      case 11: ntt_pass_tile<11, true>(bp.p, nullptr, bp.post, tile, smem); break;
      default: break;
    }
    __threadfence();  // every thread publishes its own stores before the tile is counted
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(done + s_k, 1u);
    }
  }
}

// Tiny transforms (n <= 4): direct DFT, one thread per output.
__global__ void ntt_tiny_kernel(fe* a, uint32_t log_n, fe w, const fe* pre_lo, const fe* pre_hi, uint32_t pre_shift,
                                uint32_t has_post, fe post) {
  const uint32_t n = 1u << log_n;
  const uint32_t k = threadIdx.x;
  uint32_t in[4][8];
  for (uint32_t i = 0; i < n; i++) {
    ld_fe(in[i], a + i);
    if (pre_lo) {
      uint32_t c0[8], c1[8];
      ld_fe_nc(c0, pre_lo + (i & ((1u << pre_shift) - 1)));
      ld_fe_nc(c1, pre_hi + (i >> pre_shift));
      mul_lazy<P_r>(c0, c0, c1);
      mul<P_r>(in[i], in[i], c0);
    }
  }
  uint32_t acc[8];
  if (k < n) {
    uint32_t wk[8], wik[8];
    pow_u64<P_r>(wk, w.w, k);
    set_zero(acc);
    set_one<P_r>(wik);
    for (uint32_t i = 0; i < n; i++) {
      uint32_t t[8];
      mul<P_r>(t, in[i], wik);
      add<P_r>(acc, acc, t);
      mul<P_r>(wik, wik, wk);
    }
    if (has_post) {
      mul<P_r>(acc, acc, post.w);
    }
  }
  __syncthreads();
  if (k < n) st_fe(a + k, acc);
}

// out[e] = base^(e) for e < count (per-thread square-and-multiply)
__global__ void pow_seq_kernel(fe* out, fe base, uint64_t count, uint64_t step) {
  const uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (e >= count) return;
  uint32_t r[8];
  pow_u64<P_r>(r, base.w, e * step);
  st_fe(out + e, r);
}

// 2^e mod r for the table forms of mul_w4 (2^(64 k + 96)) and mul_w2
// (2^(128 k + 160)): the product of a Montgomery w 2^256 with it is w 2^e
struct TableScale {
  fe w4[4], w2[2];
};
static TableScale table_scale() {
  static const TableScale s = {{to_fe(host::pow2(96)), to_fe(host::pow2(160)), to_fe(host::pow2(224)), to_fe(host::pow2(288))},
                               {to_fe(host::pow2(160)), to_fe(host::pow2(288))}};
  return s;
}

// Roots of a narrow pass: entry e, form k (layout in ntt_tile.cuh); special:
// the three constants of the 8-point DFT
struct Special {
  fe v[3];
};
__global__ void roots_w4_kernel(fe* out, fe wm, const Special special, const TableScale sc, int B) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const int e = (int)(i >> 2);
  if (e >= roots_entries(B)) return;
  uint32_t v[8];
  if (e < 3) {
    cpy(v, special.v[e].w);
  } else if (e >= tw_entries(B)) {
    pow_u64<P_r>(v, wm.w, (uint64_t)(e - tw_entries(B)));
  } else {
    // the round's lowest bit, its first entry, and log2 of its size below m
    int lo = B - B % 3, at = 3, up = 0;
    if (e < at + tw_first(B)) {
      up = 0;
    } else {
      at += tw_first(B);
      lo -= 3;
      while (e >= at + (7 << lo)) at += 7 << lo, lo -= 3;
      up = B - 3 - lo;
    }
    const uint32_t f = (uint32_t)((e - at) >> lo) + 1, low = (uint32_t)(e - at) & ((1u << lo) - 1u);
    pow_u64<P_r>(v, wm.w, (uint64_t)(f * low) << up);
  }
  mul<P_r>(v, v, sc.w4[i & 3].w);
  st_fe(out + i, v);
}

// twist[k * J + j] = lo[(k j) & mask] * hi[(k j) >> shift], both forms of mul_w2
__global__ void twist_table_kernel(fe* out, const fe* lo, const fe* hi, uint32_t shift, uint32_t log_J, uint64_t total,
                                   const TableScale sc) {
  const uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const uint64_t k = idx >> log_J, j = idx & ((1ull << log_J) - 1);
  const uint64_t e = k * j;
  uint32_t a[8], b[8];
  ld_fe_nc(a, lo + (e & ((1ull << shift) - 1)));
  ld_fe_nc(b, hi + (e >> shift));
  mul_lazy<P_r>(a, a, b);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    mul<P_r>(b, a, sc.w2[k].w);
    st_fe(out + 2 * idx + k, b);
  }
}

// dst[i * dst_stride] = src[i] * c^i (powc may be null: plain strided copy)
__global__ void scale_copy_kernel(fe* dst, const fe* src, uint64_t n, uint64_t dst_stride, const fe* lo, const fe* hi,
                                  uint32_t shift) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t v[8];
  ld_fe(v, src + i);
  if (lo) {
    uint32_t a[8], b[8];
    ld_fe_nc(a, lo + (i & ((1ull << shift) - 1)));
    ld_fe_nc(b, hi + (i >> shift));
    mul_lazy<P_r>(a, a, b);
    mul<P_r>(v, v, a);
  }
  st_fe(dst + i * dst_stride, v);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// Both power tables in one launch: entry e of lo is scale base^e, of hi
// base^(e 2^shift), as products of the host's base^(2^k) by the bits of e
// (without squarings, which would double the chain of dependent products).
struct PowArgs {
  fe pw[NTT_MAX_LOG];  // base^(2^k), Montgomery form
  fe scale;
  uint32_t has_scale, shift, nlo, nhi;
};
__global__ void pow_tables_kernel(fe* lo, fe* hi, const PowArgs a) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nlo + a.nhi) return;
  const bool low = i < a.nlo;
  const uint32_t e = low ? i : i - a.nlo;
  uint32_t v[8];
  if (low && a.has_scale)
    cpy(v, a.scale.w);
  else
    set_one<P_r>(v);
  for (uint32_t k = 0, b = e; b; k++, b >>= 1)
    if (b & 1u) mul_lazy<P_r>(v, v, a.pw[(low ? 0 : a.shift) + k].w);
  reduce_once<P_r>(v, v);
  st_fe((low ? lo : hi) + e, v);
}

cudaError_t pow_tables_make(PowTables* t, const host::Fr& c, int log_n, cudaStream_t s, const host::Fr* scale,
                            bool pooled) {
  PowArgs a{};
  a.shift = (uint32_t)((log_n + 1) / 2);
  a.nlo = 1u << a.shift;
  a.nhi = 1u << (log_n - (int)a.shift);
  host::Fr x = c;
  for (int k = 0; k < log_n; k++, x = host::mul(x, x)) a.pw[k] = to_fe(x);
  if (scale) {
    a.has_scale = 1;
    a.scale = to_fe(*scale);
  }
  t->lo = t->hi = nullptr;
  t->shift = a.shift;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 2 && e == cudaSuccess; k++) {
    void** p = (void**)(k ? &t->hi : &t->lo);
    const size_t bytes = (size_t)(k ? a.nhi : a.nlo) * sizeof(fe);
    e = pooled ? zk::dmalloc(p, bytes, s) : cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess) {
    if (t->lo) pooled ? cudaFreeAsync(t->lo, s) : cudaFree(t->lo);
    t->lo = t->hi = nullptr;
    return e;
  }
  pow_tables_kernel<<<(a.nlo + a.nhi + 127) / 128, 128, 0, s>>>(t->lo, t->hi, a);
  return cudaGetLastError();
}
void pow_tables_free(PowTables* t, cudaStream_t s) {
  if (t->lo) cudaFreeAsync(t->lo, s);
  if (t->hi) cudaFreeAsync(t->hi, s);
  t->lo = t->hi = nullptr;
}

// elements of a pass's root table, and its launch
static uint64_t inner_elems(int B) { return B <= kNarrowMax ? 4ull * roots_entries(B) : 1ull << (B - 1); }
static void fill_inner(fe* out, DftConsts* dft, const host::Fr& wm, int B, cudaStream_t s) {
  const unsigned count = (unsigned)inner_elems(B), grid = (count + 255) / 256;
  if (B > kNarrowMax) {
    pow_seq_kernel<<<grid, 256, 0, s>>>(out, to_fe(wm), count, 1);
    return;
  }
  const host::Fr w8 = host::pow_2k(wm, (unsigned)(B - 3)), w4 = host::mul(w8, w8), w83 = host::mul(w4, w8);
  static const host::Fr half = host::inv(host::from_u64(2));
  Special sp;
  const host::Fr c[3] = {w4, host::mul(half, host::add(w8, w83)), host::mul(half, host::sub(w8, w83))};
  for (int k = 0; k < 3; k++) {
    sp.v[k] = to_fe(c[k]);
    for (int j = 0; j < 8; j++) std::memcpy(dft->w[k] + 8 * j, host::mul(c[k], host::pow2(32 * j + 64)).v, 32);
  }
  roots_w4_kernel<<<grid, 256, 0, s>>>(out, to_fe(wm), sp, table_scale(), B);
}

static cudaError_t build_tables(NttTables* t, cudaStream_t s) {
  const NttPlan& p = t->plan;
  int done_bits = 0;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < p.npass; k++) {
    const int b = p.bits[k];
    const int log_J = p.log_n - done_bits - b;  // later passes' bits
    // this pass works on the sub-problem of size m*J whose root is w^(n / (m J))
    const host::Fr wMJ = host::pow_2k(t->omega, (unsigned)done_bits);
    const host::Fr wm = host::pow_2k(wMJ, (unsigned)log_J);
    e = cudaMalloc((void**)&t->inner[k], inner_elems(b) * sizeof(fe));
    if (e != cudaSuccess) return e;
    t->bytes += inner_elems(b) * sizeof(fe);
    fill_inner(t->inner[k], &t->dft[k], wm, b, s);
    if (k + 1 < p.npass) {
      const uint64_t total = 1ull << (b + log_J);
      e = cudaMalloc((void**)&t->twist[k], 2 * total * sizeof(fe));
      if (e != cudaSuccess) return e;
      t->bytes += 2 * total * sizeof(fe);
      PowTables pw;
      e = pow_tables_make(&pw, wMJ, b + log_J, s);
      if (e != cudaSuccess) return e;
      twist_table_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(t->twist[k], pw.lo, pw.hi, pw.shift,
                                                                          (uint32_t)log_J, total, table_scale());
      pow_tables_free(&pw, s);
    }
    done_bits += b;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(s);
}

size_t ntt_tables_elems(int log_n) {
  const NttPlan p = make_ntt_plan(log_n);
  size_t total = 0;
  int done = 0;
  for (int k = 0; k < p.npass; k++) {
    const int b = p.bits[k];
    const int log_J = p.log_n - done - b;
    total += inner_elems(b);
    if (k + 1 < p.npass) {
      const int lc = b + log_J;
      const int sh = (lc + 1) / 2;
      total += (2ull << lc) + (1ull << sh) + (1ull << (lc > sh ? lc - sh : 0));
    }
    done += b;
  }
  return total;
}

cudaError_t ntt_tables_fill(NttTables* t, const host::Fr& omega, int log_n, fe* mem, size_t cap, cudaStream_t s) {
  if (ntt_tables_elems(log_n) > cap) return cudaErrorInvalidValue;
  t->plan = make_ntt_plan(log_n);
  t->omega = omega;
  t->bytes = 0;
  const NttPlan& p = t->plan;
  fe* cur = mem;
  int done = 0;
  for (int k = 0; k < p.npass; k++) {
    const int b = p.bits[k];
    const int log_J = p.log_n - done - b;
    const host::Fr wMJ = host::pow_2k(omega, (unsigned)done);
    const host::Fr wm = host::pow_2k(wMJ, (unsigned)log_J);
    t->inner[k] = cur;
    cur += inner_elems(b);
    fill_inner(t->inner[k], &t->dft[k], wm, b, s);
    if (k + 1 < p.npass) {
      const int lc = b + log_J;
      const uint32_t sh = (uint32_t)((lc + 1) / 2);
      const uint64_t total = 1ull << lc, nlo = 1ull << sh, nhi = 1ull << (lc > (int)sh ? lc - sh : 0);
      fe* lo = cur;
      fe* hi = cur + nlo;
      t->twist[k] = cur + nlo + nhi;
      cur += nlo + nhi + 2 * total;
      pow_seq_kernel<<<(unsigned)((nlo + 255) / 256), 256, 0, s>>>(lo, to_fe(wMJ), nlo, 1);
      pow_seq_kernel<<<(unsigned)((nhi + 255) / 256), 256, 0, s>>>(hi, to_fe(host::pow_2k(wMJ, sh)), nhi, 1);
      twist_table_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(t->twist[k], lo, hi, sh, (uint32_t)log_J,
                                                                          total, table_scale());
    } else {
      t->twist[k] = nullptr;
    }
    done += b;
  }
  return cudaGetLastError();
}

bool ntt_plan_valid(const NttPlan& p) {
  if (p.log_n < 0 || p.log_n > NTT_MAX_LOG) return false;
  if (p.log_n <= 2) return p.npass == 0;
  if (p.npass < 1 || p.npass > NTT_MAX_PASS) return false;
  if (p.npass == 1) return p.bits[0] == p.log_n && p.log_n <= 11;
  int sum = 0;
  for (int k = 0; k < p.npass; k++) {
    if (p.bits[k] < 3 || p.bits[k] > 11) return false;
    sum += p.bits[k];
  }
  for (int k = p.npass; k < NTT_MAX_PASS; k++)
    if (p.bits[k] != 0) return false;
  return sum == p.log_n;
}

cudaError_t ntt_tables_build(NttTables* t, const NttPlan& plan, const host::Fr& omega, cudaStream_t s) {
  if (!ntt_plan_valid(plan)) return cudaErrorInvalidValue;
  *t = NttTables{};
  t->plan = plan;
  t->omega = omega;
  cudaError_t e = build_tables(t, s);
  if (e != cudaSuccess) ntt_tables_release(t);
  return e;
}

void ntt_tables_release(NttTables* t) {
  for (int k = 0; k < NTT_MAX_PASS; k++) {
    if (t->inner[k]) cudaFree(t->inner[k]);
    if (t->twist[k]) cudaFree(t->twist[k]);
    t->inner[k] = t->twist[k] = nullptr;
  }
  t->bytes = 0;
}

static uint64_t ntt_pass_params(const NttTables& t, int k, fe* d_a, fe* d_tmp, const NttFuse& f, PassParams* out,
                                bool batch);

// Largest transform whose passes run two elements per thread (ntt_tile.cuh):
// above it the tile kernel fills the GPU.  B200, pair / tile kernel (us): 2^10
// 19.5 / 22.8 (both near the host's time to enqueue a call), 2^14 15.3 / 33.0,
// 2^16 26.9 / 35.8, 2^17 47.1 / 41.2, 2^18 84 / 58.
constexpr int kPairMaxLog = 16;

static cudaError_t dispatch_pair(int B, const PassParams& pp, int log_n, cudaStream_t s) {
  switch (B) {
    case 3: return launch_pair<3>(pp, log_n, s);
    case 4: return launch_pair<4>(pp, log_n, s);
    case 5: return launch_pair<5>(pp, log_n, s);
    case 6: return launch_pair<6>(pp, log_n, s);
    case 7: return launch_pair<7>(pp, log_n, s);
    case 8: return launch_pair<8>(pp, log_n, s);
    default: return cudaErrorInvalidValue;
  }
}

static cudaError_t dispatch_pass(int B, const PassParams& pp, const DftConsts& dft, uint64_t ncta, cudaStream_t s) {
  switch (B) {
    case 3: return launch_pass<3>(pp, dft, ncta, s);
    case 4: return launch_pass<4>(pp, dft, ncta, s);
    case 5: return launch_pass<5>(pp, dft, ncta, s);
    case 6: return launch_pass<6>(pp, dft, ncta, s);
    case 7: case 8: case 9: case 10: case 11: return launch_pass_wide(B, pp, dft, ncta, s);
    default: return cudaErrorInvalidValue;
  }
}

uint64_t ntt_batch_pass_params(const NttTables& t, int k, fe* d_a, fe* d_tmp, const NttFuse& f, BatchPass* out) {
  if (f.post) {
    static const host::Fr w2[2] = {host::pow2(160), host::pow2(288)};
    for (int j = 0; j < 2; j++) out->post[j] = to_fe(host::mul(*f.post, w2[j]));
  }
  return ntt_pass_params(t, k, d_a, d_tmp, f, &out->p, true);
}

static uint64_t ntt_pass_params(const NttTables& t, int k, fe* d_a, fe* d_tmp, const NttFuse& f, PassParams* out,
                                bool batch) {
  const PowTables* pre = f.pre;
  const host::Fr* post = f.post;
  const NttPlan& p = t.plan;
  const int L = p.log_n;
  int done = 0;
  for (int j = 0; j < k; j++) done += p.bits[j];
  const int b = p.bits[k];
  const bool final_pass = (k + 1 == p.npass);
  PassParams pp{};
  pp.inner = t.inner[k];
  pp.twist = t.twist[k];
  pp.log_J = (uint32_t)(L - done - b);
  pp.log_O = (uint32_t)done;
  // final-pass grouping runs over consecutive first digits k_1; a single-pass
  // plan has no digits (one group, rest_count = 1)
  pp.log_m1 = p.npass > 1 ? (uint32_t)p.bits[0] : 0u;
  pp.nprev = final_pass ? (uint32_t)k : 0u;
  for (int j = 0; j < k && j < NTT_MAX_PASS; j++) pp.prev_bits[j] = (uint32_t)p.bits[j];
  pp.is_first = k == 0 ? 1u : 0u;
  pp.is_final = final_pass ? 1u : 0u;
  if (k == 0 && pre) {
    pp.pre_lo = pre->lo;
    pp.pre_hi = pre->hi;
    pp.pre_shift = pre->shift;
  }
  if (final_pass && post) {
    pp.has_post = 1;
    pp.post = to_fe(*post);
  }
  pp.out_count = (uint32_t)(f.wanted ? f.wanted : 1ull << L);
  if (final_pass && f.post_tab) {
    pp.post_lo = f.post_tab->lo;
    pp.post_hi = f.post_tab->hi;
    pp.post_shift = f.post_tab->shift;
  }
  if (k == 0 && f.nonzero) {
    // first pass reads rows of J = 2^(L - b) elements: whole zero rows are skipped
    const uint64_t J = 1ull << (L - b);
    if (f.nonzero % J == 0 && f.nonzero / J < (1ull << b)) pp.in_rows = (uint32_t)(f.nonzero / J);
  }
  // buffers: single pass in place; otherwise a -> tmp, tmp in place, tmp -> a
  if (p.npass == 1) {
    pp.in = d_a;
    pp.out = d_a;
  } else if (k == 0) {
    pp.in = d_a;
    pp.out = d_tmp;
  } else if (!final_pass) {
    pp.in = d_tmp;
    pp.out = d_tmp;
  } else {
    pp.in = d_tmp;
    pp.out = d_a;
  }
  if (k == 0 && f.src) pp.in = f.src;  // out of place: the first pass reads the source
  // Tiles of 2^10 elements (128 threads), two to a block (2^24 as 8+8+8: 2780
  // us with one tile of 2^11, 2685 with two of 2^10); a pass with too few of
  // them to give every SM a block takes one to a block (2^16: 47 -> 35 us).
  // Passes wider than kNarrowMax keep tiles of 2^11.
  const int tile_log = b > kNarrowMax ? 11 : 10;
  const uint32_t Gmax = b >= tile_log ? 1u : (1u << (tile_log - b));
  uint64_t groups_dim;
  if (!final_pass) {
    groups_dim = 1ull << pp.log_J;  // columns per outer block
  } else if (p.npass == 1) {
    groups_dim = 1;
  } else {
    groups_dim = 1ull << p.bits[0];  // consecutive k_1 digits
  }
  pp.G = (uint32_t)std::min<uint64_t>(Gmax, groups_dim);
  const uint64_t tiles = (1ull << (L - b)) / pp.G;
  pp.ntile = b <= kNarrowMax && pp.G << (b - 3) == 128 && tiles >= (batch ? 2 : 256) ? 2u : 1u;
  *out = pp;
  return tiles / pp.ntile;
}

cudaError_t ntt_run(const NttTables& t, fe* d_a, fe* d_tmp, const PowTables* pre, const host::Fr* post, cudaStream_t s) {
  NttFuse f;
  f.pre = pre;
  f.post = post;
  return ntt_run(t, d_a, d_tmp, f, s);
}

cudaError_t ntt_run(const NttTables& t, fe* d_a, fe* d_tmp, const NttFuse& f, cudaStream_t s) {
  const PowTables* pre = f.pre;
  const host::Fr* post = f.post;
  const NttPlan& p = t.plan;
  const int L = p.log_n;
  if (L <= 2) {
    if (f.post_tab) return cudaErrorInvalidValue;  // the direct kernel takes constant scales only
    fe po{};
    if (post) po = to_fe(*post);
    ntt_tiny_kernel<<<1, 32, 0, s>>>(d_a, (uint32_t)L, to_fe(t.omega), pre ? pre->lo : nullptr, pre ? pre->hi : nullptr,
                                     pre ? pre->shift : 0u, post ? 1u : 0u, po);
    return cudaGetLastError();
  }
  static const char* names[12] = {"", "", "", "ntt_pass_b3", "ntt_pass_b4", "ntt_pass_b5", "ntt_pass_b6",
                                  "ntt_pass_b7", "ntt_pass_b8", "ntt_pass_b9", "ntt_pass_b10", "ntt_pass_b11"};
  for (int k = 0; k < p.npass; k++) {
    const int b = p.bits[k];
    PassParams pp;
    const uint64_t ncta = ntt_pass_params(t, k, d_a, d_tmp, f, &pp, false);
    const double nel = (double)(1ull << L);
    // algorithmic work: radix-2 convention (n/2) * b products; bytes: read + write (+ twist table)
    ProfScope prof(names[b], s, nel / 2 * b,
                   nel * 64.0 + (pp.is_final ? 0.0 : 64.0 * (double)(1ull << (L - (int)pp.log_O))));
    const bool small = L <= kPairMaxLog && b <= kNarrowMax;
    cudaError_t e = small ? dispatch_pair(b, pp, L, s) : dispatch_pass(b, pp, t.dft[k], ncta, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

static size_t batch_smem_bytes() {
  return (size_t)8 * 2048 * 4 + std::max(tw_smem_bytes(kNarrowMax), tw_smem_bytes(11));
}

int ntt_batch_grid(int device) {
  static int cached[64] = {0};
  if (device >= 0 && device < 64 && cached[device]) return cached[device];
  cudaFuncSetAttribute(ntt_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_smem_bytes());
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ntt_batch_kernel, 256, batch_smem_bytes());
  const int g = sms * (per_sm > 0 ? per_sm : 1);
  if (device >= 0 && device < 64) cached[device] = g;
  return g;
}

cudaError_t ntt_batch_launch(const BatchPass* d_passes, uint32_t npass, uint32_t total_tiles, uint32_t* d_next,
                             uint32_t* d_done, uint32_t* d_err, int grid, cudaStream_t s, uint64_t spin_cycles) {
  ntt_batch_kernel<<<grid, 256, batch_smem_bytes(), s>>>(d_passes, npass, total_tiles, d_next, d_done, d_err,
                                                         spin_cycles);
  return cudaGetLastError();
}

cudaError_t fr_scale_copy(fe* dst, const fe* src, size_t n, size_t dst_stride, const PowTables* powc, cudaStream_t s) {
  scale_copy_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dst, src, n, dst_stride, powc ? powc->lo : nullptr,
                                                               powc ? powc->hi : nullptr, powc ? powc->shift : 0);
  return cudaGetLastError();
}

}  // namespace zk
