// msm.cu — Pippenger MSM kernels and orchestration (see msm.cuh).
#include <algorithm>

#include "curve.cuh"
#include "msm.cuh"
#include "msm_field.cuh"
#include "quad.cuh"
#include "prof.cuh"
#include "runtime.cuh"

namespace zk {

MsmPlan make_msm_plan(uint64_t n, int c_override, int device) {
  MsmPlan p;
  int lg = 1;
  while ((1ull << lg) < n) lg++;
  int c = lg - 4;
  if (c < 4) c = 4;
  if (c > 16) c = 16;
  if (c_override == 0) {  // the autotuner's choice for this device and size, if any
    int dev = device;
    if (dev >= 0 || cudaGetDevice(&dev) == cudaSuccess) c_override = tuned_msm_window(dev, lg);
  }
  if (c_override >= 3 && c_override <= 20) c = c_override;
  p.c = c;
  p.windows = (254 + c - 1) / c;
  p.buckets = 1u << (c - 1);
  // Buckets per reduction segment: a segment's quad of lanes adds 2 L times one
  // after the other, and its sums then go through the group levels, about three
  // additions per segment.  Few buckets leave the GPU idle, so short chains win;
  // from 2^12 per window on it is full, and longer segments save work.  MSM of
  // n points on B200 with L = 4 / 8 / 16 / 32 (us): 2^14 (2^9 buckets) 396 / 418
  // / 460 / 526, 2^16 (2^11) 763 / 741 / 767 / 857, 2^18 (2^13) 1659 / 1652 /
  // 1670 / 1653, 300007 (2^14) 1812 / 1755 / 1724 / 1724, 2^20 (2^15) 4013 /
  // 3862 / 3789 / 3823.
  p.seg_len = std::min<uint32_t>(p.buckets >= 4096 ? 16u : 4u, p.buckets);
  return p;
}

// bits [pos, pos + c) of a canonical 256-bit scalar (c <= 20), 0 beyond bit 255
__device__ __forceinline__ uint32_t scalar_bits(const uint32_t s[8], uint32_t pos, uint32_t c) {
  const uint32_t w = pos >> 5, b = pos & 31;
  uint64_t v = 0;
  if (w < 8) v = s[w];
  if (w + 1 < 8) v |= (uint64_t)s[w + 1] << 32;
  return (uint32_t)(v >> b) & ((1u << c) - 1u);
}

// Signed digits of one scalar, low window first; calls f(w, digit) for
// each non-zero digit (digit in [-2^(c-1), 2^(c-1)]).
template <class F>
__device__ __forceinline__ void for_each_digit(const fe* scalar, uint32_t c, uint32_t windows, F f) {
  uint32_t s[8];
  ld_fe(s, scalar);
  uint32_t one[8] = {1, 0, 0, 0, 0, 0, 0, 0};
  mul<FrP>(s, s, one);  // out of Montgomery form (cuda/curve.cuh:111 does the same)
  const int half = 1 << (c - 1);
  uint32_t carry = 0;
  for (uint32_t w = 0; w < windows; w++) {
    int v = (int)scalar_bits(s, w * c, c) + (int)carry;
    if (v > half) {
      v -= 1 << c;
      carry = 1;
    } else {
      carry = 0;
    }
    if (v != 0) f(w, v);
  }
}

// Several MSMs over one base array in one pass: scalars of job j occupy
// [off[j], off[j+1]) of the concatenated scalar array, its windows are
// j * windows + w, and its entries name the base by the local index.
__device__ __forceinline__ uint32_t job_of(const uint32_t* off, uint32_t jobs, uint32_t i) {
  uint32_t lo = 0, hi = jobs;  // off[lo] <= i < off[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (off[mid] <= i) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void msm_count_kernel(const fe* scalars, uint64_t n, uint32_t c, uint32_t windows, uint32_t* counts,
                                 const uint32_t* job_off, uint32_t jobs) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t B = 1u << (c - 1);
  const uint32_t w0 = jobs > 1 ? job_of(job_off, jobs, (uint32_t)i) * windows : 0u;
  for_each_digit(scalars + i, c, windows, [&](uint32_t w, int d) {
    const uint32_t mag = (uint32_t)(d < 0 ? -d : d);
    atomicAdd(&counts[(w0 + w) * B + mag - 1], 1u);
  });
}

__global__ void msm_scatter_kernel(const fe* scalars, uint64_t n, uint32_t c, uint32_t windows, uint32_t* cursor,
                                   uint32_t* list, const uint32_t* job_off, uint32_t jobs) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t B = 1u << (c - 1);
  uint32_t w0 = 0, local = (uint32_t)i;
  if (jobs > 1) {
    const uint32_t j = job_of(job_off, jobs, (uint32_t)i);
    w0 = j * windows;
    local = (uint32_t)i - job_off[j];
  }
  for_each_digit(scalars + i, c, windows, [&](uint32_t w, int d) {
    const uint32_t mag = (uint32_t)(d < 0 ? -d : d);
    const uint32_t pos = atomicAdd(&cursor[(w0 + w) * B + mag - 1], 1u);
    list[pos] = local | (d < 0 ? 0x80000000u : 0u);
  });
}

// Exclusive scan, three phases over 1024-element blocks.
__global__ void scan_block_kernel(const uint32_t* in, uint32_t* out, uint32_t* block_sums, uint32_t total) {
  __shared__ uint32_t sh[1024];
  const uint32_t i = blockIdx.x * 1024 + threadIdx.x;
  const uint32_t v = i < total ? in[i] : 0;
  sh[threadIdx.x] = v;
  __syncthreads();
  for (uint32_t off = 1; off < 1024; off <<= 1) {
    uint32_t t = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
    __syncthreads();
    sh[threadIdx.x] += t;
    __syncthreads();
  }
  if (i < total) out[i] = sh[threadIdx.x] - v;
  if (threadIdx.x == 1023) block_sums[blockIdx.x] = sh[1023];
}
__global__ void scan_sums_kernel(uint32_t* block_sums, uint32_t nblocks, uint32_t* total_out) {
  // one block of 1024 threads; nblocks <= 1024 * 64
  __shared__ uint32_t sh[1024];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nblocks; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < nblocks ? block_sums[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (uint32_t off = 1; off < 1024; off <<= 1) {
      uint32_t t = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
      __syncthreads();
      sh[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < nblocks) block_sums[i] = carry + sh[threadIdx.x] - v;
    const uint32_t tot = sh[1023];
    __syncthreads();
    carry += tot;
  }
  if (threadIdx.x == 0) *total_out = carry;
}
__global__ void scan_add_kernel(uint32_t* out, uint32_t* cursor, const uint32_t* block_sums, uint32_t total) {
  const uint32_t i = blockIdx.x * 1024 + threadIdx.x;
  if (i >= total) return;
  const uint32_t v = out[i] + block_sums[blockIdx.x];
  out[i] = v;
  cursor[i] = v;
}

// ---------------------------------------------------------------------------
// Batch-affine bucket accumulation.
//
// Every bucket's points are summed by pairwise AFFINE additions in rounds:
// round r replaces the c points of a bucket by ceil(c / 2) points (pair sums,
// plus the odd last point carried).  An affine addition P + Q needs
// 1 / (x_Q - x_P); the inverses of a whole round come from Montgomery's
// trick in two levels:
//   prefix  : each thread task owns BA_K consecutive pair sums and chains
//             the products of their denominators (stored, 1 product each);
//   invert  : each inversion thread takes BA_G task products, chains them,
//             inverts the chain's product once (Fermat) and walks back;
//   apply   : each task walks its chain back (2 products per sum) and
//             finishes the additions (lambda, lambda^2, lambda (x1 - x3):
//             3 products).
// That is about 6 + 3 / BA_K ~ 6.2 Fq products per point addition (the XYZZ
// mixed addition costs 10) plus one inversion per 512 additions, done by
// the branch-free divstep algorithm of fq_inv.cuh (~25k instructions of
// 32-bit integer work against ~330 dependent products for a Fermat power),
// with no serial block-wide step.  Equal x
// (P = Q: doubling, denominator 2y; P = -Q: identity) and the identity
// (x = 0: no BN254 point has x = 0, as 3 is not a square mod q) are handled
// per sum.  A bucket reaching one point writes it to `fin`; after the last
// round a tail kernel folds what remains (skewed buckets) with XYZZ mixed
// additions and writes every bucket as XYZZ for the reduction.
// ---------------------------------------------------------------------------
constexpr uint32_t BA_K = 16;  // pair sums per task (one chain of products)
constexpr uint32_t BA_G = 32;  // task products per inversion
// Apply blocks: five of 128 threads per SM fit at the 96 registers the kernel
// needs (MSM of 2^22: 11.95 ms with two of 256, 11.73 ms so).
constexpr uint32_t BA_APPLY = 128;

// ---- per-thread copy pipeline ---------------------------------------------
// The prefix and apply passes are chains of dependent gathers (bucket
// metadata -> entry list -> point) and field products.  Each thread stages
// the operands of its next pair sum into shared memory with cp.async (16-B
// copies that hold no registers while in flight) while it computes the
// current one, and loads the entry-list words one job further ahead, so the
// gather latency overlaps the products.  Stage slots are chunk-major: chunk
// k of stage s of thread t is the 16-B word ((s * CH + k) * blockDim + t),
// so the 16-B accesses of a warp to one chunk are 32 consecutive words.
// .cg: through L2 only; staged data is read once, so allocating it in L1
// only evicts other lines.  (Round 0's random 32-B and 64-B gathers move
// whole 128-B lines from DRAM either way: 6.5 GB of DRAM reads for 2.2 GB
// of x coordinates in the 2^22-point prefix pass, measured on B200.)
__device__ __forceinline__ void cp16(uint4* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// one fe (two chunks) of a stage: copy in, read out
__device__ __forceinline__ void cp_fe(uint4* my, uint32_t bd, uint32_t k, const fe* g) {
  const uint4* v = reinterpret_cast<const uint4*>(g);
  cp16(my + k * bd, v);
  cp16(my + (k + 1) * bd, v + 1);
}
__device__ __forceinline__ void sm_fe(uint32_t r[8], const uint4* my, uint32_t bd, uint32_t k) {
  const uint4 x = my[k * bd], y = my[(k + 1) * bd];
  r[0] = x.x; r[1] = x.y; r[2] = x.z; r[3] = x.w;
  r[4] = y.x; r[5] = y.y; r[6] = y.z; r[7] = y.w;
}

// one pair sum of a round: its two points in the round's source (round 0:
// entry-list words, base index plus sign bit; later rounds: positions in the
// previous round's output), its bucket, whether the second point exists,
// whether it is its bucket's first, and the bucket's points after the round
constexpr uint32_t BA_CP = 4;   // chunks per prefix stage: x of both points
constexpr uint32_t BA_CA = 10;  // chunks per apply stage: both points, one prefix product
struct BaJob {
  uint32_t pa, pb, b, nb;
  bool has2, first;
};

// point p of a round's source ((x, y) adjacent): round 0 reads the bases
// (the entry's index, sign bit cleared), later rounds their own buffer of
// affine pair sums.  (Bases kept as an x array and a y array instead were
// measured on B200 at 2^22 points: the prefix pass's x gathers hit L2 more,
// 1.28 -> 1.15 ms, and the apply pass's separate y gathers cost as much,
// 3.94 -> 4.06 ms.)
template <bool FIRST>
__device__ __forceinline__ const fe* ba_pt(const fe* src, uint32_t p) {
  return src + 2 * (uint64_t)(FIRST ? (p & 0x7fffffffu) : p);
}
// y of a round-0 point read out of its slot: q - y for a negative digit
template <bool FIRST>
__device__ __forceinline__ void ba_sign(aff_t& p, uint32_t e) {
  if (FIRST) {
    uint32_t z[8] = {0, 0, 0, 0, 0, 0, 0, 0}, n[8];
    sub_off<FqP, 1>(n, z, p.y);
    const bool neg = (e & 0x80000000u) && !is_zero(p.y);
#pragma unroll
    for (int k = 0; k < 8; k++) p.y[k] = neg ? n[k] : p.y[k];
  }
}

// bucket of job q: the largest b' with joff[b'] <= q, searched from the
// bucket of a neighbouring job (forward: joff[b] <= q; backward: q < joff[b + 1])
__device__ __forceinline__ uint32_t ba_search(const uint32_t* __restrict__ joff, uint32_t lo, uint32_t hi,
                                              uint32_t q) {
  while (hi - lo > 1) {  // joff[lo] <= q < joff[hi]
    const uint32_t mid = (lo + hi) >> 1;
    if (joff[mid] <= q) lo = mid; else hi = mid;
  }
  return lo;
}
// The bucket a thread's chain is in, kept in registers while the chain stays
// in it: a job then costs no load but its entry-list words (three dependent
// loads per job left 2.2 stalled warps per issue in the apply pass).
struct BaCursor {
  const uint32_t *joff, *in_off, *cprev;
  uint32_t T, b, j0, j1, in0, c;  // bucket, its jobs [j0, j1), its first point, its points
  __device__ __forceinline__ void load() {
    j0 = joff[b];
    j1 = joff[b + 1];
    in0 = in_off[b];
    c = cprev[b];
  }
  __device__ __forceinline__ BaCursor(const uint32_t* joff_, const uint32_t* in_off_, const uint32_t* cprev_,
                                      uint32_t T_, uint32_t q)
      : joff(joff_), in_off(in_off_), cprev(cprev_), T(T_) {
    b = ba_search(joff, 0, T, q);
    load();
  }
  // job q in the cursor's bucket or after (before) it
  __device__ __forceinline__ void forward(uint32_t q) {
    if (q < j1) return;
    b++;
    load();
    if (q < j1) return;
    b = ba_search(joff, b + 1, T, q);
    load();
  }
  __device__ __forceinline__ void backward(uint32_t q) {
    if (q >= j0) return;
    b--;
    load();
    if (q >= j0) return;
    b = ba_search(joff, 0, b, q);
    load();
  }
  template <bool FIRST>
  __device__ __forceinline__ BaJob job(uint32_t q, const uint32_t* __restrict__ list) const {
    BaJob d;
    const uint32_t j = q - j0, i0 = in0 + 2 * j;
    d.b = b;
    d.nb = (c + 1) / 2;
    d.first = j == 0;
    d.has2 = 2 * j + 1 < c;
    if (FIRST) {
      d.pa = list[i0];
      d.pb = d.has2 ? list[i0 + 1] : 0u;
    } else {
      d.pa = i0;
      d.pb = i0 + 1;
    }
    return d;
  }
};

// stage the x coordinates of a job's points (prefix pass)
template <bool FIRST>
__device__ __forceinline__ void ba_stage_x(uint4* st, uint32_t bd, const fe* src, const BaJob& d) {
  if (!d.has2) return;
  cp_fe(st, bd, 0, ba_pt<FIRST>(src, d.pa));
  cp_fe(st, bd, 2, ba_pt<FIRST>(src, d.pb));
}
// stage both points of a job and the prefix product before it (apply pass)
template <bool FIRST>
__device__ __forceinline__ void ba_stage_pq(uint4* st, uint32_t bd, const fe* src, const BaJob& d, const fe* p) {
  const fe* a = ba_pt<FIRST>(src, d.pa);
  cp_fe(st, bd, 0, a);
  cp_fe(st, bd, 2, a + 1);
  if (d.has2) {
    const fe* c = ba_pt<FIRST>(src, d.pb);
    cp_fe(st, bd, 4, c);
    cp_fe(st, bd, 6, c + 1);
  }
  if (p) cp_fe(st, bd, 8, p);
}

// denominator of one pair sum (one when no inversion is needed: a carried
// point, an identity operand, or P = -Q), from the staged x coordinates;
// equal x (doubling or P = -Q, rare) reads both points again for y
template <bool FIRST>
__device__ __forceinline__ void ba_denominator(uint32_t d[8], const uint4* st, uint32_t bd, const fe* src,
                                               const BaJob& job) {
  if (job.has2) {
    uint32_t x1[8], x2[8];
    sm_fe(x1, st, bd, 0);
    sm_fe(x2, st, bd, 2);
    if (!is_zero(x1) && !is_zero(x2)) {
      if (!eq(x1, x2)) {
        sub_off<FqP, 1>(d, x2, x1);
        return;
      }
      aff_t p, q;
      ld_aff(p, ba_pt<FIRST>(src, job.pa));
      ld_aff(q, ba_pt<FIRST>(src, job.pb));
      ba_sign<FIRST>(p, job.pa);
      ba_sign<FIRST>(q, job.pb);
      if (eq(p.y, q.y)) {
        add<FqP>(d, p.y, p.y);
        return;
      }
    }
  }
  set_one<FqP>(d);
}

// buckets with at most one entry are final before any round; every count
// is copied for the rounds
__global__ void ba_setup_kernel(const uint32_t* counts, const uint32_t* offsets, const uint32_t* list,
                                const fe* bases, uint32_t* cnt, fe* fin, uint32_t T) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= T) return;
  const uint32_t c = counts[b];
  cnt[b] = c;
  if (c == 1) {
    aff_t p;
    const uint32_t e = list[offsets[b]];
    ld_aff(p, ba_pt<true>(bases, e));
    ba_sign<true>(p, e);
    st_fe(fin + 2 * (uint64_t)b, p.x);
    st_fe(fin + 2 * (uint64_t)b + 1, p.y);
  } else if (c == 0) {
    uint32_t z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    st_fe(fin + 2 * (uint64_t)b, z);
    st_fe(fin + 2 * (uint64_t)b + 1, z);
  }
}

__global__ void ba_jobs_kernel(const uint32_t* cnt, uint32_t* cprev, uint32_t* np, uint32_t T) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= T) return;
  const uint32_t c = cnt[b];
  cprev[b] = c;
  np[b] = c >= 2 ? (c + 1) / 2 : 0;
}

// prefix: task t covers jobs [t K, t K + K) of the round (J = joff[T])
// pair sums per task in a round of J sums: BA_K when the round fills the GPU
// with tasks, fewer (down to one) in small rounds, whose latency is then one
// short chain instead of BA_K dependent gathers and products
__device__ __forceinline__ uint32_t ba_task_len(uint32_t J, uint32_t fill_k) {
  return max(1u, min(BA_K, J / fill_k));
}

// dynamic shared memory: 2 stages x BA_CP chunks x 16 B per thread
template <bool FIRST>
__global__ void __launch_bounds__(256) ba_prefix_kernel(const fe* __restrict__ src, const uint32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ in_off,
                                                        const uint32_t* __restrict__ cprev,
                                                        const uint32_t* __restrict__ joff, uint32_t T,
                                                        fe* __restrict__ pre, fe* __restrict__ tot,
                                                        uint32_t fill_k) {
  extern __shared__ uint4 ba_smem[];
  const uint32_t bd = blockDim.x;
  uint4* my = ba_smem + threadIdx.x;
  const uint32_t J = joff[T];
  const uint32_t K = ba_task_len(J, fill_k);
  const uint32_t tasks = (J + K - 1) / K;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < tasks; t += gridDim.x * blockDim.x) {
    const uint32_t q0 = t * K, q1 = min(q0 + K, J);
    BaCursor at(joff, in_off, cprev, T, q0);
    BaJob d0 = at.job<FIRST>(q0, list), d1 = d0;
    ba_stage_x<FIRST>(my, bd, src, d0);
    cp_commit();
    if (q0 + 1 < q1) {
      at.forward(q0 + 1);
      d1 = at.job<FIRST>(q0 + 1, list);
    }
    uint32_t acc[8];
    for (uint32_t q = q0; q < q1; q++) {
      const uint32_t s = (q - q0) & 1;
      if (q + 1 < q1) ba_stage_x<FIRST>(my + (s ^ 1) * BA_CP * bd, bd, src, d1);
      cp_commit();
      BaJob d2 = d1;
      if (q + 2 < q1) {
        at.forward(q + 2);
        d2 = at.job<FIRST>(q + 2, list);
      }
      cp_wait<1>();
      uint32_t d[8];
      ba_denominator<FIRST>(d, my + s * BA_CP * bd, bd, src, d0);
      if (q == q0)
        cpy(acc, d);
      else
        mul_lazy<FqP>(acc, acc, d);
      st_fe(pre + q, acc);
      d0 = d1;
      d1 = d2;
    }
    st_fe(tot + t, acc);
  }
  cp_wait<0>();
}

// invert: thread s turns tot[s G .. s G + G) into their inverses.  The
// group length G follows the round's size: up to BA_G task products per
// inversion when there are many, down to one when a round is small, so that
// the round's latency is one inversion plus a short chain.
__global__ void __launch_bounds__(128) ba_invert_kernel(fe* tot, fe* tpre, const uint32_t* joff, uint32_t T,
                                                        uint32_t fill, uint32_t fill_k) {
  const uint32_t J = joff[T];
  const uint32_t K = ba_task_len(J, fill_k);
  const uint32_t tasks = (J + K - 1) / K;
  const uint32_t G = max(1u, min(BA_G, tasks / fill));
  const uint32_t groups = (tasks + G - 1) / G;
  for (uint32_t sgi = blockIdx.x * blockDim.x + threadIdx.x; sgi < groups; sgi += gridDim.x * blockDim.x) {
    const uint32_t i0 = sgi * G, i1 = min(i0 + G, tasks);
    uint32_t acc[8], v[8];
    ld_fe(acc, tot + i0);
    st_fe(tpre + i0, acc);
    for (uint32_t i = i0 + 1; i < i1; i++) {
      ld_fe(v, tot + i);
      qmul(acc, acc, v);
      st_fe(tpre + i, acc);
    }
    uint32_t inv[8];
    fq_inv_mont(inv, acc);
    for (uint32_t i = i1 - 1; i > i0; i--) {
      uint32_t p[8], it[8];
      ld_fe(p, tpre + i - 1);
      ld_fe(v, tot + i);
      qmul(it, inv, p);
      qmul(inv, inv, v);
      st_fe(tot + i, it);
    }
    st_fe(tot + i0, inv);
  }
}

// apply: walk each task's chain back and finish its pair sums; dynamic
// shared memory: 2 stages x BA_CA chunks x 16 B per thread
template <bool FIRST>
__global__ void __launch_bounds__(BA_APPLY, 5) ba_apply_kernel(const fe* __restrict__ src,
                                                          const uint32_t* __restrict__ list,
                                                          const uint32_t* __restrict__ in_off,
                                                          const uint32_t* __restrict__ cprev,
                                                          const uint32_t* __restrict__ joff, uint32_t T,
                                                          const fe* __restrict__ pre, const fe* __restrict__ tot,
                                                          fe* __restrict__ dst, fe* __restrict__ fin,
                                                          uint32_t* __restrict__ cnt, uint32_t fill_k) {
  extern __shared__ uint4 ba_smem[];
  const uint32_t bd = blockDim.x;
  uint4* my = ba_smem + threadIdx.x;
  const uint32_t J = joff[T];
  const uint32_t K = ba_task_len(J, fill_k);
  const uint32_t tasks = (J + K - 1) / K;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < tasks; t += gridDim.x * blockDim.x) {
    const uint32_t q0 = t * K, q1 = min(q0 + K, J);
    uint32_t inv_run[8];
    ld_fe(inv_run, tot + t);
    BaCursor at(joff, in_off, cprev, T, q1 - 1);
    BaJob d0 = at.job<FIRST>(q1 - 1, list), d1 = d0;
    ba_stage_pq<FIRST>(my, bd, src, d0, q1 - 1 > q0 ? pre + q1 - 2 : nullptr);
    cp_commit();
    if (q1 - 1 > q0) {
      at.backward(q1 - 2);
      d1 = at.job<FIRST>(q1 - 2, list);
    }
    for (uint32_t q = q1, i = 0; q-- > q0; i++) {
      const uint32_t s = i & 1;
      if (q > q0) ba_stage_pq<FIRST>(my + (s ^ 1) * BA_CA * bd, bd, src, d1, q - 1 > q0 ? pre + q - 2 : nullptr);
      cp_commit();
      BaJob d2 = d1;
      if (q > q0 + 1) {
        at.backward(q - 2);
        d2 = at.job<FIRST>(q - 2, list);
      }
      cp_wait<1>();
      const uint4* st = my + s * BA_CA * bd;
      const bool has2 = d0.has2;
      aff_t P, Q, out;
      sm_fe(P.x, st, bd, 0);
      sm_fe(P.y, st, bd, 2);
      ba_sign<FIRST>(P, d0.pa);
      if (has2) {
        sm_fe(Q.x, st, bd, 4);
        sm_fe(Q.y, st, bd, 6);
        ba_sign<FIRST>(Q, d0.pb);
      }
      // the same denominator the prefix pass chained (ba_denominator)
      uint32_t d[8];
      int kind = 0;  // 0: no inversion, 1: addition, 2: doubling
      if (has2 && !is_zero(P.x) && !is_zero(Q.x)) {
        if (!eq(P.x, Q.x)) {
          sub_off<FqP, 1>(d, Q.x, P.x);
          kind = 1;
        } else if (eq(P.y, Q.y)) {
          add<FqP>(d, P.y, P.y);
          kind = 2;
        }
      }
      if (kind == 0) set_one<FqP>(d);
      uint32_t inv_d[8];
      if (q > q0) {
        uint32_t p[8];
        sm_fe(p, st, bd, 8);
        mul_lazy<FqP>(inv_d, inv_run, p);
        mul_lazy<FqP>(inv_run, inv_run, d);
      } else {
        cpy(inv_d, inv_run);
      }
      if (!has2 || is_zero(Q.x)) {
        out = P;
      } else if (is_zero(P.x)) {
        out = Q;
      } else if (kind == 0) {  // P = -Q
        set_zero(out.x);
        set_zero(out.y);
      } else {
        // coordinates are canonical, products below 2q; each difference gets
        // the multiple of q that keeps it positive
        uint32_t lam[8], t1[8];
        if (kind == 1) {
          sub_off<FqP, 1>(t1, Q.y, P.y);
        } else {  // doubling: 3 x^2 / (2 y)
          mul_out<FqP>(t1, P.x, P.x);
          uint32_t t2[8];
          add_lazy<FqP>(t2, t1, t1);
          add_lazy<FqP>(t1, t2, t1);
        }
        mul_lazy<FqP>(lam, t1, inv_d);
        mul_lazy<FqP>(t1, lam, lam);
        add_raw(d, P.x, Q.x);  // Q.x = P.x when doubling
        sub_off<FqP, 2>(out.x, t1, d);
        cond_sub<FqP, 2>(out.x);
        cond_sub<FqP, 1>(out.x);
        sub_off<FqP, 1>(t1, P.x, out.x);
        mul_lazy<FqP>(t1, lam, t1);
        sub_off<FqP, 1>(out.y, t1, P.y);
        cond_sub<FqP, 2>(out.y);
        cond_sub<FqP, 1>(out.y);
      }
      fe* o = d0.nb == 1 ? fin + 2 * (uint64_t)d0.b : dst + 2 * (uint64_t)q;
      st_fe(o, out.x);
      st_fe(o + 1, out.y);
      if (d0.first) cnt[d0.b] = d0.nb;
      d0 = d1;
      d1 = d2;
    }
  }
  cp_wait<0>();
}

// Tail: what the rounds left (a few points per bucket, or many in a skewed
// bucket such as the one small scalars carry into), or, without rounds, the
// entries themselves, is folded with XYZZ mixed additions in chunks of at most
// BA_TS points, one thread per chunk; a bucket's chunk sums are then added by
// one quad of lanes (quad.cuh), or by blocks when there are many.
// Points per tail chunk: a chunk more costs an addition of two sums (14
// products) for one of its mixed additions (10), and short chunks of equal
// length keep a warp's lanes together.
constexpr uint32_t BA_TS = 8;
constexpr uint32_t BA_TSEQ = 24;     // chunk sums a bucket adds one by one
constexpr uint32_t BA_HEAVY = 2048;  // chunk sums a block adds

__device__ __forceinline__ uint32_t ba_chunk_count(uint32_t c) { return c <= 1 ? 1u : (c + BA_TS - 1) / BA_TS; }
__global__ void ba_chunks_kernel(const uint32_t* cnt, uint32_t* nch, uint32_t T) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= T) return;
  nch[b] = ba_chunk_count(cnt[b]);
}

// ENTRIES: the points are the bases named by the sorted list; otherwise the
// last round's sums (buckets of one point in `fin`).  A bucket's chunks share
// its points evenly, so that a warp's lanes run chains of similar length.  The
// next point is copied to the thread's slot of shared memory while the current
// one is added (two stages, as in the rounds).
template <bool ENTRIES>
__global__ void __launch_bounds__(256, 2) ba_fold_kernel(const uint32_t* __restrict__ cnt,
                                                         const uint32_t* __restrict__ in_off,
                                                         const fe* __restrict__ src, const uint32_t* __restrict__ list,
                                                         const fe* __restrict__ fin, const uint32_t* __restrict__ coff,
                                                         uint32_t T, fe* __restrict__ chunk_res) {
  __shared__ uint4 stage[2 * 4 * 256];
  uint4* my = stage + threadIdx.x;
  const uint32_t C = coff[T];
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < C; u += gridDim.x * blockDim.x) {
    const uint32_t b = ba_search(coff, 0, T, u);
    const uint32_t c = cnt[b], o = in_off[b], k = u - coff[b], nk = ba_chunk_count(c);
    const uint32_t i0 = (uint32_t)((uint64_t)c * k / nk), i1 = (uint32_t)((uint64_t)c * (k + 1) / nk);
    xyzz_t acc;
    xyzz_set_inf(acc);
    aff_t p;
    if (!ENTRIES && c <= 1) {
      ld_aff(p, fin + 2 * (uint64_t)b);
      xyzz_from_aff(acc, p);  // (0, 0) -> identity
    } else if (i0 < i1) {
      uint32_t e = ENTRIES ? list[o + i0] : o + i0, e1 = e;
      const fe* g = ba_pt<ENTRIES>(src, e);
      cp_fe(my, 256, 0, g);
      cp_fe(my, 256, 2, g + 1);
      cp_commit();
      if (i0 + 1 < i1) e1 = ENTRIES ? list[o + i0 + 1] : o + i0 + 1;
      for (uint32_t i = i0; i < i1; i++) {
        const uint32_t s = (i - i0) & 1u;
        uint32_t e2 = e1;
        if (i + 1 < i1) {
          g = ba_pt<ENTRIES>(src, e1);
          cp_fe(my + (s ^ 1u) * 1024, 256, 0, g);
          cp_fe(my + (s ^ 1u) * 1024, 256, 2, g + 1);
          if (i + 2 < i1) e2 = ENTRIES ? list[o + i + 2] : o + i + 2;
        }
        cp_commit();
        cp_wait<1>();
        sm_fe(p.x, my + s * 1024, 256, 0);
        sm_fe(p.y, my + s * 1024, 256, 2);
        ba_sign<ENTRIES>(p, e);
        xyzz_madd<true>(acc, p);
        e = e1;
        e1 = e2;
      }
    }
    st_xyzz(chunk_res + 4 * (uint64_t)u, acc);
  }
  cp_wait<0>();
}

// heavy: items (bucket, first chunk) of the buckets with more than BA_TSEQ
// chunk sums, one per BA_HEAVY of them; heavy_count = {items, buckets}
__global__ void __launch_bounds__(128) ba_bucket_sum_kernel(const uint32_t* coff, const fe* chunk_res, fe* buckets,
                                                            uint2* heavy, uint32_t* heavy_b, uint32_t* heavy_count,
                                                            uint32_t T) {
  const Quad z;
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  if (b >= T) return;
  const uint32_t o = coff[b], k = coff[b + 1] - o;
  if (k > BA_TSEQ) {
    if (z.j == 0) {
      const uint32_t n = (k + BA_HEAVY - 1) / BA_HEAVY, at = atomicAdd(heavy_count, n);
      for (uint32_t i = 0; i < n; i++) heavy[at + i] = make_uint2(b, i * BA_HEAVY);
      heavy_b[atomicAdd(heavy_count + 1, 1u)] = b;
    }
    return;
  }
  uint32_t acc[8], x[8];
  const fe* src = chunk_res + 4 * (uint64_t)o + z.j;
  ld_fe(acc, src);
  for (uint32_t j = 1; j < k; j++) {
    ld_fe(x, src + 4 * j);
    quad_add(z, acc, x);
  }
  st_fe(buckets + 4 * (uint64_t)b + z.j, acc);
}

// The block's sum of points src[first], src[first + step], .. below `end`, by
// its 64 quads: strided partial sums, then a tree in shared memory; quad 0
// holds it.
__device__ __forceinline__ void block_sum(const Quad& z, uint32_t acc[8], fe* sh, const fe* src, uint32_t first,
                                          uint32_t end, uint32_t step) {
  const uint32_t t = threadIdx.x >> 2, nt = blockDim.x >> 2;
  uint32_t x[8];
  set_zero(acc);
  for (uint32_t j = first + t * step; j < end; j += nt * step) {
    ld_fe(x, src + 4 * (uint64_t)j + z.j);
    quad_add(z, acc, x);
  }
  st_fe(sh + 4 * t + z.j, acc);
  __syncthreads();
  for (uint32_t half = nt / 2; half > 0; half >>= 1) {
    if (t < half) {
      ld_fe(x, sh + 4 * (t + half) + z.j);
      quad_add(z, acc, x);
      st_fe(sh + 4 * t + z.j, acc);
    }
    __syncthreads();
  }
}
// Heavy buckets in two steps: each item's chunk sums into its first one, then
// each bucket's items.
__global__ void __launch_bounds__(256) ba_heavy_items_kernel(const uint32_t* coff, fe* chunk_res, const uint2* heavy,
                                                             const uint32_t* heavy_count) {
  __shared__ __align__(16) fe sh[256];
  const Quad z;
  const uint32_t n = heavy_count[0];
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint2 it = heavy[i];
    const uint32_t o = coff[it.x] + it.y, end = min(o + BA_HEAVY, coff[it.x + 1]);
    uint32_t acc[8];
    block_sum(z, acc, sh, chunk_res, o, end, 1);
    if (threadIdx.x < 4) st_fe(chunk_res + 4 * (uint64_t)o + z.j, acc);
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256) ba_heavy_kernel(const uint32_t* coff, const fe* chunk_res, fe* buckets,
                                                       const uint32_t* heavy_b, const uint32_t* heavy_count) {
  __shared__ __align__(16) fe sh[256];
  const Quad z;
  const uint32_t n = heavy_count[1];
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t b = heavy_b[i];
    uint32_t acc[8];
    block_sum(z, acc, sh, chunk_res, coff[b], coff[b + 1], BA_HEAVY);
    if (threadIdx.x < 4) st_fe(buckets + 4 * (uint64_t)b + z.j, acc);
    __syncthreads();
  }
}

// Bucket reduction.  A window's sum is W = sum_j (j + 1) B_j over its B
// buckets.  Level 1, a quad of lanes (quad.cuh) per segment of L buckets:
// running sums from the top give T_s = sum_i (i + 1) B_{sL+i} and
// S_s = sum_i B_{sL+i}, so W = sum_s T_s + L sum_s s S_s.
__global__ void __launch_bounds__(128) msm_segment_kernel(const fe* buckets, fe* seg_t, fe* seg_s, uint32_t B,
                                                          uint32_t L, uint32_t total_segs) {
  const Quad z;
  const uint32_t gs = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  if (gs >= total_segs) return;
  const uint32_t S_per_w = B / L;
  const uint32_t w = gs / S_per_w, s = gs % S_per_w;
  const fe* bk = buckets + 4 * ((uint64_t)w * B + (uint64_t)s * L) + z.j;
  uint32_t run[8], tot[8], x[8];
  ld_fe(run, bk + 4 * (L - 1));
  cpy(tot, run);
  for (int j = (int)L - 2; j >= 0; j--) {
    ld_fe(x, bk + 4 * j);
    quad_add(z, run, x);
    quad_add(z, tot, run);
  }
  st_fe(seg_t + 4 * (uint64_t)gs + z.j, tot);
  st_fe(seg_s + 4 * (uint64_t)gs + z.j, run);
}

// Level 2 and up, a group of S <= 16 quads per S segments: with segments of L
// buckets, (T_s, S_s), the group is a segment of S L buckets with
// T = sum_t T_t + L sum_{t>=1} P_t, P_t = sum_{u>=t} S_u, and S = P_0.  A suffix
// scan gives the P_t, a tree adds T_t + L P_t: logarithmic depth, where running
// sums would take three additions per segment one after the other.  The last
// level's groups are the windows.  Points pass between quads through shared
// memory; a window's work is spread over groups because a block's products are
// one SM's (one block per window, scanning 1024 segments, took 240 us).
constexpr uint32_t kGroup = 16;
__global__ void __launch_bounds__(4 * kGroup) msm_group_kernel(const fe* in_t, const fe* in_s, fe* out_t, fe* out_s,
                                                               uint32_t S, uint32_t L) {
  __shared__ __align__(16) fe sh[2][4 * kGroup];
  const Quad z;
  const uint32_t g = blockIdx.x, t = threadIdx.x >> 2;
  uint32_t v[8], c[8], x[8];
  const uint64_t base = 4 * ((uint64_t)g * S + t) + z.j;
  ld_fe(v, in_s + base);
  ld_fe(c, in_t + base);
  uint32_t cur = 0;
  st_fe(&sh[0][4 * t + z.j], v);
  __syncthreads();
  for (uint32_t off = 1; off < S; off <<= 1) {
    if (t + off < S) {
      ld_fe(x, &sh[cur][4 * (t + off) + z.j]);
      quad_add(z, v, x);
    }
    cur ^= 1u;
    st_fe(&sh[cur][4 * t + z.j], v);
    __syncthreads();
  }
  if (t == 0) {
    if (out_s) st_fe(out_s + 4 * (uint64_t)g + z.j, v);
  } else {
    for (uint32_t m = L; m > 1; m >>= 1) quad_dbl(z, v);
    quad_add(z, c, v);
  }
  for (uint32_t half = S / 2; half > 0; half >>= 1) {
    cur ^= 1u;
    if (t >= half && t < 2 * half) st_fe(&sh[cur][4 * t + z.j], c);
    __syncthreads();
    if (t < half) {
      ld_fe(x, &sh[cur][4 * (t + half) + z.j]);
      quad_add(z, c, x);
    }
  }
  if (t == 0) st_fe(out_t + 4 * (uint64_t)g + z.j, c);
}

__global__ void zero_out_kernel(uint64_t* out) {
  if (threadIdx.x < 12) out[threadIdx.x] = 0;
}

namespace {
// tasks of a round of at most jb pair sums (ba_task_len: K = clamp(J / fill_k, 1, BA_K))
uint64_t ba_tasks_bound(uint64_t jb, uint64_t fill_k) {
  return std::max<uint64_t>(2 * fill_k, jb / BA_K + 1);
}
constexpr uint32_t kFillK = 148 * 64;  // task threads that fill a B200 (148 SMs) at 64 per SM

// dynamic shared memory of the round kernels (two stages): 32 and 40 KiB, below
// the 48 KiB a kernel gets without asking
constexpr int kPrefixSmem = 2 * BA_CP * 16 * 256;
constexpr int kApplySmem = 2 * BA_CA * 16 * BA_APPLY;
static_assert(kPrefixSmem <= 48 << 10 && kApplySmem <= 48 << 10, "needs cudaFuncSetAttribute");

int sm_count(int dev = -1) {
  int sms = 148;
  if (dev < 0) cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Buffer sizes of one MSM pass (msm_run_impl allocates exactly these;
// msm_scratch_bytes reports them for admission).
struct MsmLayout {
  MsmPlan p;
  uint32_t Wj = 0, W = 0, B = 0, L = 0, T = 0, nblk = 0, segs = 0, rounds = 0;
  uint64_t E = 0;                // entries (point-window pairs), upper bound
  uint64_t jb[2] = {0, 0};       // pair sums of rounds 0 and 1, upper bounds
  uint64_t tasks0 = 0;
  uint64_t chunks = 0;           // tail chunks, upper bound
  uint64_t heavy = 0;            // heavy buckets and their items, upper bound
  bool ok = false;
  uint64_t bytes(bool own_winsum) const {
    const uint64_t T1 = T + 1ull;
    uint64_t b = 0;
    b += T * 4ull * 2 + T1 * 4 + (nblk + 1ull) * 4 + E * 4;        // counts, cursor, offsets, bsums, list
    b += T1 * 4;                                                  // chunk offsets
    if (rounds) {
      b += T * 4ull * 3 + T1 * 4 + T * 64ull;                        // cnt, cprev, np, second offsets, fin
      b += jb[0] * 64 + (rounds > 1 ? jb[1] * 64 : 0) + jb[0] * 32;  // round buffers, prefixes
      b += tasks0 * 32 * 2;                                         // task products, their prefixes
    }
    b += T * 4ull + chunks * 128 + heavy * 12 + 8;                // tail: chunk counts, chunk sums, heavy lists
    b += T * 128ull + segs * 512ull + (own_winsum ? W * 128ull : 0);  // buckets, segment T_s and S_s
    return b + 32 * 256;  // alignment of the pieces
  }
};

// Entries (point-window pairs) from which the batch-affine rounds pay: 6.2
// products per addition against 10, but each round is a chain of launches
// around an inversion, and its sums travel through memory.  MSM with rounds /
// without on B200: 5.1e6 entries (300007 points) 2124 / 2054 us, 1.7e7 (2^20)
// 4148 / 4496 us, 4.3e5 (2^14) 1042 / 766 us.
constexpr uint64_t kRoundsMinEntries = 1ull << 23;

MsmLayout msm_layout(uint64_t n, uint32_t jobs, int c_override, int device = -1) {
  MsmLayout l;
  if (jobs == 0) jobs = 1;
  l.p = make_msm_plan((n + jobs - 1) / jobs, c_override, device);  // one window size: the mean job size's plan
  l.Wj = (uint32_t)l.p.windows;
  l.B = l.p.buckets;
  l.L = l.p.seg_len;
  const uint64_t W = (uint64_t)l.Wj * jobs;
  if (W * l.B >= (1ull << 31)) return l;
  l.W = (uint32_t)W;
  l.T = l.W * l.B;
  l.nblk = (l.T + 1023) / 1024;
  if (l.nblk > 1024u * 64u) return l;  // the three-phase scan's limit
  l.segs = l.T / l.L;
  l.E = n * (uint64_t)l.Wj;
  if (l.E >= (1ull << 32)) return l;  // entry offsets are 32-bit; pair sums < E / 2 + T < 2^32
  // rounds: enough to bring a bucket of the mean size plus a wide margin to
  // one point; anything left after them is folded by the tail kernel
  const uint64_t mean = (l.E + l.T - 1) / l.T;
  uint32_t lg = 0;
  while ((1ull << lg) < mean) lg++;
  // batch-affine rounds while buckets hold more than about four points;
  // later levels cost more in per-round latency than they save
  l.rounds = l.E < kRoundsMinEntries ? 0 : lg > 3 ? lg - 2 : 1;
  uint64_t left = l.E;  // points the tail folds, upper bound
  if (l.rounds) {
    l.jb[0] = l.E / 2 + l.T;
    l.jb[1] = l.jb[0] / 2 + l.T;
    l.tasks0 = ba_tasks_bound(l.jb[0], kFillK);
    left = l.jb[0];
    for (uint32_t r = 1; r < l.rounds; r++) left = left / 2 + l.T;
  }
  l.chunks = l.T + left / BA_TS + 1;  // bound on sum_b max(1, ceil(cnt_b / BA_TS))
  l.heavy = std::min<uint64_t>(l.T, l.chunks / (BA_TSEQ + 1)) + l.chunks / BA_HEAVY + 1;
  l.ok = true;
  return l;
}

// n: scalars (all jobs); jobs > 1: job_off (device, jobs + 1 entries) splits
// them and every job reads bases [0, nbases); the window sums of job j are
// windows [j W, (j + 1) W) of wout.
cudaError_t msm_run_impl(const fe* d_scalars, const fe* d_bases, uint64_t n, uint64_t* d_out, cudaStream_t s,
                         int c_override, uint64_t* launches, MsmWindowsOut* wout, const uint32_t* job_off,
                         uint32_t jobs) {
  uint64_t nl = 0;
  if (n == 0) {
    if (wout) {
      wout->windows = 0;
      if (launches) *launches = 0;
      return cudaSuccess;
    }
    zero_out_kernel<<<1, 32, 0, s>>>(d_out);
    if (launches) *launches = 1;
    return cudaGetLastError();
  }
  if (jobs == 0) jobs = 1;
  const MsmLayout l = msm_layout(n, jobs, c_override);
  if (!l.ok) return cudaErrorInvalidValue;
  const MsmPlan& p = l.p;
  if (wout) {
    if ((uint32_t)p.windows > MSM_MAX_WINDOWS || !wout->d_winsum) return cudaErrorInvalidValue;
    wout->windows = (uint32_t)p.windows;
    wout->c = (uint32_t)p.c;
  }
  const uint32_t Wj = l.Wj, B = l.B, L = l.L, W = l.W, T = l.T, nblk = l.nblk, segs = l.segs;
  const uint64_t entries = l.E;
  uint32_t *counts = nullptr, *offsets = nullptr, *cursor = nullptr, *bsums = nullptr, *list = nullptr;
  uint32_t *cnt = nullptr, *cprev = nullptr, *np = nullptr, *joff[2] = {nullptr, nullptr};
  fe *fin = nullptr, *buf[2] = {nullptr, nullptr}, *pre = nullptr, *tot = nullptr, *tpre = nullptr;
  fe *buckets = nullptr, *segres = nullptr, *segsum = nullptr, *winsum = nullptr;
  fe* chunk_res = nullptr;
  uint32_t *nch = nullptr, *heavy_b = nullptr, *heavy_count = nullptr;
  uint2* heavy = nullptr;
  // one allocation, cut into aligned pieces
  char* arena = nullptr;
  const uint64_t arena_bytes = l.bytes(!wout);
  uint64_t used = 0;
  cudaError_t e = zk::dmalloc((void**)&arena, arena_bytes, s);
  auto alloc = [&](void** ptr, size_t bytes) {
    *ptr = arena + used;
    used += (bytes + 255) & ~(uint64_t)255;
    if (e == cudaSuccess && used > arena_bytes) e = cudaErrorInvalidValue;
  };
  alloc((void**)&counts, T * 4ull);
  alloc((void**)&offsets, (T + 1ull) * 4);
  alloc((void**)&cursor, T * 4ull);
  alloc((void**)&bsums, (nblk + 1ull) * 4);
  alloc((void**)&list, entries * 4ull);
  alloc((void**)&joff[0], (T + 1ull) * 4);
  if (l.rounds) {
    alloc((void**)&cnt, T * 4ull);
    alloc((void**)&cprev, T * 4ull);
    alloc((void**)&np, T * 4ull);
    alloc((void**)&joff[1], (T + 1ull) * 4);
    alloc((void**)&fin, T * 64ull);
    alloc((void**)&buf[0], l.jb[0] * 64);
    if (l.rounds > 1) alloc((void**)&buf[1], l.jb[1] * 64);
    alloc((void**)&pre, l.jb[0] * 32);
    alloc((void**)&tot, l.tasks0 * 32);
    alloc((void**)&tpre, l.tasks0 * 32);
  }
  alloc((void**)&nch, T * 4ull);
  alloc((void**)&heavy, l.heavy * 8);
  alloc((void**)&heavy_b, l.heavy * 4);
  alloc((void**)&heavy_count, 8);
  alloc((void**)&chunk_res, l.chunks * 128);
  alloc((void**)&buckets, T * 128ull);
  alloc((void**)&segres, segs * 256ull);  // one level and the next
  alloc((void**)&segsum, segs * 256ull);
  if (wout)
    winsum = wout->d_winsum;  // caller's buffer, left for the host's Horner step
  else
    alloc((void**)&winsum, W * 128ull);
  if (e == cudaSuccess) {
    const double nd = (double)n;
    const int sms = sm_count();
    const uint32_t fill_k = kFillK;  // matches the task buffers' bound (layout)
    cudaMemsetAsync(counts, 0, T * 4ull, s);
    const unsigned g = (unsigned)((n + 255) / 256);
    const unsigned gb = (T + 255) / 256;
    {
      ProfScope ps("msm_count", s, nd, nd * 32);
      msm_count_kernel<<<g, 256, 0, s>>>(d_scalars, n, (uint32_t)p.c, Wj, counts, job_off, jobs);
    }
    scan_block_kernel<<<nblk, 1024, 0, s>>>(counts, offsets, bsums, T);
    scan_sums_kernel<<<1, 1024, 0, s>>>(bsums, nblk, offsets + T);
    scan_add_kernel<<<nblk, 1024, 0, s>>>(offsets, cursor, bsums, T);
    {
      ProfScope ps("msm_scatter", s, nd, nd * 32 + (double)entries * 4);
      msm_scatter_kernel<<<g, 256, 0, s>>>(d_scalars, n, (uint32_t)p.c, Wj, cursor, list, job_off, jobs);
    }
    nl += 5;
    {
      // convention: 6 Fq products per point-window (the batch-affine cost);
      // algorithmic bytes: each entry's index and signed base read once
      ProfScope ps("msm_bucket", s, (double)entries * 6, (double)entries * 68);
      if (l.rounds) {
        ba_setup_kernel<<<gb, 256, 0, s>>>(counts, offsets, list, d_bases, cnt, fin, T);
        nl++;
      }
      uint64_t jb = l.jb[0];
      for (uint32_t r = 0; r < l.rounds; r++) {
        const bool first = r == 0;
        uint32_t* jo = joff[r & 1];
        const uint32_t* in_off = first ? offsets : joff[(r + 1) & 1];
        const fe* src = first ? d_bases : buf[(r + 1) & 1];
        fe* dst = buf[r & 1];
        ba_jobs_kernel<<<gb, 256, 0, s>>>(cnt, cprev, np, T);
        scan_block_kernel<<<nblk, 1024, 0, s>>>(np, jo, bsums, T);
        scan_sums_kernel<<<1, 1024, 0, s>>>(bsums, nblk, jo + T);
        scan_add_kernel<<<nblk, 1024, 0, s>>>(jo, cursor, bsums, T);
        // inversion threads: enough to fill the GPU (fill groups), each group
        // at most BA_G task products; the grid covers the one-task groups of
        // a small round
        const uint64_t tasks = ba_tasks_bound(jb, fill_k);
        const uint32_t fill = (uint32_t)sms * 32;
        const unsigned gt = (unsigned)std::min<uint64_t>((tasks + 255) / 256, (uint64_t)sms * 6);
        const unsigned ga = (unsigned)std::min<uint64_t>((tasks + BA_APPLY - 1) / BA_APPLY, (uint64_t)sms * 10);
        const uint64_t groups = tasks < fill ? tasks : std::max<uint64_t>(2ull * fill, tasks / BA_G + 1);
        const unsigned gi = (unsigned)std::min<uint64_t>((groups + 127) / 128, (uint64_t)sms * 8);
        if (first)
          ba_prefix_kernel<true><<<gt, 256, kPrefixSmem, s>>>(src, list, in_off, cprev, jo, T, pre, tot, fill_k);
        else
          ba_prefix_kernel<false><<<gt, 256, kPrefixSmem, s>>>(src, list, in_off, cprev, jo, T, pre, tot, fill_k);
        ba_invert_kernel<<<gi, 128, 0, s>>>(tot, tpre, jo, T, fill, fill_k);
        if (first)
          ba_apply_kernel<true><<<ga, BA_APPLY, kApplySmem, s>>>(src, list, in_off, cprev, jo, T, pre, tot, dst, fin,
                                                            cnt, fill_k);
        else
          ba_apply_kernel<false><<<ga, BA_APPLY, kApplySmem, s>>>(src, list, in_off, cprev, jo, T, pre, tot, dst, fin,
                                                             cnt, fill_k);
        nl += 7;
        jb = jb / 2 + T;
      }
      // tail: chunk counts -> scan (offsets in the joff not in use) -> folds -> bucket sums
      const uint32_t last = (l.rounds - 1) & 1;
      uint32_t* coff = l.rounds ? joff[last ^ 1] : joff[0];
      const uint32_t* left = l.rounds ? cnt : counts;
      ba_chunks_kernel<<<gb, 256, 0, s>>>(left, nch, T);
      scan_block_kernel<<<nblk, 1024, 0, s>>>(nch, coff, bsums, T);
      scan_sums_kernel<<<1, 1024, 0, s>>>(bsums, nblk, coff + T);
      scan_add_kernel<<<nblk, 1024, 0, s>>>(coff, cursor, bsums, T);
      cudaMemsetAsync(heavy_count, 0, 8, s);
      const unsigned gf = (unsigned)std::min<uint64_t>((l.chunks + 255) / 256, (uint64_t)sms * 16);
      if (l.rounds)
        ba_fold_kernel<false><<<gf, 256, 0, s>>>(cnt, joff[last], buf[last], nullptr, fin, coff, T, chunk_res);
      else
        ba_fold_kernel<true><<<gf, 256, 0, s>>>(counts, offsets, d_bases, list, nullptr, coff, T, chunk_res);
      ba_bucket_sum_kernel<<<(T + 31) / 32, 128, 0, s>>>(coff, chunk_res, buckets, heavy, heavy_b, heavy_count, T);
      const unsigned gh = (unsigned)std::min<uint64_t>(l.heavy, (uint64_t)sms * 2);
      ba_heavy_items_kernel<<<gh, 256, 0, s>>>(coff, chunk_res, heavy, heavy_count);
      ba_heavy_kernel<<<gh, 256, 0, s>>>(coff, chunk_res, buckets, heavy_b, heavy_count);
      nl += 8;
    }
    {
      ProfScope ps("msm_segment", s, (double)T * 2 * 14, T * 128.0);
      msm_segment_kernel<<<(segs + 31) / 32, 128, 0, s>>>(buckets, segres, segsum, B, L, segs);
    }
    uint32_t S = B / L, len = L;  // segments per window, buckets per segment
    fe *it = segres, *is = segsum, *ot = segres + 4ull * segs, *os = segsum + 4ull * segs;
    for (; S > kGroup; S /= kGroup, len *= kGroup) {
      msm_group_kernel<<<W * (S / kGroup), 4 * kGroup, 0, s>>>(it, is, ot, os, kGroup, len);
      std::swap(it, ot);
      std::swap(is, os);
      nl++;
    }
    msm_group_kernel<<<W, 4 * S, 0, s>>>(it, is, winsum, nullptr, S, len);
    nl += 2;
    e = cudaGetLastError();
    if (!wout && e == cudaSuccess) {
      e = msm_combine(winsum, W, (uint32_t)p.c, d_out, s);
      nl++;
    }
  }
  if (arena) cudaFreeAsync(arena, s);
  if (launches) *launches = nl;
  return e;
}
}  // namespace

uint64_t msm_scratch_bytes(uint64_t n_total, uint32_t jobs, bool own_winsum, int device) {
  if (n_total == 0) return 256;
  const MsmLayout l = msm_layout(n_total, jobs, 0, device);
  if (!l.ok) return ~0ull >> 2;
  return l.bytes(own_winsum);
}

cudaError_t msm_run(const fe* d_scalars, const fe* d_bases, uint64_t n, uint64_t* d_out, cudaStream_t s,
                    int c_override, uint64_t* launches, MsmWindowsOut* wout) {
  return msm_run_impl(d_scalars, d_bases, n, d_out, s, c_override, launches, wout, nullptr, 1);
}

cudaError_t msm_run_multi(const fe* d_scalars, const fe* d_bases, const uint32_t* d_job_off, uint32_t jobs,
                          uint64_t n_total, cudaStream_t s, uint64_t* launches, MsmWindowsOut* wout) {
  if (!wout || !wout->d_winsum || jobs == 0 || !d_job_off || n_total >= (1ull << 32)) return cudaErrorInvalidValue;
  return msm_run_impl(d_scalars, d_bases, n_total, nullptr, s, 0, launches, wout, d_job_off, jobs);
}

}  // namespace zk
