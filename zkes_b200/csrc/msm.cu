// Pippenger multi-scalar multiplication over BN254 G1, for one row or for many rows that share
// the bases (the d_x / d_y loops of kzh2.rs:653-660, kzh3.rs:680-687,743-750).
//
//   1. k_msm_bits     largest magnitude of the sign-folded scalars -> window width W, windows K
//   2. k_msm_digits   signed W-bit digits; MODE 0 counts (row, window, bucket) keys, MODE 1
//                     scatters point indices (sign in bit 31) to their bucket's slots.  Full-width scalars are split
//                     into two halves by the curve's endomorphism (glv.cuh): the images of the bases (bit 30) are points of
//                     their own, and there are half the windows.  Many rows of them share one set of buckets over all
//                     windows (k_multiples): no step 6
//   3. k_msm_accumulate  equal chunks of the sorted entry list are summed by one thread each with
//                     mixed additions; a bucket inside one chunk is written directly, pieces of
//                     buckets that cross chunk borders go to per-chunk head / tail slots
//   4. k_msm_fixup    buckets that span chunks: tail of the first chunk + heads of the others
//   5. k_msm_bucket_reduce  sum_j (j+1) B_j per (row, window) by running sums per thread,
//                     a small scalar multiple for the thread's offset, then a block tree
//   6. k_msm_combine  Horner over the windows (W doublings each), Jacobian out
// Small scalars (quantised int8 / int16 weights and activations, negatives stored as r - |v|)
// fold to a few bits, so they use one narrow window: no doublings, few buckets.
#include "msm.hpp"
#include "msm_plan.hpp"

#include <algorithm>
#include "reduce.cuh"
#include "batch_affine.cuh"
#include "quad.cuh"
#include "glv.cuh"

namespace zk {
namespace {

__device__ __forceinline__ Fr ld_scalar(const Fr* p) {
  const uint4 lo = __ldg(reinterpret_cast<const uint4*>(p));
  const uint4 hi = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  return fr_from_chunks(lo, hi);
}

// Canonical value of a Montgomery-form scalar, folded to min(s, r - s); returns the sign.
__device__ __forceinline__ bool fold_scalar(const Fr& mont, uint32_t (&mag)[8]) {
  const Fr c = from_mont(mont);
  uint32_t m[8], d[8];
#pragma unroll
  for (int i = 0; i < 8; i++) m[i] = FrParams::mod(i);
  (void)sub8(d, m, c.v);  // r - s
  // s > r - s  <=>  borrow when computing (r - s) - s
  uint32_t t[8];
  const bool negv = sub8(t, d, c.v) != 0 && !c.is_zero();
#pragma unroll
  for (int i = 0; i < 8; i++) mag[i] = negv ? d[i] : c.v[i];
  return negv;
}

__device__ __forceinline__ int bit_length(const uint32_t (&mag)[8]) {
  int bits = 0;
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (mag[i]) bits = 32 * i + (32 - __clz(mag[i]));
  return bits;
}

// Scalars whose folded magnitude is below 2^30 also have a compact form: a signed 32-bit integer.
// When every scalar of a call has one (quantised weights and activations), the digit passes read
// these 4 bytes instead of converting the 32-byte Montgomery value again.
constexpr int32_t kNotCompact = INT32_MIN;

// bits: largest bit length; among the scalars below 2^32 mag: largest magnitude, span: largest of v and
// -v - 1, whose bit length is that of the two's complement form without its sign.  nonzero: how many are not zero.
struct MsmBits {
  unsigned int bits, mag, span, pad;
  unsigned long long nonzero;
};
__global__ void k_msm_bits(const Fr* __restrict__ scalars, uint64_t total, MsmBits* found, int32_t* compact) {
  __shared__ unsigned int s_found[4];
  if (threadIdx.x < 4) s_found[threadIdx.x] = 0;
  __syncthreads();
  int best = 0;
  uint32_t nonzero = 0;
  uint32_t best_mag = 0, best_span = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t mag[8];
    const bool negv = fold_scalar(ld_scalar(scalars + i), mag);
    const int b = bit_length(mag);
    best = b > best ? b : best;
    nonzero += b != 0;
    if (b <= 32) {
      best_mag = mag[0] > best_mag ? mag[0] : best_mag;
      const uint32_t span = negv && mag[0] ? mag[0] - 1 : mag[0];
      best_span = span > best_span ? span : best_span;
    }
    if (compact) compact[i] = b <= kCompactBits ? (negv ? -(int32_t)mag[0] : (int32_t)mag[0]) : kNotCompact;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const int o = __shfl_down_sync(0xffffffffu, best, off);
    best = o > best ? o : best;
    const uint32_t m = __shfl_down_sync(0xffffffffu, best_mag, off);
    best_mag = m > best_mag ? m : best_mag;
    const uint32_t p = __shfl_down_sync(0xffffffffu, best_span, off);
    best_span = p > best_span ? p : best_span;
    nonzero += __shfl_down_sync(0xffffffffu, nonzero, off);
  }
  // one set of global atomics a block: with one a warp they were a third of the time of a small call's pass
  if ((threadIdx.x & 31) == 0 && best) {
    atomicMax(&s_found[0], (unsigned int)best);
    atomicMax(&s_found[1], best_mag);
    atomicMax(&s_found[2], best_span);
    atomicAdd(&s_found[3], nonzero);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_found[0]) {
    atomicMax(&found->bits, s_found[0]);
    atomicMax(&found->mag, s_found[1]);
    atomicMax(&found->span, s_found[2]);
    atomicAdd(&found->nonzero, (unsigned long long)s_found[3]);
  }
}

// Folded magnitude and sign of scalar g, from the compact form when the call has one.
template <bool COMPACT>
__device__ __forceinline__ bool load_mag(const Fr* __restrict__ scalars, const int32_t* __restrict__ compact, uint64_t g,
                                         uint32_t (&mag)[8]) {
  if (COMPACT) {
    const int32_t v = __ldg(compact + g);
#pragma unroll
    for (int i = 1; i < 8; i++) mag[i] = 0;
    mag[0] = v < 0 ? (uint32_t)(-v) : (uint32_t)v;
    return v < 0;
  } else {
    return fold_scalar(ld_scalar(scalars + g), mag);
  }
}

// W-bit field of mag starting at bit `pos` (pos + W may run past its end: zeros).
template <int N>
__device__ __forceinline__ uint32_t bit_field(const uint32_t (&mag)[N], int pos, int w) {
  const int limb = pos >> 5, sh = pos & 31;
  uint64_t v = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    if (i == limb) v |= (uint64_t)mag[i];
    if (i == limb + 1) v |= (uint64_t)mag[i] << 32;
  }
  return (uint32_t)(v >> sh) & ((1u << w) - 1u);
}

// An entry of a bucket: the point's index, kEntryEndo for its image under the endomorphism, kEntryNeg for the negative.
constexpr uint32_t kEntryNeg = 0x80000000u, kEntryEndo = 0x40000000u;

// The signed digits of one magnitude that are not zero: use(window, |digit| - 1, digit negative).
template <int N, class F>
__device__ __forceinline__ void signed_digits(const uint32_t (&mag)[N], int w, int k_windows, F use) {
  const uint32_t half = 1u << (w - 1);
  uint32_t carry = 0;
  for (int k = 0; k < k_windows; k++) {
    uint32_t raw = bit_field(mag, k * w, w) + carry;
    bool dneg = false;
    if (raw > half) {
      raw = (1u << w) - raw;
      dneg = true;
      carry = 1;
    } else {
      carry = 0;
    }
    if (raw) use((uint32_t)k, raw - 1, dneg);
  }
}

enum ScalarForm : int {
  kWide = 0,      // folded to a sign and a magnitude
  kCompact = 1,   // the same from the compact form of small scalars
  kEndo = 2       // split into two halves by the endomorphism
};

// The digits of scalar g: use(window, bucket of the window, flags of the entry).
template <int FORM, class F>
__device__ __forceinline__ void scalar_digits(const Fr* __restrict__ scalars, const int32_t* __restrict__ compact, uint64_t g, int w, int k_windows,
                                              F use) {
  uint32_t mag[8];
  const bool negv = load_mag<FORM == kCompact>(scalars, compact, g, mag);
  if constexpr (FORM == kEndo) {
    uint32_t m[2][4];
    bool n[2];
    glv_split(mag, m[0], &n[0], m[1], &n[1]);
#pragma unroll 1
    for (int e = 0; e < 2; e++) {
      uint32_t part[4];
#pragma unroll
      for (int i = 0; i < 4; i++) part[i] = e ? m[1][i] : m[0][i];
      const bool neg = negv != (e ? n[1] : n[0]);
      signed_digits(part, w, k_windows, [&](uint32_t k, uint32_t d, bool dneg) { use(k, d, (neg != dneg ? kEntryNeg : 0u) | (e ? kEntryEndo : 0u)); });
    }
  } else {
    signed_digits(mag, w, k_windows, [&](uint32_t k, uint32_t d, bool dneg) { use(k, d, negv != dneg ? kEntryNeg : 0u); });
  }
}

// table_step: not 0 where the windows of a row share its buckets, window k taking its points from `table_step` k on (k_multiples).
template <int MODE, int FORM>  // MODE 0: count keys, 1: scatter entries
__global__ void k_msm_digits(const Fr* __restrict__ scalars, const int32_t* __restrict__ compact,
                             const uint32_t* __restrict__ row_ids, uint64_t n, uint32_t rows,
                             int w, int k_windows, uint32_t table_step, uint32_t* counts_or_cursor, uint32_t* entries) {
  const uint64_t total = row_ids ? n : n * rows;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x) {
    // dense rows: scalar g belongs to row g / n; listed rows: the caller names the row of every scalar
    const uint32_t row = row_ids ? row_ids[g] : (uint32_t)(g / n);
    const uint32_t col = row_ids ? (uint32_t)g : (uint32_t)(g - (uint64_t)row * n);
    scalar_digits<FORM>(scalars, compact, g, w, k_windows, [&](uint32_t k, uint32_t digit, uint32_t flags) {
      const uint32_t key = ((table_step ? row : row * (uint32_t)k_windows + k) << (w - 1)) + digit;
      if (MODE == 0) {
        atomicAdd(counts_or_cursor + key, 1u);
      } else {
        const uint32_t slot = atomicAdd(counts_or_cursor + key, 1u);
        entries[slot] = (col + k * table_step) | flags;
      }
    });
  }
}

// Same two passes for a small key space (at most kSmallKeys buckets in total): keys are counted in
// shared memory first, so the global counters see one atomic per (block, bucket) instead of
// one per digit.  In scatter mode the block reserves a contiguous range per bucket.
constexpr uint32_t kSmallKeys = 4096;

template <int MODE, int FORM>
__global__ void __launch_bounds__(256) k_msm_digits_small(const Fr* __restrict__ scalars, const int32_t* __restrict__ compact,
                                                          const uint32_t* __restrict__ row_ids,
                                                          uint64_t n, uint32_t rows, int w, int k_windows, uint32_t table_step,
                                                          uint32_t n_keys, uint64_t per_block, uint32_t* counts_or_cursor, uint32_t* entries) {
  __shared__ uint32_t hist[kSmallKeys];
  __shared__ uint32_t basepos[kSmallKeys];
  const uint64_t total = row_ids ? n : n * rows;
  const uint64_t begin = (uint64_t)blockIdx.x * per_block;
  const uint64_t end = begin + per_block < total ? begin + per_block : total;
  for (uint32_t k = threadIdx.x; k < n_keys; k += blockDim.x) hist[k] = 0;
  __syncthreads();
  for (int pass = 0; pass < (MODE == 0 ? 1 : 2); pass++) {
    for (uint64_t g = begin + threadIdx.x; g < end; g += blockDim.x) {
      const uint32_t row = row_ids ? row_ids[g] : (uint32_t)(g / n);
      const uint32_t col = row_ids ? (uint32_t)g : (uint32_t)(g - (uint64_t)row * n);
      scalar_digits<FORM>(scalars, compact, g, w, k_windows, [&](uint32_t k, uint32_t digit, uint32_t flags) {
        const uint32_t key = ((table_step ? row : row * (uint32_t)k_windows + k) << (w - 1)) + digit;
        if (pass == 0) {
          atomicAdd(hist + key, 1u);
        } else {
          const uint32_t slot = basepos[key] + atomicAdd(hist + key, 1u);
          entries[slot] = (col + k * table_step) | flags;
        }
      });
    }
    __syncthreads();
    if (pass == 0) {
      for (uint32_t k = threadIdx.x; k < n_keys; k += blockDim.x) {
        const uint32_t c = hist[k];
        if (MODE == 0) {
          if (c) atomicAdd(counts_or_cursor + k, c);
        } else {
          basepos[k] = c ? atomicAdd(counts_or_cursor + k, c) : 0;
          hist[k] = 0;
        }
      }
      __syncthreads();
    }
  }
}

__device__ __forceinline__ Fq ld_fq(const Fq* p) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  Fq r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}
__device__ __forceinline__ void st_fq(Fq* p, const Fq& x) {
  reinterpret_cast<uint4*>(p)[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  reinterpret_cast<uint4*>(p)[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

// Many rows over the same bases: the multiples 2^(w k) of every base for all windows k, so that the digits of all windows of a row
// fall into one set of buckets: the windows can be wider, there is one bucket sum per row instead of one per row and window, and no
// Horner chain.  The chain of w (windows - 1) doublings is here instead, once per base; four lanes take a point (quad.cuh).
// A latency chain (226 us for a hundred points, 555 for 2^14), beside the passes over the digits.  A KZH3 commitment and opening of
// 2^22 values, half of them full width: accumulation 15 957 -> 13 315 us, bucket reduction 2 685 -> 1 327, Horner chains 1 120 -> 0, for
// 935 us of multiples; 24 286 -> 19 108 us in all together with the split.  (Counting the buckets of a row in shared
// memory instead of by global atomics made no difference.)
__global__ void __launch_bounds__(128) k_multiples(const Affine* __restrict__ bases, uint64_t n, int w, int k_windows, Xyzz* out) {
  const uint64_t i = (uint64_t)blockIdx.x * 32 + (threadIdx.x >> 2);
  const int role = threadIdx.x & 3;
  const uint64_t at = i < n ? i : n - 1;
  const Fq bx = ld_fq(&bases[at].x), by = ld_fq(&bases[at].y);
  QuadXyzz p;
  p.x = bx;
  p.y = by;
  p.z = bx.is_zero() && by.is_zero() ? Fq::zero() : Fq::one();
  if (i < n) quad_store(out + i, p, role);
#pragma unroll 1
  for (int k = 1; k < k_windows; k++) {
#pragma unroll 1
    for (int j = 0; j < w; j++) p = quad_dbl(p, role);
    if (i < n) quad_store(out + (uint64_t)k * n + i, p, role);
  }
}

// Affine form of many points, kMultiplesPer a thread and inversion, and the x of their images under the endomorphism.
constexpr int kMultiplesPer = 4;
__global__ void __launch_bounds__(kBatchThreads, 4) k_multiples_affine(const Xyzz* __restrict__ points, uint64_t n, Affine* out, Fq* images) {
  constexpr int kPer = kMultiplesPer;
  __shared__ Fq sh[kBatchThreads];
  const uint64_t t0 = (uint64_t)blockIdx.x * (kBatchThreads * kPer) + threadIdx.x;
  Fq pre[kPer], run = Fq::one(), beta;
#pragma unroll
  for (int i = 0; i < 8; i++) beta.v[i] = Glv::beta(i);
#pragma unroll 1
  for (int j = 0; j < kPer; j++) {
    const uint64_t t = t0 + (uint64_t)j * kBatchThreads;
    if (t >= n) break;
    const Fq z = ld_fq(&points[t].zzz);
    pre[j] = run;
    if (!z.is_zero()) run = fq_mul_fn(run, z);
  }
  Fq inv = block_inverse(run, sh);
#pragma unroll 1
  for (int j = kPer - 1; j >= 0; j--) {
    const uint64_t t = t0 + (uint64_t)j * kBatchThreads;
    if (t >= n) continue;
    const Fq zzz = ld_fq(&points[t].zzz);
    Fq x = Fq::zero(), y = Fq::zero();
    if (!zzz.is_zero()) {
      const Fq izzz = fq_mul_fn(inv, pre[j]);
      inv = fq_mul_fn(inv, zzz);
      const Fq iz = fq_mul_fn(izzz, ld_fq(&points[t].zz));  // 1 / zz = (zz / zzz)^2
      x = fq_mul_fn(ld_fq(&points[t].x), fq_mul_fn(iz, iz));
      y = fq_mul_fn(ld_fq(&points[t].y), izzz);
    }
    st_fq(&out[t].x, x);
    st_fq(&out[t].y, y);
    st_fq(images + t, fq_mul_fn(beta, x));
  }
}

// images[i] = beta x of base i: the x of its image under the endomorphism (y is its own)
__global__ void __launch_bounds__(256) k_endo_images(const Affine* __restrict__ bases, uint64_t n, Fq* images) {
  Fq beta;
#pragma unroll
  for (int i = 0; i < 8; i++) beta.v[i] = Glv::beta(i);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    st_fq(images + i, mul(beta, ld_fq(&bases[i].x)));
}

__device__ __forceinline__ Affine ld_affine(const Affine* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  const uint4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2), d = __ldg(q + 3);
  Affine r;
  r.x.v[0] = a.x; r.x.v[1] = a.y; r.x.v[2] = a.z; r.x.v[3] = a.w;
  r.x.v[4] = b.x; r.x.v[5] = b.y; r.x.v[6] = b.z; r.x.v[7] = b.w;
  r.y.v[0] = c.x; r.y.v[1] = c.y; r.y.v[2] = c.z; r.y.v[3] = c.w;
  r.y.v[4] = d.x; r.y.v[5] = d.y; r.y.v[6] = d.z; r.y.v[7] = d.w;
  return r;
}

__device__ __forceinline__ void st_xyzz(Xyzz* p, const Xyzz& v) {
  uint4* q = reinterpret_cast<uint4*>(p);
  const Fq* f[4] = {&v.x, &v.y, &v.zz, &v.zzz};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    q[2 * i] = make_uint4(f[i]->v[0], f[i]->v[1], f[i]->v[2], f[i]->v[3]);
    q[2 * i + 1] = make_uint4(f[i]->v[4], f[i]->v[5], f[i]->v[6], f[i]->v[7]);
  }
}
__device__ __forceinline__ Xyzz ld_xyzz(const Xyzz* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  Xyzz v;
  Fq* f[4] = {&v.x, &v.y, &v.zz, &v.zzz};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 a = q[2 * i], b = q[2 * i + 1];
    f[i]->v[0] = a.x; f[i]->v[1] = a.y; f[i]->v[2] = a.z; f[i]->v[3] = a.w;
    f[i]->v[4] = b.x; f[i]->v[5] = b.y; f[i]->v[6] = b.z; f[i]->v[7] = b.w;
  }
  return v;
}

// First bucket whose range ends after entry e: smallest b with offsets[b + 1] > e.
__device__ __forceinline__ uint32_t bucket_of(const uint32_t* __restrict__ offsets, uint32_t n_buckets, uint32_t e) {
  uint32_t lo = 0, hi = n_buckets - 1;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (offsets[mid + 1] > e) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// The mixed addition with its ten products as calls of one shared routine, for the kernels that hold other additions
// besides.  The kernels whose loop is the addition alone (k_msm_accumulate, k_rows_sums) inline it: with the product at some
// 185 instructions the loop body fits the instruction cache, and the calls' register moves cost 2.5 to 4 % (2 809 us against
// 2 739 us for 2^24 entries, 1 820 against 1 740 us for 11.2 M table additions).
__device__ __noinline__ Fq fq_mul_call(const Fq a, const Fq b) { return mul(a, b); }
__device__ __noinline__ Fq fq_sqr_call(const Fq a) { return sqr(a); }

__device__ __forceinline__ Xyzz add_mixed_calls(const Xyzz& p, const Affine& q) {
  if (q.is_inf()) return p;
  if (p.is_inf()) return Xyzz::from_affine(q);
  const Fq u2 = fq_mul_call(q.x, p.zz), s2 = fq_mul_call(q.y, p.zzz);
  const Fq pp_ = sub(u2, p.x), r_ = sub(s2, p.y);
  if (pp_.is_zero()) {
    if (!r_.is_zero()) return Xyzz::inf();
    Xyzz d;
    dbl_affine_rare(&d, &q);
    return d;
  }
  Xyzz r;
  const Fq pp = fq_sqr_call(pp_), ppp = fq_mul_call(pp_, pp), q_ = fq_mul_call(p.x, pp);
  r.x = sub(sub(fq_sqr_call(r_), ppp), dbl(q_));
  r.y = sub(fq_mul_call(r_, sub(q_, r.x)), fq_mul_call(p.y, ppp));
  r.zz = fq_mul_call(p.zz, pp);
  r.zzz = fq_mul_call(p.zzz, ppp);
  return r;
}

__global__ void __launch_bounds__(128, kAccBlocks) k_msm_accumulate(const Affine* __restrict__ bases,
                                                        const Fq* __restrict__ images, const uint32_t* __restrict__ gather,
                                                        const uint32_t* __restrict__ entries,
                                                        const uint32_t* __restrict__ offsets, uint32_t n_buckets,
                                                        uint32_t n_entries, uint32_t seg, uint32_t n_chunks,
                                                        Xyzz* bucket_sums, Xyzz* heads, Xyzz* tails) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_chunks) return;
  const uint32_t begin = c * seg;
  const uint32_t end = (begin + seg < n_entries) ? begin + seg : n_entries;
  uint32_t b = bucket_of(offsets, n_buckets, begin);
  uint32_t b_end = offsets[b + 1];
  bool began_before = offsets[b] < begin;  // the current bucket started in an earlier chunk
  Xyzz acc = Xyzz::inf();
  for (uint32_t e = begin; e < end; e++) {
    if (e == b_end) {  // bucket b is complete
      if (began_before) st_xyzz(heads + c, acc); else st_xyzz(bucket_sums + b, acc);
      acc = Xyzz::inf();
      began_before = false;
      do { b++; b_end = offsets[b + 1]; } while (b_end <= e);
    }
    const uint32_t ent = entries[e];
    Affine pt;
    if (images) {
      const uint32_t col = ent & ~(kEntryNeg | kEntryEndo);
      pt.x = ld_fq((ent & kEntryEndo) ? images + col : &bases[col].x);
      pt.y = ld_fq(&bases[col].y);
    } else {
      const uint32_t col = ent & ~kEntryNeg;
      pt = ld_affine(bases + (gather ? gather[col] : col));
    }
    if (ent & kEntryNeg) pt = neg(pt);
    acc = add_mixed(acc, pt);
  }
  // the bucket in progress at the end of the chunk
  const bool continues = b_end > end;
  if (began_before)
    st_xyzz(heads + c, acc);            // spans the whole chunk, or ends exactly at its end
  else if (continues)
    st_xyzz(tails + c, acc);
  else
    st_xyzz(bucket_sums + b, acc);
}

constexpr uint32_t kFewPieces = 8, kManyPieces = 24;
constexpr int kFixupThreads = 256;

// One thread per bucket: buckets cut into at most `few` pieces are summed in place.  The others are listed for k_msm_fixup, those of
// more than kManyPieces from the front of `list`, the rest from its end (listed[0] and listed[1] of them).
// few is kManyPieces where there are more buckets of that kind than k_msm_fixup has warps (k_total64 counts them): a chain of that
// many additions a thread is then the least work.  Else it is kFewPieces: for some of them it would be the longest chain of the
// call (65536 scalars of 64 bits, whose top window has 256 buckets of sixteen pieces: 681 us against 537).
__global__ void __launch_bounds__(256) k_msm_fixup_few(const uint32_t* __restrict__ offsets, uint32_t n_buckets, uint32_t seg, uint32_t few,
                                                       Xyzz* bucket_sums, const Xyzz* heads, const Xyzz* tails,
                                                       uint32_t* list, uint32_t* listed) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_buckets) return;
  const uint32_t s = offsets[b], e = offsets[b + 1];
  if (e <= s) return;
  const uint32_t c0 = s / seg, c1 = (e - 1) / seg;
  if (c0 == c1) return;
  if (c1 - c0 >= few) {
    if (c1 - c0 >= kManyPieces)
      list[atomicAdd(listed, 1u)] = b;
    else
      list[n_buckets - 1 - atomicAdd(listed + 1, 1u)] = b;
    return;
  }
  Xyzz acc = ld_xyzz(tails + c0);
  for (uint32_t c = c0 + 1; c <= c1; c++) acc = add(acc, ld_xyzz(heads + c));  // one call site: inlined
  st_xyzz(bucket_sums + b, acc);
}

// sh[0] = sh[0] + ... + sh[n - 1] for a power of two n of at most twice the block: a thread per addition while there are
// enough of them, four lanes per addition for the last levels.  The whole block calls it after a barrier.
__device__ __forceinline__ void tree_sum(Xyzz* sh, uint32_t n) {
  uint32_t off = n >> 1;
#pragma unroll 1
  for (; off > blockDim.x / 4; off >>= 1) {
    if (threadIdx.x < off) add_to(&sh[threadIdx.x], &sh[threadIdx.x + off]);
    __syncthreads();
  }
#pragma unroll 1
  for (; off > 0; off >>= 1) {
    const uint32_t q = threadIdx.x >> 2, i = q < off ? q : 0;
    if ((threadIdx.x & ~31u) < 4 * off) {  // whole warps
      const int role = threadIdx.x & 3;
      const QuadXyzz v = quad_add(quad_load(&sh[i], role), quad_load(&sh[i + off], role), role);
      __syncwarp();
      if (q < off) quad_store(&sh[q], v, role);
    }
    __syncthreads();
  }
}

// The listed buckets.  The time is the longest chain of dependent additions.
//   Many pieces: a bucket per block and pass.  The top window of full-width scalars has a handful of buckets that between them
//   take every point, a thousand pieces each: 256 threads leave pieces / 256 additions plus eight levels of a tree, where a warp
//   per bucket left pieces / 32 plus five (100003 full-width scalars: 490 us against 131 us).
//   Up to kManyPieces: a block each too while there are blocks for them, whose quads are quicker (4096 full-width scalars, with a
//   handful of them: 21 us of this kernel, 45 us with a warp each); else a warp each (64 rows of 16384 int8 values, 8192 buckets
//   of eight or nine pieces: the call took 1089 us with a block each, and takes 579 us with a warp or with what
//   k_msm_fixup_few keeps).
__global__ void __launch_bounds__(kFixupThreads, 2) k_msm_fixup(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ list,
                                                             const uint32_t* __restrict__ listed, uint32_t n_buckets, uint32_t seg,
                                                             Xyzz* bucket_sums, const Xyzz* heads, const Xyzz* tails) {
  __shared__ Xyzz sh[kFixupThreads];
  // pieces of a bucket: tail of chunk c0, heads of chunks c0+1 .. c1; the sum of every `step`-th of them from `first` on
  auto pieces_of = [&](uint32_t b, uint32_t* c0, uint32_t* c1) {
    const uint32_t s = offsets[b], e = offsets[b + 1];
    *c0 = s / seg;
    *c1 = (e - 1) / seg;
  };
  auto share = [&](uint32_t c0, uint32_t c1, uint32_t first, uint32_t step) {
    Xyzz acc = Xyzz::inf();
    for (uint32_t c = c0 + first; c <= c1; c += step) {
      const Xyzz h = ld_xyzz(c == c0 ? tails + c : heads + c);
      add_to(&acc, &h);
    }
    return acc;
  };
  const uint32_t n_long = listed[0], n_mid = listed[1], lane = threadIdx.x & 31;
  const uint32_t by_warps = n_mid > gridDim.x ? n_mid : 0, by_blocks = n_long + n_mid - by_warps;
  uint32_t c0, c1;
  Xyzz* mine = sh + (threadIdx.x & ~31u);
  for (uint32_t item = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; item < by_warps; item += gridDim.x * (kFixupThreads / 32)) {
    const uint32_t b = list[n_buckets - 1 - item];
    pieces_of(b, &c0, &c1);
    mine[lane] = share(c0, c1, lane, 32);
    __syncwarp();
    if (c1 - c0 >= 16 && lane < 16) add_to(&mine[lane], &mine[lane + 16]);
    __syncwarp();
#pragma unroll 1
    for (uint32_t off = 8; off > 0; off >>= 1) {
      const uint32_t q = lane >> 2, i = q < off ? q : 0;
      quad_add_to(&mine[i], &mine[i + off], q < off);
    }
    if (lane == 0) st_xyzz(bucket_sums + b, mine[0]);
    __syncwarp();
  }
  __syncthreads();
  for (uint32_t item = blockIdx.x; item < by_blocks; item += gridDim.x) {
    const uint32_t b = item < n_long ? list[item] : list[n_buckets - 1 - (item - n_long)];
    pieces_of(b, &c0, &c1);
    sh[threadIdx.x] = share(c0, c1, threadIdx.x, kFixupThreads);
    __syncthreads();
    uint32_t live = kFixupThreads;  // the shares beyond the number of pieces are infinity
    while (live > 1 && live / 2 >= c1 - c0 + 1) live >>= 1;
    tree_sum(sh, live);
    if (threadIdx.x == 0) st_xyzz(bucket_sums + b, sh[0]);
    __syncthreads();
  }
}

// Few buckets, cut into many pieces: `groups` blocks per bucket, of which those that a bucket's pieces keep busy stay (one per
// kFixupShare pieces: uniform digits give every bucket the same, but all of them may as well lie in one bucket), each leaving a
// partial sum; the block that finishes a bucket last adds the partial sums.
// turn[b] == offsets[b + 1] on entry (the cursor of the scatter) counts the blocks that are through.  2^18 int8 scalars, 99 % of
// them equal: 1299 us with a block per bucket, 408 us with up to 128 (uniform ones: 404 and 377 us).
__device__ __forceinline__ Xyzz ld_partial(const Xyzz* p) {  // written by another block of this launch: past the L1 cache
  const uint4* q = reinterpret_cast<const uint4*>(p);
  Xyzz v;
  Fq* f[4] = {&v.x, &v.y, &v.zz, &v.zzz};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint4 a = __ldcg(q + 2 * i), b = __ldcg(q + 2 * i + 1);
    f[i]->v[0] = a.x; f[i]->v[1] = a.y; f[i]->v[2] = a.z; f[i]->v[3] = a.w;
    f[i]->v[4] = b.x; f[i]->v[5] = b.y; f[i]->v[6] = b.z; f[i]->v[7] = b.w;
  }
  return v;
}
__global__ void __launch_bounds__(128) k_msm_fixup_block(const uint32_t* __restrict__ offsets, uint32_t seg, uint32_t groups, uint32_t* turn,
                                                         Xyzz* bucket_sums, const Xyzz* heads, const Xyzz* tails, Xyzz* partial) {
  __shared__ Xyzz sh[128];
  __shared__ bool last;
  const uint32_t b = blockIdx.x, g = blockIdx.y;
  const uint32_t s = offsets[b], e = offsets[b + 1];
  if (e <= s) return;
  const uint32_t c0 = s / seg, c1 = (e - 1) / seg;
  if (c0 == c1) return;  // the accumulation wrote this bucket directly
  const uint32_t want = (c1 - c0) / kFixupShare + 1, share = want < groups ? want : groups;
  if (g >= share) return;
  // pieces: tail of chunk c0, heads of chunks c0+1 .. c1
  Xyzz acc = Xyzz::inf();
  for (uint32_t c = c0 + g + share * threadIdx.x; c <= c1; c += share * blockDim.x) {
    const Xyzz h = ld_xyzz(c == c0 ? tails + c : heads + c);
    add_to(&acc, &h);
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  uint32_t live = 128;  // the shares beyond the number of pieces are infinity
  while (live > 1 && live / 2 >= (c1 - c0) / share + 1) live >>= 1;
  tree_sum(sh, live);
  if (share > 1) {
    if (threadIdx.x == 0) {
      st_xyzz(partial + (size_t)b * groups + g, sh[0]);
      __threadfence();
      last = atomicAdd(turn + b, 1u) == e + share - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < kFixupGroups) sh[threadIdx.x] = threadIdx.x < share ? ld_partial(partial + (size_t)b * groups + threadIdx.x) : Xyzz::inf();
    __syncthreads();
    tree_sum(sh, kFixupGroups);
  }
  if (threadIdx.x == 0) st_xyzz(bucket_sums + b, sh[0]);
}

// sum_j (j + 1) B_j over the `half` buckets of an item, one item per (row, window).  A run of len consecutive buckets is
// carried as the pair A = sum_j (j - lo + 1) B_j, D = len * sum_j B_j, and two neighbouring runs of equal length join as
// A = A1 + A2 + D2, D = 2 (D1 + D2): no multiples by an offset, and the two halves of a join are independent, so two threads
// work on it.  A thread starts with a run of `per` buckets (running sums), a block joins its 128 runs, and a second launch
// joins the blocks' runs of an item.  What bounds it is the chain of dependent additions (2 per + 2 per level of the tree),
// so an item is spread over half / (128 per) blocks: 19 items of 8192 buckets take 224 + 24 us; one block per item with up to
// 32 buckets a thread took 774 us and kept 19 of 148 SMs busy.

// Joins n runs (a power of two, at most kReduceThreads) in A[], D[] (shared memory) into A[0], D[0].
__device__ __forceinline__ void join_runs(Xyzz* A, Xyzz* D, uint32_t n) {
  uint32_t pairs = n >> 1;
#pragma unroll 1
  for (; pairs > 16; pairs >>= 1) {  // a thread per half of a join, the D halves in warps of their own
    const uint32_t t = threadIdx.x;
    const bool is_a = t < pairs, is_d = t >= pairs && t < 2 * pairs;
    const uint32_t i = is_a ? t : t - pairs;
    Xyzz v;
    if (is_a) {
      v = A[2 * i];
      add_to(&v, &A[2 * i + 1]);
      add_to(&v, &D[2 * i + 1]);
    } else if (is_d) {
      v = D[2 * i];
      add_to(&v, &D[2 * i + 1]);
      dbl_in_place(&v);
    }
    __syncthreads();
    if (is_a) A[i] = v;
    if (is_d) D[i] = v;
    __syncthreads();
  }
  // four lanes per half: the first two warps take the A halves, the others the D halves
#pragma unroll 1
  for (; pairs > 0; pairs >>= 1) {
    const uint32_t q = (threadIdx.x & 63) >> 2, i = q < pairs ? q : 0;
    const int role = threadIdx.x & 3;
    const bool is_d = threadIdx.x >= 64;
    Xyzz* R = is_d ? D : A;
    QuadXyzz v = quad_add(quad_load(&R[2 * i], role), quad_load(&R[2 * i + 1], role), role);
    if (is_d) v = quad_dbl(v, role); else v = quad_add(v, quad_load(&D[2 * i + 1], role), role);
    __syncthreads();
    if (q < pairs) quad_store(&R[q], v, role);
    __syncthreads();
  }
}

// runs[2 * block], runs[2 * block + 1] = A and D of the block's buckets; with one block per item A goes to window_sums.
__global__ void __launch_bounds__(kReduceThreads) k_msm_bucket_reduce(const Xyzz* __restrict__ bucket_sums, uint32_t half,
                                                                      uint32_t per, uint32_t blocks_per_item, Xyzz* runs,
                                                                      Xyzz* window_sums) {
  __shared__ Xyzz A[kReduceThreads], D[kReduceThreads];
  const uint32_t item = blockIdx.x / blocks_per_item, part = blockIdx.x % blocks_per_item;
  const Xyzz* B = bucket_sums + (size_t)item * half;
  const uint32_t lo = (part * kReduceThreads + threadIdx.x) * per;
  Xyzz running = Xyzz::inf(), acc = Xyzz::inf();
  if (lo < half) {  // per divides half
    for (uint32_t j = lo + per; j-- > lo;) {
      const Xyzz bj = ld_xyzz(B + j);
      add_to(&running, &bj);
      add_to(&acc, &running);
    }
    // D is for joining: an item that is one run has no use for it (half of the kernel's 12 us for two buckets)
    if (per < half)
      for (uint32_t k = per; k > 1; k >>= 1) dbl_in_place(&running);
  }
  A[threadIdx.x] = acc;
  D[threadIdx.x] = running;
  __syncthreads();
  uint32_t n = half / per;  // runs of the item
  if (n > kReduceThreads) n = kReduceThreads;
  join_runs(A, D, n);
  if (threadIdx.x == 0) {
    if (blocks_per_item == 1) {
      st_xyzz(window_sums + item, A[0]);
    } else {
      st_xyzz(runs + 2 * (size_t)blockIdx.x, A[0]);
      st_xyzz(runs + 2 * (size_t)blockIdx.x + 1, D[0]);
    }
  }
}

__global__ void __launch_bounds__(kReduceThreads) k_msm_join_items(const Xyzz* __restrict__ runs, uint32_t blocks_per_item,
                                                                   Xyzz* window_sums) {
  __shared__ Xyzz A[kReduceThreads], D[kReduceThreads];
  if (threadIdx.x < blocks_per_item) {
    const size_t at = 2 * ((size_t)blockIdx.x * blocks_per_item + threadIdx.x);
    A[threadIdx.x] = ld_xyzz(runs + at);
    D[threadIdx.x] = ld_xyzz(runs + at + 1);
  }
  __syncthreads();
  join_runs(A, D, blocks_per_item);
  if (threadIdx.x == 0) st_xyzz(window_sums + blockIdx.x, A[0]);
}

// Many items (the d_x / d_y rows of a commitment: a thousand or more (row, window) items): a block per item leaves most of
// its additions to idle lanes.  Here `lanes` lanes (a power of two, 1 to 32) share an item.  Lane l takes `per` consecutive
// buckets: running sums give its local weighted sum A_l = sum_j (j - lo + 1) B_j and its plain sum R_l.  The item's result is
// sum_l A_l + per * sum_{l >= 1} S_l with S_l = sum_{u >= l} R_u (a suffix scan over the item's lanes), so
// every lane doubles its own S_l log2(per) times, adds A_l, and one tree over the lanes finishes.  The fewest lanes that still
// fill the GPU are taken: 6 656 items of 512 buckets take 1.8 ms with eight lanes each.  The four reductions of a KZH3 commitment
// and opening at 2^22 took 5.8 ms with a block per item everywhere (32 threads for these), and take 3.8 ms.
__global__ void __launch_bounds__(128) k_msm_bucket_reduce_rows(const Xyzz* __restrict__ bucket_sums, uint32_t half,
                                                               uint32_t n_items, uint32_t lanes, Xyzz* window_sums) {
  __shared__ Xyzz sh[128];
  const uint32_t t = threadIdx.x, l = t & (lanes - 1);
  const uint32_t item = blockIdx.x * (128 / lanes) + t / lanes;
  const bool live = item < n_items;
  const uint32_t per = half / lanes;  // a power of two, at least 1
  const Xyzz* B = bucket_sums + (size_t)(live ? item : 0) * half;
  Xyzz running = Xyzz::inf(), acc = Xyzz::inf();
  if (live) {
    const uint32_t lo = l * per;
    for (uint32_t j = lo + per; j-- > lo;) {
      const Xyzz bj = ld_xyzz(B + j);
      add_to(&running, &bj);
      add_to(&acc, &running);
    }
  }
  // inclusive suffix scan of the running sums over the item's lanes
  sh[t] = running;
  __syncwarp();
#pragma unroll 1
  for (uint32_t off = 1; off < lanes; off <<= 1) {
    Xyzz other = Xyzz::inf();
    if (l + off < lanes) other = sh[t + off];
    __syncwarp();
    add_to(&running, &other);
    sh[t] = running;
    __syncwarp();
  }
  // lane l >= 1 contributes per * S_l
  if (l == 0) running = Xyzz::inf();
  for (uint32_t k = per; k > 1; k >>= 1) dbl_in_place(&running);
  add_to(&acc, &running);
  sh[t] = acc;
  __syncwarp();
#pragma unroll 1
  for (uint32_t off = lanes / 2; off > 0; off >>= 1) {
    Xyzz other = Xyzz::inf();
    if (l < off) other = sh[t + off];
    __syncwarp();
    add_to(&acc, &other);
    sh[t] = acc;
    __syncwarp();
  }
  if (live && l == 0) st_xyzz(window_sums + item, acc);
}

__global__ void k_msm_combine(const Xyzz* __restrict__ window_sums, uint32_t rows, int w, int k_windows, Jacobian* out) {
  const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  Xyzz acc = Xyzz::inf();
  for (int k = k_windows - 1; k >= 0; k--) {
    for (int i = 0; i < w; i++) dbl_in_place(&acc);
    const Xyzz ws = ld_xyzz(window_sums + (size_t)row * k_windows + k);
    add_to(&acc, &ws);
  }
  out[row] = to_jacobian(acc);
}

// The same Horner sum for few rows, where the chain of W * K dependent doublings is the whole time (254 of them took a
// thread 1.13 ms).  A warp takes a row and four lanes a point (quad.cuh).  The eight quads of a warp take an eighth of the
// windows each, shift their sums up by their own number of doublings, and a tree over the quads finishes, so that the general
// additions stay off the chain: 254 doublings and the additions take 560 us.
__global__ void __launch_bounds__(32) k_msm_combine_quads(const Xyzz* __restrict__ window_sums, int w, int k_windows, Jacobian* out) {
  __shared__ Xyzz sh[8];
  const int lane = threadIdx.x, group = lane >> 2, role = lane & 3;
  const Xyzz* ws = window_sums + (size_t)blockIdx.x * k_windows;
  const int per = (k_windows + 7) >> 3, lo = group * per;
  QuadXyzz p;
  p.x = p.y = p.z = Fq::zero();
  // the quad's windows: sum_k 2^(W (k - lo)) ws[k]; the last window by address stands in for those past the end
#pragma unroll 1
  for (int s = per - 1; s >= 0; s--) {
    const int k = lo + s;
    if (s != per - 1)
#pragma unroll 1
      for (int i = 0; i < w; i++) p = quad_dbl(p, role);
    const QuadXyzz r = quad_add(p, quad_load(ws + (k < k_windows ? k : k_windows - 1), role), role);
    if (k < k_windows) p = r;
  }
  // shifted up by W lo bits (a quad without windows holds infinity)
  const int live = (k_windows + per - 1) / per;  // quads with windows
  const int most = (live - 1) * per * w;
#pragma unroll 1
  for (int i = 0; i < most; i++) {
    const QuadXyzz r = quad_dbl(p, role);
    if (i < lo * w) p = r;
  }
  quad_store(sh + group, p, role);
  __syncwarp();
#pragma unroll 1
  for (int off = 4; off > 0; off >>= 1) quad_add_to(&sh[group & (off - 1)], &sh[(group & (off - 1)) + off], group < off);
  if (lane == 0) out[blockIdx.x] = to_jacobian(sh[0]);
}

// 64-bit total of the per-bucket counts (the 32-bit prefix sums would wrap silently past 2^32), and how many of them lie in
// [from, to).
struct BucketCounts {
  unsigned long long total;
  unsigned int within;
};
__global__ void k_total64(const uint32_t* __restrict__ counts, uint32_t n, uint32_t from, uint32_t to, BucketCounts* found) {
  unsigned long long s = 0;
  uint32_t within = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t c = counts[i];
    s += c;
    within += c >= from && c < to;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, off);
    within += __shfl_down_sync(0xffffffffu, within, off);
  }
  if ((threadIdx.x & 31) == 0 && s) {
    atomicAdd(&found->total, s);
    if (within) atomicAdd(&found->within, within);
  }
}

__global__ void k_set_infinity(Jacobian* out, uint32_t rows) {
  const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row < rows) out[row] = to_jacobian(Xyzz::inf());
}

// ---- Sums of selected SRS points: the commitment of a selection polynomial (every listed entry is one).
// sparse_kzh2_commit / sparse_kzh3_commit (sparse_kzh2.rs:27-80, sparse_kzh3.rs:45-110) with all values one are
// C = sum_i h_full[idx_i] and d_x[r] = sum_{i in row r} h_mid[idx_i mod 2^low_bits], row r = idx >> low_bits.  With the
// indices in non-decreasing order a row is a contiguous run of the list, so the digit, sort and bucket passes of
// the general MSM are not needed: sixteen lanes take a row, each lane sums its share with mixed additions, a tree over
// the lanes (through shared memory) finishes the row, and the same walk adds the row's share of C.
constexpr int kSelLanes = 16;  // lanes per row (a full warp per row measured 20-35 % slower: twice the tree additions)

__device__ __forceinline__ uint32_t sel_lower_bound(const uint32_t* __restrict__ idx, uint32_t n, uint64_t key) {
  uint32_t lo = 0, hi = n;  // first position with idx >= key
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (idx[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// A block takes kSelRows rows; its first 128 threads add the rows' points from h_mid, the others the same entries' points from h_full,
// so that a thread has one chain of additions (inlined, the next point on its way) and a scheduler four warps.  Bound by the chain and the
// trees.  2^18 entries: 162 us; with both chains in one thread, called products and half the warps 177.
constexpr int kSelRows = 128 / kSelLanes;
__global__ void __launch_bounds__(256, 2) k_select_sums(const Affine* __restrict__ full, const Affine* __restrict__ mid,
                                                     const uint32_t* __restrict__ idx, const uint32_t* __restrict__ bad, uint32_t n,
                                                     uint32_t low_bits, uint32_t rows, Jacobian* d_x, Xyzz* c_partial) {
  if (bad[0] | bad[1]) return;  // the list is not in order: the host finds the same and goes another way
  const uint32_t slot = threadIdx.x & 127u, gl = slot % kSelLanes;
  const uint32_t group = blockIdx.x * kSelRows + slot / kSelLanes;
  const bool for_c = threadIdx.x >= 128;
  uint32_t lo = 0, hi = 0;
  if (group < rows) {
    lo = sel_lower_bound(idx, n, (uint64_t)group << low_bits);
    hi = sel_lower_bound(idx, n, ((uint64_t)group + 1) << low_bits);
  }
  const uint32_t mask = for_c || low_bits >= 32 ? 0xffffffffu : (1u << low_bits) - 1u;
  const Affine* bases = for_c ? full : mid;
  Xyzz acc = Xyzz::inf();
  uint32_t i = lo + gl;
  if (i < hi) {
    Affine next = ld_affine(bases + (idx[i] & mask));
    uint32_t v = i + kSelLanes < hi ? idx[i + kSelLanes] : 0u;
#pragma unroll 1
    for (; i < hi; i += kSelLanes) {
      const Affine pt = next;
      if (i + kSelLanes < hi) next = ld_affine(bases + (v & mask));
      if (i + 2 * kSelLanes < hi) v = idx[i + 2 * kSelLanes];
      acc = add_mixed(acc, pt);
    }
  }
  // The lanes' shares of a row: a tree through shared memory.  The time of this kernel follows the number of
  // warp-wide additions it issues, so the additions of a level are packed into as few warps as they fill: the row
  // sums' pairs take the first threads of the block, C's pairs the next, and whole warps sit a level out
  // (128, 64, 32 and 16 additions for the four levels, against two additions by every warp at every level).
  // The last three levels of the rows and the levels of C across the rows have few additions: four lanes each (quad.cuh; this
  // kernel 210 -> 187 us and the total of the blocks 62 -> 37 us at 2^18 entries).
  __shared__ Xyzz sh[2 * 128];  // [0, 128): shares of the rows' sums; [128, 256): shares of C
  sh[threadIdx.x] = acc;
  __syncthreads();
  constexpr int kRowsPerBlock = kSelRows;
#pragma unroll 1
  for (int off = kSelLanes / 2; off > 0; off >>= 1) {
    const int per_kind = kRowsPerBlock * off;  // additions of this level for one of the two sums
    if (2 * per_kind > 64) {
      if ((int)threadIdx.x < 2 * per_kind) {
        const int kind = (int)threadIdx.x / per_kind, t = (int)threadIdx.x % per_kind;
        Xyzz* at = sh + kind * 128 + (t / off) * kSelLanes + (t % off);
        add_to(at, at + off);
      }
    } else if ((threadIdx.x & ~31u) < 8u * per_kind) {
      const int q = (int)threadIdx.x >> 2, kind = q / per_kind, t = q % per_kind;
      Xyzz* at = sh + (kind & 1) * 128 + (t / off) * kSelLanes + (t % off);
      quad_add_to(at, at + off, kind < 2);
    }
    __syncthreads();
  }
  if (group < rows && gl == 0 && !for_c) d_x[group] = to_jacobian(sh[threadIdx.x]);
  // the shares of C of the block's rows
  Xyzz* sh_c = sh + 128;
#pragma unroll 1
  for (int off = kRowsPerBlock / 2; off > 0; off >>= 1) {
    if (threadIdx.x < 32) {
      const int q = (int)threadIdx.x >> 2, i = q < off ? q : 0;
      quad_add_to(&sh_c[kSelLanes * i], &sh_c[kSelLanes * (i + off)], q < off);
    }
  }
  if (threadIdx.x == 0) st_xyzz(c_partial + blockIdx.x, sh_c[0]);
}

// C = the sum of the blocks' shares (one block).
__global__ void __launch_bounds__(512) k_select_total(const Xyzz* __restrict__ c_partial, const uint32_t* __restrict__ bad, uint32_t rows, Jacobian* c_out) {
  __shared__ Xyzz sh[256];
  if (bad[0] | bad[1]) return;
  Xyzz acc = Xyzz::inf();
  if (threadIdx.x < 256) {
    for (uint32_t r = threadIdx.x; r < rows; r += 256) {
      const Xyzz v = ld_xyzz(c_partial + r);
      add_to(&acc, &v);
    }
    sh[threadIdx.x] = acc;
  }
  __syncthreads();
  tree_sum(sh, 256);  // 512 threads: four lanes for every addition
  if (threadIdx.x == 0) *c_out = to_jacobian(sh[0]);
}

// ---- Many dense rows of small scalars over the same bases (the d_x rows of a quantised weight matrix, kzh2.rs:653-660),
// by the method of the four Russians: the bases are taken in groups of `s`, all 2^s subset sums of a group are tabulated
// once for all the rows, and a row adds, for every bit plane of its scalars (two's complement), one table entry per group.
// That is planes * n / s additions a row and 2^s * n / s for the table, where buckets take n a row plus their reduction: for
// 4096 rows of 4096 int8 values 11.2 M + 1.4 M additions against 16.8 M + 0.5 M, and nothing is sorted: the d_x rows of that
// commitment take 2.4 ms (sums 1.82, tables 0.34, bits 0.07, joining 0.19) where counting, scattering, adding and reducing
// the buckets took 3.9 ms.

// idx[g][row * planes + k]: the bits of plane k of the scalars of group g.  A thread takes a (row, group).  n of the scalars of a
// row, which are `stride` apart from the next row's.
__global__ void __launch_bounds__(256) k_rows_bits(const int32_t* __restrict__ compact, uint64_t stride, uint32_t n, uint32_t rows, int planes,
                                                   int s, uint32_t groups, uint16_t* idx) {
  const uint64_t total = (uint64_t)rows * groups;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t row = (uint32_t)(t % rows), g = (uint32_t)(t / rows);
    const int32_t* v = compact + row * stride + (uint64_t)g * s;
    const int have = n - g * s < (uint32_t)s ? (int)(n - g * s) : s;
    uint16_t* out = idx + (uint64_t)g * rows * planes + (uint64_t)row * planes;
    int32_t w[kRowsGroupMax];
#pragma unroll
    for (int i = 0; i < kRowsGroupMax; i++) w[i] = i < have ? __ldg(v + i) : 0;
    for (int k = 0; k < planes; k++) {
      uint32_t bits = 0;
#pragma unroll
      for (int i = 0; i < kRowsGroupMax; i++) bits |= (((uint32_t)w[i] >> k) & 1u) << i;
      out[k] = (uint16_t)bits;
    }
  }
}

// Subset sums of the low and of the high half of a group's bases, 2^lo_bits + 2^hi_bits affine points a group.
__global__ void __launch_bounds__(128) k_rows_halves(const Affine* __restrict__ bases, uint32_t n, int s, int lo_bits, uint32_t groups,
                                                     Affine* halves) {
  const uint32_t per = (1u << lo_bits) + (1u << (s - lo_bits));
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= groups * per) return;
  const uint32_t g = t / per, m = t % per;
  const bool hi = m >= (1u << lo_bits);
  const uint32_t mask = hi ? m - (1u << lo_bits) : m;
  const uint32_t first = g * (uint32_t)s + (hi ? (uint32_t)lo_bits : 0u);
  Xyzz acc = Xyzz::inf();
#pragma unroll 1
  for (int i = 0; (mask >> i) != 0; i++)
    if (((mask >> i) & 1u) && first + i < n) acc = add_mixed_calls(acc, ld_affine(bases + first + i));
  Affine r;
  r.x = r.y = Fq::zero();
  if (!acc.is_inf()) {
    const Fq izzz = fq_inverse_fn(acc.zzz);
    const Fq iz = fq_mul_fn(izzz, acc.zz);  // 1 / zz = (zz / zzz)^2
    r.x = fq_mul_fn(acc.x, fq_mul_fn(iz, iz));
    r.y = fq_mul_fn(acc.y, izzz);
  }
  halves[t] = r;
}

// table[g][m] = halves[g][low bits of m] + halves[g][high bits of m]: kBatchTable sums a thread share an inversion.
constexpr int kBatchTable = 8;
__global__ void __launch_bounds__(kBatchThreads, 4) k_rows_table(const Affine* __restrict__ halves, int s, int lo_bits, uint32_t groups,
                                                                 Affine* table) {
  __shared__ Fq sh[kBatchThreads];
  const uint32_t per = (1u << lo_bits) + (1u << (s - lo_bits)), total = groups << s;
  const uint32_t t0 = blockIdx.x * (kBatchThreads * kBatchTable) + threadIdx.x;
  Fq pre[kBatchTable], run = Fq::one();
#pragma unroll 1
  for (int j = 0; j < kBatchTable; j++) {
    const uint32_t t = t0 + j * kBatchThreads;
    if (t >= total) continue;
    const uint32_t g = t >> s, m = t & ((1u << s) - 1u);
    const Affine p = ld_affine(halves + g * per + (m & ((1u << lo_bits) - 1u)));
    const Affine q = ld_affine(halves + g * per + (1u << lo_bits) + (m >> lo_bits));
    Fq den;
    add_kind(p, q, &den);
    pre[j] = run;
    run = fq_mul_fn(run, den);
  }
  Fq inv = block_inverse(run, sh);
#pragma unroll 1
  for (int j = kBatchTable - 1; j >= 0; j--) {
    const uint32_t t = t0 + j * kBatchThreads;
    if (t >= total) continue;
    const uint32_t g = t >> s, m = t & ((1u << s) - 1u);
    const Affine p = ld_affine(halves + g * per + (m & ((1u << lo_bits) - 1u)));
    const Affine q = ld_affine(halves + g * per + (1u << lo_bits) + (m >> lo_bits));
    Fq den;
    const AddKind kind = add_kind(p, q, &den);
    const Fq mine = fq_mul_fn(inv, pre[j]);
    inv = fq_mul_fn(inv, den);
    table[t] = add_with_inverse(p, q, kind, mine);
  }
}

// pieces[q][u]: unit u = (row, plane) over the groups [q seg, (q + 1) seg).  The lanes of a warp are neighbouring units at the
// same group, so their table reads fall into one group's 2^s entries and their idx reads are consecutive.
__global__ void __launch_bounds__(128, kAccBlocks) k_rows_sums(const Affine* __restrict__ table, const uint16_t* __restrict__ idx, uint32_t units,
                                                   int s, uint32_t groups, uint32_t seg, uint32_t n_pieces, Xyzz* pieces) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_pieces) return;
  const uint32_t q = c / units, u = c % units;
  const uint32_t g1 = (q + 1) * seg < groups ? (q + 1) * seg : groups;
  Xyzz acc = Xyzz::inf();
  for (uint32_t g = q * seg; g < g1; g++) {
    const uint32_t m = idx[(uint64_t)g * units + u];
    if (m) acc = add_mixed(acc, ld_affine(table + ((uint64_t)g << s) + m));
  }
  st_xyzz(pieces + c, acc);
}

// The sum of a unit's pieces: four lanes a unit, lane l of a unit takes the pieces l, l + 4, ...; written over piece 0.
__global__ void __launch_bounds__(128) k_rows_units(Xyzz* pieces, uint32_t units, uint32_t parts) {
  __shared__ Xyzz sh[128];
  // thread = lane-of-unit * 32 + unit-in-block: the lanes of a warp read neighbouring units
  const uint32_t l = threadIdx.x >> 5, u = blockIdx.x * 32 + (threadIdx.x & 31);
  Xyzz acc = Xyzz::inf();
  if (u < units)
    for (uint32_t q = l; q < parts; q += 4) {
      const Xyzz v = ld_xyzz(pieces + (uint64_t)q * units + u);
      add_to(&acc, &v);
    }
  sh[threadIdx.x] = acc;
  __syncthreads();
  if (l < 2) {
    add_to(&acc, &sh[threadIdx.x + 64]);
    sh[threadIdx.x] = acc;
  }
  __syncthreads();
  if (l == 0) {
    add_to(&acc, &sh[threadIdx.x + 32]);
    if (u < units) st_xyzz(pieces + u, acc);
  }
}

// A row's result: sum_k 2^k (plane k), the top plane (the sign bits) subtracted.
__global__ void __launch_bounds__(64) k_rows_planes(const Xyzz* __restrict__ unit_sums, uint32_t rows, int planes, Jacobian* out) {
  const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  Xyzz acc = Xyzz::inf();
#pragma unroll 1
  for (int k = planes - 1; k >= 0; k--) {
    Xyzz v = ld_xyzz(unit_sums + (uint64_t)row * planes + k);
    if (k == planes - 1) v = neg(v);
    dbl_in_place(&acc);
    add_to(&acc, &v);
  }
  out[row] = to_jacobian(acc);
}

}  // namespace

int msm_run(zk_ctx* ctx, const Affine* bases, const uint32_t* gather, const Fr* scalars, uint64_t n, uint32_t rows,
            Jacobian* out_dev, MsmStats* stats, MsmPrep* prep) {
  return msm_run_rows(ctx, bases, gather, nullptr, scalars, n, rows, out_dev, stats, prep);
}

// Horner over the windows on the host, for one row or a few (combine_by).
static int combine_on_host(zk_ctx* ctx, const Xyzz* window_sums, uint32_t rows, int w, int k_windows, Jacobian* out_dev) {
  static_assert(kHostCombineRows * 128 * sizeof(Xyzz) + kHostCombineRows * sizeof(Jacobian) <= kHostPointsBytes, "128 windows of two bits at most");
  Xyzz* ws = reinterpret_cast<Xyzz*>(ctx->host_points);
  Jacobian* out = reinterpret_cast<Jacobian*>(ws + kHostCombineRows * 128);
  ZK_CUDA(cudaMemcpyAsync(ws, window_sums, (size_t)rows * k_windows * sizeof(Xyzz), cudaMemcpyDeviceToHost, ctx->stream));
  ZK_CUDA(cudaStreamSynchronize(ctx->stream));
  for (uint32_t r = 0; r < rows; r++) {
    Xyzz acc = Xyzz::inf();
    for (int k = k_windows - 1; k >= 0; k--) {
      for (int i = 0; i < w && !acc.is_inf(); i++) acc = dbl(acc);
      acc = add(acc, ws[(size_t)r * k_windows + k]);
    }
    out[r] = to_jacobian(acc);
  }
  ZK_CUDA(cudaMemcpyAsync(out_dev, out, rows * sizeof(Jacobian), cudaMemcpyHostToDevice, ctx->stream));
  return 0;
}

// base: plan.scratch() bytes.
static int rows_run(zk_ctx* ctx, const Affine* bases, const int32_t* compact, uint32_t n, uint32_t rows, const RowsPlan& plan,
                    char* base, Jacobian* out_dev, MsmStats* stats, int max_bits, cudaStream_t st) {
  const int sm = ctx->sm_count, s = plan.group, lo_bits = (s + 1) / 2;
  const uint32_t groups = plan.groups, seg = plan.seg, parts = plan.parts;
  const uint64_t units = (uint64_t)rows * plan.planes;
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += align256(bytes); return p; };
  uint16_t* idx = (uint16_t*)take(plan.idx_bytes);
  Affine* halves = (Affine*)take(plan.halves_bytes);
  Affine* table = (Affine*)take(plan.table_bytes);
  Xyzz* pieces = (Xyzz*)take(plan.pieces_bytes);
  for (uint32_t q0 = 0; q0 < parts; q0 += plan.slab) {  // the chains [q0, q0 + chains) and their groups [g0, g0 + held)
    const uint32_t chains = std::min(plan.slab, parts - q0), g0 = q0 * seg, held = std::min(groups - g0, chains * seg);
    const uint32_t first = g0 * (uint32_t)s, left = n - first;
    const uint32_t half_points = held * ((1u << lo_bits) + (1u << (s - lo_bits)));
    const uint64_t bit_blocks = ((uint64_t)rows * held + 255) / 256;
    const uint64_t per_block = kBatchThreads * kBatchTable, table_blocks = (((uint64_t)held << s) + per_block - 1) / per_block;
    const uint32_t sums = chains * (uint32_t)units;
    k_rows_bits<<<(unsigned)std::min<uint64_t>(bit_blocks, (uint64_t)sm * 32), 256, 0, st>>>(compact + first, n, left, rows, plan.planes, s, held, idx);
    k_rows_halves<<<(half_points + 127) / 128, 128, 0, st>>>(bases + first, left, s, lo_bits, held, halves);
    k_rows_table<<<(unsigned)table_blocks, kBatchThreads, 0, st>>>(halves, s, lo_bits, held, table);
    k_rows_sums<<<(sums + 127) / 128, 128, 0, st>>>(table, idx, (uint32_t)units, s, held, seg, sums, pieces + (uint64_t)q0 * units);
    ctx->launches += 4;
  }
  if (parts > 1) {
    k_rows_units<<<(unsigned)((units + 31) / 32), 128, 0, st>>>(pieces, (uint32_t)units, parts);
    ctx->launches++;
  }
  k_rows_planes<<<(rows + 63) / 64, 64, 0, st>>>(pieces, rows, plan.planes, out_dev);
  ctx->launches++;
  ZK_CUDA(cudaGetLastError());
  const uint64_t lookups = units * groups;  // one mixed addition each, but for the empty subsets
  ctx->msm_entries_sum += lookups;
  ctx->msm_calls++;
  if (stats) {
    stats->window_bits = 1;
    stats->windows = plan.planes;
    stats->entries = lookups;
    stats->buckets = 0;
    stats->max_bits = max_bits;
  }
  return 0;
}

template <int MODE>
static void launch_digits(ScalarForm form, uint32_t small_keys, uint32_t dig_blocks, uint64_t per_block, int sm, const Fr* scalars, const int32_t* compact,
                          const uint32_t* row_ids, uint64_t n, uint32_t rows, int w, int k_windows, uint32_t table_step,
                          uint32_t* counts_or_cursor, uint32_t* entries, cudaStream_t s) {
  auto launch = [&](auto small, auto large) {
    if (small_keys)
      small<<<dig_blocks, 256, 0, s>>>(scalars, compact, row_ids, n, rows, w, k_windows, table_step, small_keys, per_block, counts_or_cursor, entries);
    else
      large<<<sm * 8, 256, 0, s>>>(scalars, compact, row_ids, n, rows, w, k_windows, table_step, counts_or_cursor, entries);
  };
  switch (form) {
    case kCompact: launch(k_msm_digits_small<MODE, kCompact>, k_msm_digits<MODE, kCompact>); break;
    case kEndo: launch(k_msm_digits_small<MODE, kEndo>, k_msm_digits<MODE, kEndo>); break;
    case kWide: launch(k_msm_digits_small<MODE, kWide>, k_msm_digits<MODE, kWide>); break;
  }
}

// The tables of subset sums for the rows of a call whose scalars are small; no group: buckets are the better way.
static RowsPlan small_rows_plan(const MsmPrep& prep, uint64_t n, uint32_t rows, const BucketPlan& plan, int sm) {
  const size_t buckets = plan.n_buckets >= (1ull << 31) ? ~(size_t)0 : plan.scratch + align256(scan_scratch_elems(plan.n_buckets + 1) * 4);
  return rows_plan(n, rows, prep.max_span, prep.nonzero, plan, sm, buckets);
}

// The rows of a commitment beside its C, both over the same small scalars: the rows' tables and sums on the side stream while C sorts
// its digits, whichever is done first leaving the GPU to the other.  A commitment of 2^24 int8 values in 2^12 rows takes 5 633 us, one after
// the other 6 079; of 2^20 741 and 982, of 2^25 10 914 and 11 525; int16 942 and 1 289, 7 762 and 8 277, 14 949 and 15 655 (2^20, 2^24, 2^25).
// Their scratch lies beside C's then and stays in the lane's: 153 MB for 2^24 int8 values, 357 MB for 2^25 of 24 bits.  kBesideMost bounds
// that memory; every shape of up to 2^25 values is below it, and faster like this.
constexpr size_t kBesideMost = 512u << 20;

// row_ids == nullptr: `rows` dense rows of n scalars each over the same n bases.  Otherwise: n scalars in
// all, scalar i contributes scalars[i] * bases[gather ? gather[i] : i] to output row row_ids[i] < rows.
// plain: without what takes scratch beside the buckets, where there was no room for it.
static int msm_run_impl(zk_ctx* ctx, const Affine* bases, const uint32_t* gather, const uint32_t* row_ids, const Fr* scalars,
                        uint64_t n, uint32_t rows, Jacobian* out_dev, MsmStats* stats, MsmPrep* prep, bool plain, MsmRowsBeside* also) {
  cudaStream_t s = ctx->stream;
  const uint64_t total = row_ids ? n : n * rows;
  const int sm = ctx->sm_count;
  if (rows == 0) return 0;
  if (n == 0) {
    k_set_infinity<<<(rows + 127) / 128, 128, 0, s>>>(out_dev, rows);
    ctx->launches++;
    return 0;
  }
  if (n >= (1ull << 31)) return fail(-1, "msm: at most 2^31 - 1 points per row");
  // ---- pass 1: scalar magnitude (and the compact form of small scalars); a caller that runs several
  // MSMs over the same scalars passes `prep` and the pass runs once
  MsmPrep own;
  if (!prep) prep = &own;
  if (!(prep->valid && prep->scalars == scalars && prep->total == total)) {
    MsmBits* d_found = reinterpret_cast<MsmBits*>(ctx->rs.sink.counter + 8);  // spare words of the context's counter block
    int32_t* cbuf = nullptr;
    int crc = ctx->reserve_cmp(total * 4 + 256, (void**)&cbuf);
    if (crc) return crc;
    ZK_CUDA(cudaMemsetAsync(d_found, 0, sizeof(MsmBits), s));
    k_msm_bits<<<sm * 8, 256, 0, s>>>(scalars, total, d_found, cbuf);
    ctx->launches++;
    ZK_CUDA(cudaMemcpyAsync(ctx->host_small, d_found, sizeof(MsmBits), cudaMemcpyDeviceToHost, s));
    ZK_CUDA(cudaStreamSynchronize(s));
    MsmBits found;
    memcpy(&found, ctx->host_small, sizeof(found));
    prep->valid = true;
    prep->scalars = scalars;
    prep->total = total;
    prep->max_bits = found.bits;
    prep->max_mag = found.mag;
    prep->max_span = found.span;
    prep->nonzero = found.nonzero;
    prep->compact = found.bits <= (unsigned)kCompactBits ? cbuf : nullptr;
  }
  const unsigned int max_bits = prep->max_bits;
  const int32_t* compact = prep->compact;
  if (max_bits == 0) {
    k_set_infinity<<<(rows + 127) / 128, 128, 0, s>>>(out_dev, rows);
    ctx->launches++;
    return 0;
  }
  // Full-width scalars are split into two halves by the endomorphism: as many digits, half the windows (buckets, doublings).  100003
  // points: kernels 752 -> 728 us (bucket reduction 153 -> 118), the chain of doublings on the host half as long, the call 929 -> 862 us.
  // Scalars of up to 160 bits stay whole: they have fewer digits than 2 x 126 bits have.
  const bool endo = !compact && !row_ids && !gather && max_bits > kEndoBits && n <= kEndoMost && !plain;
  const int bits = endo ? kEndoMagnitude : (int)max_bits;
  const bool merged = endo && merged_rows(n, rows);
  // Separate windows of several rows: a bit more than for whole scalars, as there are half as many (pick_window).
  const int w = merged ? merged_window(n) : pick_window(row_ids ? (n / rows ? n / rows : 1) : n, rows, bits) + (endo && rows > 1 ? 1 : 0);
  // small scalars: the exact largest magnitude is known, which can save the window that would only
  // hold carries (int8 values reach 128 = one 8-bit signed digit)
  const int digit_windows = compact ? windows_for(prep->max_mag, w) : (bits + 1 + w - 1) / w;
  const int k_windows = merged ? 1 : digit_windows;  // with buckets of their own
  const uint64_t digits = (uint64_t)digit_windows * (endo ? 2 : 1);  // of a scalar, at most
  const BucketPlan plan = bucket_plan(endo ? (merged ? 2 * total * digit_windows : 2 * total) : total, rows, w, k_windows, sm);
  const uint32_t half = plan.half;
  const bool too_many = plan.n_buckets >= (1ull << 31);
  const uint32_t n_buckets = (uint32_t)plan.n_buckets;
  const size_t scan_bytes = too_many ? 0 : align256(scan_scratch_elems(n_buckets + 1) * 4);
  if (compact && rows > 1 && !row_ids && !gather) {
    const RowsPlan by_sums = small_rows_plan(*prep, n, rows, plan, sm);
    if (by_sums.group) {
      char* base = nullptr;
      int rc = ctx->reserve_aux(by_sums.scratch(), (void**)&base);
      if (!rc) rc = rows_run(ctx, bases, compact, (uint32_t)n, rows, by_sums, base, out_dev, stats, (int)max_bits, s);
      if (rc != -2 /*ZK_ERR_OOM*/) return rc;  // no room for the tables: the buckets of a small call may still have it
    }
  }
  auto plainly = [&] { return msm_run_impl(ctx, bases, gather, row_ids, scalars, n, rows, out_dev, stats, prep, true, nullptr); };
  if (too_many && endo) return plainly();
  if (too_many) return fail(-1, "msm: %llu buckets exceed the 32-bit key space; split the rows", (unsigned long long)plan.n_buckets);

  // ---- scratch layout (second scratch region of the context; the first holds caller data)
  const uint64_t table_points = merged ? n * (uint64_t)digit_windows : 0;
  const uint32_t table_step = merged ? (uint32_t)n : 0;
  static_assert(sizeof(Affine) + sizeof(Xyzz) + sizeof(Fq) == kMultipleBytes, "what the plan counts for a multiple");
  const size_t endo_bytes = (endo ? align256((merged ? table_points : n) * sizeof(Fq)) : 0) + align256(table_points * sizeof(Affine)) +
                            align256(table_points * sizeof(Xyzz));
  RowsPlan also_plan;
  also_plan.group = 0;
  if (also && compact && also->rows > 1 && also->n * also->rows == total && !ctx->prof_on) {
    const int also_w = pick_window(also->n, also->rows, (int)max_bits);
    also_plan = small_rows_plan(*prep, also->n, also->rows, bucket_plan(total, also->rows, also_w, windows_for(prep->max_mag, also_w), sm), sm);
    if (also_plan.group && also_plan.scratch() > kBesideMost) also_plan.group = 0;
  }
  const size_t own_bytes = align256(plan.scratch + scan_bytes + endo_bytes);
  char* base = nullptr;
  int rc = ctx->reserve_aux(own_bytes + (also_plan.group ? also_plan.scratch() : 0), (void**)&base);
  if (rc == -2 /*ZK_ERR_OOM*/ && also_plan.group) {
    also_plan.group = 0;
    rc = ctx->reserve_aux(own_bytes, (void**)&base);
  }
  if (rc == -2 /*ZK_ERR_OOM*/ && endo) return plainly();
  if (rc) return rc;
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += align256(bytes); return p; };
  uint32_t* offsets = (uint32_t*)take((n_buckets + 2) * 4ull);
  uint32_t* cursor = (uint32_t*)take((n_buckets + 2) * 4ull);
  uint32_t* scan_tmp = (uint32_t*)take(scan_bytes);
  Xyzz* bucket_sums = (Xyzz*)take((size_t)n_buckets * sizeof(Xyzz));
  Xyzz* window_sums = (Xyzz*)take((size_t)rows * k_windows * sizeof(Xyzz));
  uint32_t* entries = (uint32_t*)take(plan.max_entries * 4);
  Xyzz* heads = (Xyzz*)take((plan.chunks + 1) * sizeof(Xyzz));
  Xyzz* tails = (Xyzz*)take((plan.chunks + 1) * sizeof(Xyzz));
  Xyzz* fix_part = (Xyzz*)take((size_t)kFixupPartials * sizeof(Xyzz));
  Xyzz* runs = (Xyzz*)take(plan.n_runs * sizeof(Xyzz));
  Fq* images = endo ? (Fq*)take((merged ? table_points : n) * sizeof(Fq)) : nullptr;
  Affine* table = (Affine*)take(table_points * sizeof(Affine));
  Xyzz* multiples = (Xyzz*)take(table_points * sizeof(Xyzz));
  struct Join {  // however this call ends, the stream goes on after the side stream
    zk_ctx* ctx = nullptr;
    ~Join() {
      if (ctx && cudaEventRecord(ctx->ev_join, ctx->side_stream) == cudaSuccess) cudaStreamWaitEvent(ctx->stream, ctx->ev_join, 0);
    }
  } join;
  if (also_plan.group) {
    ZK_CUDA(cudaEventRecord(ctx->ev_fork, s));
    ZK_CUDA(cudaStreamWaitEvent(ctx->side_stream, ctx->ev_fork, 0));
    join.ctx = ctx;
    rc = rows_run(ctx, also->bases, compact, (uint32_t)also->n, also->rows, also_plan, base + own_bytes, also->out_dev, nullptr, (int)max_bits,
                  ctx->side_stream);
    if (rc) return rc;
    also->done = true;
  }
  // ---- pass 2: count, scan, scatter
  ZK_CUDA(cudaMemsetAsync(offsets, 0, (n_buckets + 2) * 4ull, s));
  const ScalarForm form = compact ? kCompact : endo ? kEndo : kWide;
  // The multiples are a chain of doublings that leaves most of the GPU idle: beside the digit passes, on the side stream.  With the
  // per-kernel profiler on they stay in line.
  const bool beside = merged && !ctx->prof_on;
  if (merged) {
    cudaStream_t s2 = beside ? ctx->side_stream : s;
    if (beside) {
      ZK_CUDA(cudaEventRecord(ctx->ev_fork, s));
      ZK_CUDA(cudaStreamWaitEvent(s2, ctx->ev_fork, 0));
    }
    k_multiples<<<(unsigned)((n + 31) / 32), 128, 0, s2>>>(bases, n, w, digit_windows, multiples);
    const uint64_t per = kBatchThreads * kMultiplesPer;
    k_multiples_affine<<<(unsigned)((table_points + per - 1) / per), kBatchThreads, 0, s2>>>(multiples, table_points, table, images);
    ctx->launches += 2;
    if (beside) ZK_CUDA(cudaEventRecord(ctx->ev_join, s2));
  } else if (endo) {
    k_endo_images<<<(unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)sm * 16), 256, 0, s>>>(bases, n, images);
    ctx->launches++;
  }
  // 4096 digits a block, not scalars: 1000 full-width scalars of 37 digits each were one block's work (638 us, 561 us with ten)
  uint32_t dig_blocks = (uint32_t)std::min<uint64_t>((total * digits + 4095) / 4096, 1u << 20);
  if (dig_blocks > (uint32_t)sm * 8) dig_blocks = sm * 8;
  const uint64_t per_block = (total + dig_blocks - 1) / dig_blocks;
  const uint32_t small_keys = n_buckets <= kSmallKeys ? n_buckets : 0;  // counted in shared memory
  launch_digits<0>(form, small_keys, dig_blocks, per_block, sm, scalars, compact, row_ids, n, rows, w, digit_windows, table_step, offsets, nullptr, s);
  ctx->launches++;
  BucketCounts* d_counts = reinterpret_cast<BucketCounts*>(ctx->rs.sink.counter + 10);
  ZK_CUDA(cudaMemsetAsync(d_counts, 0, sizeof(BucketCounts), s));
  const uint32_t chunk = chunk_entries((uint32_t)std::min<uint64_t>(prep->nonzero * digits, 0xffffffffull), sm);  // or a little less
  k_total64<<<sm * 4, 256, 0, s>>>(offsets, n_buckets, kFewPieces * chunk, kManyPieces * chunk, d_counts);
  ctx->launches++;
  ZK_CUDA(cudaMemcpyAsync(ctx->host_small, d_counts, sizeof(BucketCounts), cudaMemcpyDeviceToHost, s));
  ZK_CUDA(cudaStreamSynchronize(s));
  BucketCounts counts;
  memcpy(&counts, ctx->host_small, sizeof(counts));
  if (beside && counts.total > 0xffffffffull) ZK_CUDA(cudaStreamWaitEvent(s, ctx->ev_join, 0));
  if (counts.total > 0xffffffffull && endo) return plainly();  // of other window widths, a few digits less
  if (counts.total > 0xffffffffull) return fail(-1, "msm: %llu digit entries exceed 2^32 - 1; split the call", counts.total);
  const uint32_t n_entries = (uint32_t)counts.total;
  ctx->launches += exclusive_scan_u32(offsets, n_buckets, scan_tmp, true, s);
  ZK_CUDA(cudaMemcpyAsync(cursor, offsets, (n_buckets + 1) * 4ull, cudaMemcpyDeviceToDevice, s));
  launch_digits<1>(form, small_keys, dig_blocks, per_block, sm, scalars, compact, row_ids, n, rows, w, digit_windows, table_step, cursor, entries, s);
  ctx->launches++;

  // ---- accumulate
  if (beside) ZK_CUDA(cudaStreamWaitEvent(s, ctx->ev_join, 0));
  ZK_CUDA(cudaMemsetAsync(bucket_sums, 0, (size_t)n_buckets * sizeof(Xyzz), s));
  if (n_entries) {
    const uint32_t seg = chunk_entries(n_entries, sm);
    const uint32_t n_chunks = (n_entries + seg - 1) / seg;
    k_msm_accumulate<<<(n_chunks + 127) / 128, 128, 0, s>>>(merged ? table : bases, images, gather, entries, offsets, n_buckets, n_entries, seg,
                                                           n_chunks, bucket_sums, heads, tails);
    // cursor[] is free again after the scatter: it stands at the ends of the buckets
    if (n_buckets <= kFixupBuckets) {
      const uint64_t longest = row_ids ? n_entries : endo ? n * (merged ? digits : 2) : n;
      const uint32_t groups = fixup_groups(n_buckets, n_chunks, longest, seg);
      k_msm_fixup_block<<<dim3(n_buckets, groups), 128, 0, s>>>(offsets, seg, groups, cursor, bucket_sums, heads, tails, fix_part);
    } else {
      uint32_t* listed = ctx->rs.sink.counter + 12;
      ZK_CUDA(cudaMemsetAsync(listed, 0, 8, s));
      const uint32_t few = counts.within > 2u * (uint32_t)sm * (kFixupThreads / 32) ? kManyPieces : kFewPieces;
      k_msm_fixup_few<<<(n_buckets + 255) / 256, 256, 0, s>>>(offsets, n_buckets, seg, few, bucket_sums, heads, tails, cursor /* the list of long buckets */, listed);
      k_msm_fixup<<<sm * 2, kFixupThreads, 0, s>>>(offsets, cursor, listed, n_buckets, seg, bucket_sums, heads, tails);
      ctx->launches++;
    }
    ctx->launches += 2;
  }
  // ---- reduce buckets, combine windows
  const uint32_t n_items = rows * (uint32_t)k_windows;
  const uint32_t lanes = reduce_lanes(n_items, half, sm);
  if (lanes) {
    k_msm_bucket_reduce_rows<<<(n_items + 128 / lanes - 1) / (128 / lanes), 128, 0, s>>>(bucket_sums, half, n_items, lanes, window_sums);
  } else {
    k_msm_bucket_reduce<<<n_items * plan.red_parts, kReduceThreads, 0, s>>>(bucket_sums, half, plan.red_per, plan.red_parts, runs, window_sums);
    if (plan.red_parts > 1) {
      k_msm_join_items<<<n_items, kReduceThreads, 0, s>>>(runs, plan.red_parts, window_sums);
      ctx->launches++;
    }
  }
  switch (combine_by(rows, w, k_windows, sm)) {
    case Combine::kHost:
      rc = combine_on_host(ctx, window_sums, rows, w, k_windows, out_dev);
      if (rc) return rc;
      break;
    case Combine::kWarps:
      k_msm_combine_quads<<<rows, 32, 0, s>>>(window_sums, w, k_windows, out_dev);
      ctx->launches++;
      break;
    case Combine::kThreads:
      k_msm_combine<<<(rows + 63) / 64, 64, 0, s>>>(window_sums, rows, w, k_windows, out_dev);
      ctx->launches++;
      break;
  }
  ctx->launches++;  // the bucket reduction
  ZK_CUDA(cudaGetLastError());
  ctx->msm_entries_sum += n_entries;
  ctx->msm_bucket_sum += n_buckets;
  ctx->msm_calls++;
  if (stats) {
    stats->window_bits = w;
    stats->windows = k_windows;
    stats->entries = n_entries;
    stats->buckets = n_buckets;
    stats->max_bits = (int)max_bits;
  }
  return 0;
}

int msm_run_rows(zk_ctx* ctx, const Affine* bases, const uint32_t* gather, const uint32_t* row_ids, const Fr* scalars,
                 uint64_t n, uint32_t rows, Jacobian* out_dev, MsmStats* stats, MsmPrep* prep) {
  return msm_run_impl(ctx, bases, gather, row_ids, scalars, n, rows, out_dev, stats, prep, false, nullptr);
}

int msm_run_commit(zk_ctx* ctx, const Affine* bases, const Fr* scalars, uint64_t n, Jacobian* out_dev, MsmStats* stats, MsmPrep* prep,
                   MsmRowsBeside* rows) {
  return msm_run_impl(ctx, bases, nullptr, nullptr, scalars, n, 1, out_dev, stats, prep, false, rows);
}

// C (out_dev[rows]) and d_x (out_dev[0 .. rows)) of a selection polynomial over n indices in non-decreasing order
// (device, 32-bit), below rows << low_bits; nothing is read or written where one of the two words of bad (device) is not zero.
// scratch: rows Xyzz elements of device memory.
int msm_select_sums(zk_ctx* ctx, const Affine* full, const Affine* mid, const uint32_t* idx_dev, const uint32_t* bad, uint32_t n,
                    uint32_t low_bits, uint32_t rows, Jacobian* out_dev, void* scratch) {
  cudaStream_t s = ctx->stream;
  Xyzz* partial = reinterpret_cast<Xyzz*>(scratch);
  const uint32_t blocks = (rows + kSelRows - 1) / kSelRows;
  k_select_sums<<<blocks, 256, 0, s>>>(full, mid, idx_dev, bad, n, low_bits, rows, out_dev, partial);
  k_select_total<<<1, 512, 0, s>>>(partial, bad, blocks, out_dev + rows);
  ctx->launches += 2;
  ctx->msm_calls += 2;
  ctx->msm_entries_sum += 2ull * n;
  ctx->msm_bucket_sum += rows + 1;
  ZK_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace zk
