// Affine point additions that share their field inversions ("Montgomery's trick"): the pieces common to the kernels that
// add many independent pairs at a time.
//
// An affine addition is lambda = (y2 - y1) / (x2 - x1), x3 = lambda^2 - x1 - x2, y3 = lambda (x1 - x3) - y1: three products
// once the inverse is known.  A thread that works on K independent additions at once multiplies their denominators into a
// running product, has the product inverted, and peels the inverses off backwards: three more products an addition, six
// in all where the mixed addition into extended Jacobian coordinates takes ten.  The inversion itself (about 60 products'
// time for a warp) is shared by the four threads of a block that have the same lane, so it costs a thread some 15 products
// per K additions.
//
// It pays where the additions are independent and each is done once (k_rows_table: 1.4 M sums in 242 us).  Chains of additions,
// one step of K chains at a time, were slower than extended Jacobian sums (bucket sums of 2^24 entries with K = 8: 3.75 ms
// against 2.71 ms): every step waits for an inversion, and the running sums and products live in local memory.
#pragma once
#include "ec.cuh"

namespace zk {

constexpr int kBatchThreads = 128;  // four warps share an inversion; four such blocks live on an SM, so that the
                                    // others work while one of them waits for its inversion

static __device__ __noinline__ Fq fq_mul_fn(const Fq a, const Fq b) { return mul(a, b); }
static __device__ __noinline__ Fq fq_sqr_fn(const Fq a) { return sqr(a); }
static __device__ __noinline__ Fq fq_inverse_fn(const Fq a) { return inverse(a); }

// Every thread's inverse of its own non-zero value; sh: kBatchThreads elements of shared memory.  All threads call it.
__device__ __forceinline__ Fq block_inverse(const Fq& v, Fq* sh) {
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
  if (t < 32) {
    const Fq p1 = sh[32 + t], p2 = sh[64 + t], p3 = sh[96 + t];
    const Fq q1 = fq_mul_fn(v, p1), q2 = fq_mul_fn(q1, p2);
    Fq inv = fq_inverse_fn(fq_mul_fn(q2, p3));
    sh[96 + t] = fq_mul_fn(inv, q2);
    inv = fq_mul_fn(inv, p3);
    sh[64 + t] = fq_mul_fn(inv, q1);
    inv = fq_mul_fn(inv, p2);
    sh[32 + t] = fq_mul_fn(inv, v);
    sh[t] = fq_mul_fn(inv, p1);
  }
  __syncthreads();
  const Fq r = sh[t];
  return r;
}

// How p + q is to be computed, from the coordinates alone.
enum AddKind : int {
  kAddTakeP = 0,   // q is infinity
  kAddTakeQ = 1,   // p is infinity
  kAddNone = 2,    // q = -p: infinity
  kAddDouble = 3,  // q = p: denominator 2 y
  kAddChord = 4    // denominator x2 - x1
};

// Kind of p + q and its denominator (one when nothing is divided).  The coordinates of infinity are zero.
__device__ __forceinline__ AddKind add_kind(const Affine& p, const Affine& q, Fq* den) {
  *den = Fq::one();
  if (q.is_inf()) return kAddTakeP;
  if (p.is_inf()) return kAddTakeQ;
  const Fq dx = sub(q.x, p.x);
  if (!dx.is_zero()) {
    *den = dx;
    return kAddChord;
  }
  if (p.y != q.y || p.y.is_zero()) return kAddNone;
  *den = dbl(p.y);
  return kAddDouble;
}

// The sum, given the inverse of the denominator.
__device__ __forceinline__ Affine add_with_inverse(const Affine& p, const Affine& q, AddKind kind, const Fq& inv) {
  if (kind == kAddTakeP) return p;
  if (kind == kAddTakeQ) return q;
  Affine r;
  if (kind == kAddNone) {
    r.x = r.y = Fq::zero();
    return r;
  }
  Fq num = sub(q.y, p.y);
  if (kind == kAddDouble) {
    const Fq x2 = fq_sqr_fn(p.x);
    num = add(dbl(x2), x2);
  }
  const Fq lambda = fq_mul_fn(num, inv);
  r.x = sub(sub(fq_sqr_fn(lambda), p.x), q.x);
  r.y = sub(fq_mul_fn(lambda, sub(p.x, r.x)), p.y);
  return r;
}

}  // namespace zk
