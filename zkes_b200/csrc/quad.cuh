// Point operations by four neighbouring lanes: for the places where a kernel is down to a few dependent additions or
// doublings (the ends of trees, Horner chains) and its time is their latency.  A field product is one thread's work of
// ~0.3 us; a general addition is fourteen of them and a doubling nine, but in four and three dependent steps of at most
// four products each, which the lanes of a quad compute at the same time and hand round by shuffles.
//
// All lanes of the warp call these together (the shuffles name the whole warp); a quad without work passes on = false and
// any readable operands.
#pragma once
#include "ec.cuh"

namespace zk {

static __device__ __noinline__ Fq quad_mul(const Fq a, const Fq b) { return mul(a, b); }

__device__ __forceinline__ Fq quad_get(const Fq& v, int role) {  // the quad's lane `role` has it
  Fq r;
#pragma unroll
  for (int k = 0; k < 8; k++) r.v[k] = __shfl_sync(0xffffffffu, v.v[k], role, 4);
  return r;
}
__device__ __forceinline__ Fq quad_pick(int role, const Fq& a, const Fq& b, const Fq& c, const Fq& d) {
  Fq r;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint32_t lo = (role & 1) ? b.v[k] : a.v[k], hi = (role & 1) ? d.v[k] : c.v[k];
    r.v[k] = (role & 2) ? hi : lo;
  }
  return r;
}

// A point spread over a quad: x and y in all four lanes, z = ZZ in lanes 0 and 2, ZZZ in lanes 1 and 3.
struct QuadXyzz {
  Fq x, y, z;
};

__device__ __forceinline__ QuadXyzz quad_load(const Xyzz* p, int role) {
  QuadXyzz r;
  r.x = p->x;
  r.y = p->y;
  r.z = (role & 1) ? p->zzz : p->zz;
  return r;
}
__device__ __forceinline__ void quad_store(Xyzz* p, const QuadXyzz& v, int role) {
  if (role == 0) p->x = v.x;
  if (role == 1) p->zzz = v.z;
  if (role == 2) p->zz = v.z;
  if (role == 3) p->y = v.y;
}

// 2 p (dbl-2008-s-1); infinity (zz = zzz = 0) stays infinity, and so does a point with y = 0 become it.
__device__ __forceinline__ QuadXyzz quad_dbl(const QuadXyzz& p, int role) {
  const Fq u = dbl(p.y);
  const Fq s0 = quad_pick(role, u, p.x, u, p.x);
  const Fq m1 = quad_mul(s0, s0);                      // V | X^2 | V | X^2
  const Fq v = quad_get(m1, 0), xx = quad_get(m1, 1);
  const Fq m = add(dbl(xx), xx);
  const Fq m2 = quad_mul(quad_pick(role, p.x, u, p.z, m), quad_pick(role, v, v, v, m));  // S | W | ZZ' | M^2
  const Fq s = quad_get(m2, 0), w = quad_get(m2, 1), mm = quad_get(m2, 3);
  QuadXyzz r;
  r.x = sub(mm, dbl(s));
  const Fq t = sub(s, r.x);
  const Fq m3 = quad_mul(quad_pick(role, m, p.z, m, w), quad_pick(role, t, w, t, p.y));  // M (S - X') | ZZZ' | . | W Y
  r.y = sub(quad_get(m3, 0), quad_get(m3, 3));
  const Fq zz = quad_get(m2, 2), zzz = quad_get(m3, 1);
  r.z = quad_pick(role, zz, zzz, zz, zzz);
  return r;
}

// p + q (add-2008-s) with the exceptional cases.
__device__ __forceinline__ QuadXyzz quad_add(const QuadXyzz& p, const QuadXyzz& q, int role) {
  // lane 0: X1 ZZ2, lane 1: Y1 ZZZ2, lane 2: X2 ZZ1, lane 3: Y2 ZZZ1
  const Fq m1 = quad_mul(quad_pick(role, p.x, p.y, q.x, q.y), quad_pick(role, q.z, q.z, p.z, p.z));
  const Fq u1 = quad_get(m1, 0), s1 = quad_get(m1, 1);
  const Fq d = sub(quad_get(m1, 2), u1), e = sub(quad_get(m1, 3), s1);  // P, R
  const Fq m2 = quad_mul(quad_pick(role, d, e, p.z, p.z), quad_pick(role, d, e, q.z, q.z));  // P^2 | R^2 | ZZ1 ZZ2 | ZZZ1 ZZZ2
  const Fq pp = quad_get(m2, 0), rr = quad_get(m2, 1);
  const Fq m3 = quad_mul(quad_pick(role, d, u1, m2, m2), pp);                                  // PPP | Q | ZZ3 | .
  const Fq ppp = quad_get(m3, 0), t = quad_get(m3, 1);
  QuadXyzz r;
  r.x = sub(sub(rr, ppp), dbl(t));
  const Fq tx = sub(t, r.x);
  const Fq m4 = quad_mul(quad_pick(role, e, s1, e, m2), quad_pick(role, tx, ppp, tx, ppp));  // R (Q - X3) | S1 PPP | . | ZZZ3
  r.y = sub(quad_get(m4, 0), quad_get(m4, 1));
  const Fq zz = quad_get(m3, 2), zzz = quad_get(m4, 3);
  r.z = quad_pick(role, zz, zzz, zz, zzz);
  // every lane of a quad sees the same cases: zz and zzz are zero together
  const bool p_inf = p.z.is_zero(), q_inf = q.z.is_zero(), same_x = d.is_zero();
  const bool twice = !p_inf && !q_inf && same_x && e.is_zero();
  if (__any_sync(0xffffffffu, twice)) {  // rare: the whole warp doubles
    const QuadXyzz d2 = quad_dbl(p, role);
    if (twice) r = d2;
  }
  if (p_inf) r = q;
  if (q_inf) r = p;
  if (!p_inf && !q_inf && same_x && !e.is_zero()) r.z = Fq::zero();
  return r;
}

// a += b for points in shared memory, one copy of the code.
static __device__ __noinline__ void quad_add_to(Xyzz* a, const Xyzz* b, bool on) {
  const int role = threadIdx.x & 3;
  const QuadXyzz r = quad_add(quad_load(a, role), quad_load(b, role), role);
  __syncwarp();
  if (on) quad_store(a, r, role);
  __syncwarp();
}

}  // namespace zk
