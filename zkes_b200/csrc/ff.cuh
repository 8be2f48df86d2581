// 256-bit Montgomery arithmetic on 8 x 32-bit limbs for BN254 Fr (scalars) and Fq (coordinates).
//
// Replaces the arkworks Fp256 arithmetic the reference takes from ark-ff / ark-bn254
// (every + - * in src/crypto/sumcheck/linear_prover.rs and src/util/poly.rs).  The in-memory
// form is the same as arkworks': little-endian limbs of a*R mod p with R = 2^256.
//
// Device code is PTX carry chains (mad.lo.cc / madc.hi.cc pairs that ptxas fuses into 32x32+64
// wide multiply-adds).  A carry flag never crosses an asm statement: every chain is one
// statement.  The same functions compile for the host with plain 64-bit C so the algorithms
// built on the chains can be unit-tested without a GPU.
#pragma once
#include <cstdint>
#include <cstddef>

#if defined(__CUDACC__)
#define ZK_HD __host__ __device__ __forceinline__
#define ZK_D __device__ __forceinline__
#else
#define ZK_HD inline
#define ZK_D inline
#endif

namespace zk {

// ------------------------------------------------------------------------------------------
// Carry-chain primitives.  acc[] indices are constant after unrolling so everything stays in
// registers.

// (acc[2k+1]:acc[2k]) += x_k * y for k = 0..3 as one carry chain; returns the carry out of acc[7].
ZK_HD uint32_t madwide4_c(uint32_t* acc, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t y) {
#ifdef __CUDA_ARCH__
  uint32_t c;
  asm("mad.lo.cc.u32   %0, %9,  %13, %0;\n\t"
      "madc.hi.cc.u32  %1, %9,  %13, %1;\n\t"
      "madc.lo.cc.u32  %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32  %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32  %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32  %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32  %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32  %7, %12, %13, %7;\n\t"
      "addc.u32        %8, 0, 0;"
      : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
        "+r"(acc[7]), "=r"(c)
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
  return c;
#else
  const uint32_t x[4] = {x0, x1, x2, x3};
  uint64_t carry = 0;
  for (int k = 0; k < 4; k++) {
    uint64_t p = (uint64_t)x[k] * y;
    uint64_t lo = (uint64_t)acc[2 * k] + (uint32_t)p + carry;
    acc[2 * k] = (uint32_t)lo;
    uint64_t hi = (uint64_t)acc[2 * k + 1] + (p >> 32) + (lo >> 32);
    acc[2 * k + 1] = (uint32_t)hi;
    carry = hi >> 32;
  }
  return (uint32_t)carry;
#endif
}

// Same chain when the caller has proved that nothing is carried out of acc[7].
ZK_HD void madwide4(uint32_t* acc, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t y) {
#ifdef __CUDA_ARCH__
  asm("mad.lo.cc.u32   %0, %8,  %12, %0;\n\t"
      "madc.hi.cc.u32  %1, %8,  %12, %1;\n\t"
      "madc.lo.cc.u32  %2, %9,  %12, %2;\n\t"
      "madc.hi.cc.u32  %3, %9,  %12, %3;\n\t"
      "madc.lo.cc.u32  %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32  %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32  %6, %11, %12, %6;\n\t"
      "madc.hi.u32     %7, %11, %12, %7;"
      : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
        "+r"(acc[7])
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
#else
  (void)madwide4_c(acc, x0, x1, x2, x3, y);
#endif
}

// r = a + b over 8 limbs, returns the carry out.
ZK_HD uint32_t add8(uint32_t* r, const uint32_t* a, const uint32_t* b) {
#ifdef __CUDA_ARCH__
  uint32_t c;
  asm("add.cc.u32  %0, %9,  %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32    %8, 0, 0;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(c)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
  return c;
#else
  uint64_t c = 0;
  uint32_t t[8];
  for (int k = 0; k < 8; k++) {
    c += (uint64_t)a[k] + b[k];
    t[k] = (uint32_t)c;
    c >>= 32;
  }
  for (int k = 0; k < 8; k++) r[k] = t[k];
  return (uint32_t)c;
#endif
}

// r += b over sixteen limbs as one chain; the caller has proved no carry out.
ZK_HD void add16(uint32_t* r, const uint32_t* b) {
#ifdef __CUDA_ARCH__
  asm("add.cc.u32  %0, %0, %16;\n\t"
      "addc.cc.u32 %1, %1, %17;\n\t"
      "addc.cc.u32 %2, %2, %18;\n\t"
      "addc.cc.u32 %3, %3, %19;\n\t"
      "addc.cc.u32 %4, %4, %20;\n\t"
      "addc.cc.u32 %5, %5, %21;\n\t"
      "addc.cc.u32 %6, %6, %22;\n\t"
      "addc.cc.u32 %7, %7, %23;\n\t"
      "addc.cc.u32 %8, %8, %24;\n\t"
      "addc.cc.u32 %9, %9, %25;\n\t"
      "addc.cc.u32 %10, %10, %26;\n\t"
      "addc.cc.u32 %11, %11, %27;\n\t"
      "addc.cc.u32 %12, %12, %28;\n\t"
      "addc.cc.u32 %13, %13, %29;\n\t"
      "addc.cc.u32 %14, %14, %30;\n\t"
      "addc.u32    %15, %15, %31;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
        "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
      : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]),
        "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]), "r"(b[15]));
#else
  uint64_t c = 0;
  for (int k = 0; k < 16; k++) {
    c += (uint64_t)r[k] + b[k];
    r[k] = (uint32_t)c;
    c >>= 32;
  }
#endif
}

// r = a - b over 8 limbs, returns 1 when a < b (borrow), else 0.
ZK_HD uint32_t sub8(uint32_t* r, const uint32_t* a, const uint32_t* b) {
#ifdef __CUDA_ARCH__
  uint32_t c;
  asm("sub.cc.u32  %0, %9,  %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(c)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
  return c & 1u;
#else
  int64_t c = 0;
  uint32_t t[8];
  for (int k = 0; k < 8; k++) {
    c += (int64_t)a[k] - (int64_t)b[k];
    t[k] = (uint32_t)c;
    c >>= 32;  // arithmetic shift keeps the borrow as -1
  }
  for (int k = 0; k < 8; k++) r[k] = t[k];
  return c ? 1u : 0u;
#endif
}

// One row of a Montgomery product in the even / odd form (see mul): the carry out of the eight limbs of E belongs at limb
// 8 of the running value, which is O[7]; the caller has proved that nothing is carried out of there.
// E += (x0, x2, x4, x6) * y.
ZK_HD void row_even(uint32_t* E, uint32_t& o7, uint32_t x0, uint32_t x2, uint32_t x4, uint32_t x6, uint32_t y) {
#ifdef __CUDA_ARCH__
  asm("mad.lo.cc.u32   %0, %9,  %13, %0;\n\t"
      "madc.hi.cc.u32  %1, %9,  %13, %1;\n\t"
      "madc.lo.cc.u32  %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32  %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32  %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32  %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32  %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32  %7, %12, %13, %7;\n\t"
      "addc.u32        %8, %8, 0;"
      : "+r"(E[0]), "+r"(E[1]), "+r"(E[2]), "+r"(E[3]), "+r"(E[4]), "+r"(E[5]), "+r"(E[6]), "+r"(E[7]), "+r"(o7)
      : "r"(x0), "r"(x2), "r"(x4), "r"(x6), "r"(y));
#else
  o7 += madwide4_c(E, x0, x2, x4, x6, y);
#endif
}

// The division by 2^32 together with the next row's odd products: with E[0] = 0 the value (E + 2^32 O) / 2^32 has the
// even part O + E[1] and the odd part E[2..7].  Only limb 0 of the even part is added here; its carry belongs at limb 1,
// where the odd part begins, so it is the carry into the chain that adds (x1, x3, x5, x7) * y to the odd part.
// On return O is the new even part and E the new odd part.
// e8: the ninth limb of the old even part, for the callers that have one.
ZK_HD void row_odd_shift(uint32_t* E, uint32_t* O, uint32_t x1, uint32_t x3, uint32_t x5, uint32_t x7, uint32_t y,
                         uint32_t e8 = 0) {
  uint32_t t[8];
#ifdef __CUDA_ARCH__
  asm("add.cc.u32      %8, %8, %9;\n\t"
      "madc.lo.cc.u32  %0, %16, %20, %10;\n\t"
      "madc.hi.cc.u32  %1, %16, %20, %11;\n\t"
      "madc.lo.cc.u32  %2, %17, %20, %12;\n\t"
      "madc.hi.cc.u32  %3, %17, %20, %13;\n\t"
      "madc.lo.cc.u32  %4, %18, %20, %14;\n\t"
      "madc.hi.cc.u32  %5, %18, %20, %15;\n\t"
      "madc.lo.cc.u32  %6, %19, %20, %21;\n\t"
      "madc.hi.u32     %7, %19, %20, 0;"
      : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "+r"(O[0])
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(x1), "r"(x3), "r"(x5), "r"(x7), "r"(y),
        "r"(e8));
#else
  uint64_t c = (uint64_t)O[0] + E[1];
  O[0] = (uint32_t)c;
  c >>= 32;
  const uint32_t x[4] = {x1, x3, x5, x7};
  for (int k = 0; k < 4; k++) {
    const uint64_t p = (uint64_t)x[k] * y;
    c += (uint64_t)(uint32_t)p + (k < 3 ? E[2 * k + 2] : e8);
    t[2 * k] = (uint32_t)c;
    c >>= 32;
    c += (p >> 32) + (k < 3 ? E[2 * k + 3] : 0u);
    t[2 * k + 1] = (uint32_t)c;
    c >>= 32;
  }
#endif
#pragma unroll
  for (int k = 0; k < 8; k++) E[k] = t[k];
}

// The same division when the next row's multiplier m = (new even limb 0) * inv depends on it (reduction rows without a
// product): returns m.
ZK_HD uint32_t redc_odd_shift(uint32_t* E, uint32_t* O, uint32_t x1, uint32_t x3, uint32_t x5, uint32_t x7, uint32_t inv,
                              uint32_t e8 = 0) {
  const uint32_t m = (O[0] + E[1]) * inv;
  row_odd_shift(E, O, x1, x3, x5, x7, m, e8);
  return m;
}

// Last division by 2^32: r = O + (E >> 32) with E[0] = 0; the caller has proved no carry out.
ZK_HD void row_finish(uint32_t* r, const uint32_t* E, const uint32_t* O) {
  uint32_t s[8];
#pragma unroll
  for (int k = 0; k < 7; k++) s[k] = E[k + 1];
  s[7] = 0;
  (void)add8(r, O, s);
}

// ------------------------------------------------------------------------------------------
// Field parameters.  mod(i), r2(i), one(i) return limb i; loops over them are fully unrolled
// so the values become immediates.

struct FrParams {  // BN254 scalar field
  static ZK_HD constexpr uint32_t mod(int i) {
    constexpr uint32_t m[8] = {0xf0000001u, 0x43e1f593u, 0x79b97091u, 0x2833e848u,
                               0x8181585du, 0xb85045b6u, 0xe131a029u, 0x30644e72u};
    return m[i];
  }
  static constexpr uint32_t inv = 0xefffffffu;  // -mod^-1 mod 2^32
  static ZK_HD constexpr uint32_t r2(int i) {   // R^2 mod p
    constexpr uint32_t m[8] = {0xae216da7u, 0x1bb8e645u, 0xe35c59e3u, 0x53fe3ab1u,
                               0x53bb8085u, 0x8c49833du, 0x7f4e44a5u, 0x0216d0b1u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t one(int i) {  // R mod p
    constexpr uint32_t m[8] = {0x4ffffffbu, 0xac96341cu, 0x9f60cd29u, 0x36fc7695u,
                               0x7879462eu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t r3(int i) {  // R^3 mod p
    constexpr uint32_t m[8] = {0xb4bf0040u, 0x5e94d8e1u, 0x1cfbb6b8u, 0x2a489cbeu,
                               0xa19fcfedu, 0x893cc664u, 0x7fcc657cu, 0x0cf8594bu};
    return m[i];
  }
};

struct FqParams {  // BN254 base field
  static ZK_HD constexpr uint32_t mod(int i) {
    constexpr uint32_t m[8] = {0xd87cfd47u, 0x3c208c16u, 0x6871ca8du, 0x97816a91u,
                               0x8181585du, 0xb85045b6u, 0xe131a029u, 0x30644e72u};
    return m[i];
  }
  static constexpr uint32_t inv = 0xe4866389u;
  static ZK_HD constexpr uint32_t r2(int i) {
    constexpr uint32_t m[8] = {0x538afa89u, 0xf32cfc5bu, 0xd44501fbu, 0xb5e71911u,
                               0x0a417ff6u, 0x47ab1effu, 0xcab8351fu, 0x06d89f71u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t one(int i) {
    constexpr uint32_t m[8] = {0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u,
                               0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t r3(int i) {
    constexpr uint32_t m[8] = {0xda1530dfu, 0xb1cd6dafu, 0xa7283db6u, 0x62f210e6u,
                               0x0ada0afbu, 0xef7f0b0cu, 0x2d592544u, 0x20fd6e90u};
    return m[i];
  }
};

// ------------------------------------------------------------------------------------------
template <class P>
struct alignas(16) Fp {
  uint32_t v[8];

  static ZK_HD Fp zero() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = 0;
    return r;
  }
  static ZK_HD Fp one() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = P::one(i);
    return r;
  }
  static ZK_HD Fp modulus() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = P::mod(i);
    return r;
  }
  static ZK_HD Fp r2() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = P::r2(i);
    return r;
  }
  static ZK_HD Fp r3() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = P::r3(i);
    return r;
  }
  ZK_HD bool is_zero() const {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) o |= v[i];
    return o == 0;
  }
  ZK_HD bool operator==(const Fp& b) const {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) o |= v[i] ^ b.v[i];
    return o == 0;
  }
  ZK_HD bool operator!=(const Fp& b) const { return !(*this == b); }
};

// r = (a < mod) ? a : a - mod, for a < 2*mod (carry = the 257th bit of a).
template <class P>
ZK_HD void final_sub(uint32_t* a, uint32_t carry) {
  uint32_t d[8], m[8];
#pragma unroll
  for (int i = 0; i < 8; i++) m[i] = P::mod(i);
  uint32_t borrow = sub8(d, a, m);
  // keep the difference when it did not borrow, or when the sum had overflowed 2^256
  bool take = (borrow == 0) | (carry != 0);
#pragma unroll
  for (int i = 0; i < 8; i++) a[i] = take ? d[i] : a[i];
}

template <class P>
ZK_HD Fp<P> add(const Fp<P>& a, const Fp<P>& b) {
  Fp<P> r;
  uint32_t c = add8(r.v, a.v, b.v);
  final_sub<P>(r.v, c);
  return r;
}

template <class P>
ZK_HD Fp<P> sub(const Fp<P>& a, const Fp<P>& b) {
  Fp<P> r;
  uint32_t borrow = sub8(r.v, a.v, b.v);
  uint32_t m[8], t[8];
#pragma unroll
  for (int i = 0; i < 8; i++) m[i] = borrow ? P::mod(i) : 0u;
  (void)add8(t, r.v, m);
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = t[i];
  return r;
}

template <class P>
ZK_HD Fp<P> neg(const Fp<P>& a) {
  return sub(Fp<P>::zero(), a);
}

template <class P>
ZK_HD Fp<P> dbl(const Fp<P>& a) {
  return add(a, a);
}

// Montgomery product a*b/R mod p.  `a` must be < p; `b` may be any 256-bit value.
//
// Operand scanning with two accumulators: E holds the 64-bit columns that start at even
// limbs, O the columns that start at odd limbs (O is offset by one limb), so every row of
// partial products is a chain of non-overlapping 32x32+64 multiply-adds.  After the
// reduction row the low limb of E is zero; dividing by 2^32 turns the odd columns into the
// even ones and vice versa, so the two arrays swap roles instead of shifting, and the one limb
// that has to move (E[1] onto O[0]) is the head of the next row's odd chain, which takes its carry.
// What bounds it is the multiply pipe: 128 wide multiply-adds.  Moving E[1] by an eight-limb addition per row and
// catching the carries in a ninth limb cost some 70 more instructions a product: 83 G products/s (two chains per thread,
// 16 warps per SM) against 105 G/s as it is.
// Bounds: the running value E + 2^32*O stays below a + p, and below 2^32 (a + p) < 2^288 inside a
// row, so eight limbs of E and of O hold it, with E's carry put into O[7].
template <class P>
ZK_HD Fp<P> mul_rows(const Fp<P>& a, const Fp<P>& b) {
  uint32_t X[8], Y[8];
#pragma unroll
  for (int i = 0; i < 8; i++) X[i] = Y[i] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t* E = (i & 1) ? Y : X;  // the even columns of this row; the arrays swap roles from row to row
    uint32_t* O = (i & 1) ? X : Y;
    const uint32_t bi = b.v[i];
    if (i == 0)
      madwide4(O, a.v[1], a.v[3], a.v[5], a.v[7], bi);
    else
      row_odd_shift(O, E, a.v[1], a.v[3], a.v[5], a.v[7], bi);
    row_even(E, O[7], a.v[0], a.v[2], a.v[4], a.v[6], bi);
    const uint32_t m = E[0] * P::inv;
    madwide4(O, P::mod(1), P::mod(3), P::mod(5), P::mod(7), m);
    row_even(E, O[7], P::mod(0), P::mod(2), P::mod(4), P::mod(6), m);
  }
  Fp<P> r;  // after eight rows the even columns are in Y, the odd ones in X; the value is below 2p
  row_finish(r.v, Y, X);
  final_sub<P>(r.v, 0);
  return r;
}

// The same product on the host: four 64-bit limbs, which read the eight 32-bit ones in place (R = 2^256 either way).  A CPU
// core takes about 25 ns for it and 240 ns for the rows above; the multiplier table of a challenge (make_fixed_mul, 17
// products) is made before every fold.
template <class P>
inline Fp<P> mul_host(const Fp<P>& a, const Fp<P>& b) {
  typedef unsigned __int128 u128;
  uint64_t x[4], y[4], p[4], t[6] = {0, 0, 0, 0, 0, 0};
  for (int i = 0; i < 4; i++) {
    x[i] = (uint64_t)a.v[2 * i] | ((uint64_t)a.v[2 * i + 1] << 32);
    y[i] = (uint64_t)b.v[2 * i] | ((uint64_t)b.v[2 * i + 1] << 32);
    p[i] = (uint64_t)P::mod(2 * i) | ((uint64_t)P::mod(2 * i + 1) << 32);
  }
  // -p^-1 mod 2^64 from its low half by one Newton step: with n = -p^-1 mod 2^32, n (2 + n p) is it mod 2^64
  const uint64_t n32 = P::inv, inv = n32 * (2 + n32 * p[0]);
  for (int i = 0; i < 4; i++) {
    u128 c = 0;
    for (int j = 0; j < 4; j++) {
      c += (u128)x[j] * y[i] + t[j];
      t[j] = (uint64_t)c;
      c >>= 64;
    }
    c += t[4];
    t[4] = (uint64_t)c;
    t[5] = (uint64_t)(c >> 64);
    const uint64_t q = t[0] * inv;
    c = ((u128)q * p[0] + t[0]) >> 64;
    for (int j = 1; j < 4; j++) {
      c += (u128)q * p[j] + t[j];
      t[j - 1] = (uint64_t)c;
      c >>= 64;
    }
    c += t[4];
    t[3] = (uint64_t)c;
    t[4] = t[5] + (uint64_t)(c >> 64);
  }
  uint64_t d[4], borrow = 0;  // the value is below 2p < 2^256: subtract p unless that borrows
  for (int i = 0; i < 4; i++) {
    const u128 v = (u128)t[i] - p[i] - borrow;
    d[i] = (uint64_t)v;
    borrow = (uint64_t)(v >> 64) & 1;
  }
  const uint64_t keep = 0 - borrow;
  Fp<P> r;
  for (int i = 0; i < 4; i++) {
    const uint64_t v = (t[i] & keep) | (d[i] & ~keep);
    r.v[2 * i] = (uint32_t)v;
    r.v[2 * i + 1] = (uint32_t)(v >> 32);
  }
  return r;
}

template <class P>
ZK_HD Fp<P> mul(const Fp<P>& a, const Fp<P>& b) {
#ifdef __CUDA_ARCH__
  return mul_rows(a, b);
#else
  return mul_host(a, b);
#endif
}

// Multiplication by a value that is fixed for a whole launch (a round challenge).
//
// For a fixed x the table holds c[j] = x * 2^(32 j + 64) mod p as plain integers.  Then for any
// d in Montgomery form, sum_j d_j c[j] = 2^64 * (x d) (mod p) needs 8 rows of 8 multiply-adds
// and no 512-bit intermediate; two Montgomery rounds remove the factor 2^64 and bring the
// 291-bit sum below 2^227 + p, so one conditional subtraction completes it: 82 multiply-adds
// against 136 for a general product.  The result is x*d in Montgomery form (d's own factor R).
template <class P>
struct FixedMul {
  uint32_t c[8][8];
};

// Build the table from x in Montgomery form (host or device).
template <class P>
ZK_HD FixedMul<P> make_fixed_mul(const Fp<P>& x_mont) {
  FixedMul<P> t;
  Fp<P> two64 = Fp<P>::zero();
  two64.v[2] = 1;
  Fp<P> two32 = Fp<P>::zero();
  two32.v[1] = 1;
  const Fp<P> step = to_mont(two32);  // 2^32 * R
  Fp<P> cur = mul(x_mont, two64);     // x * 2^64 as a plain integer mod p
  for (int j = 0; j < 8; j++) {
    for (int k = 0; k < 8; k++) t.c[j][k] = cur.v[k];
    cur = mul(cur, step);             // times 2^32
  }
  return t;
}

// The two Montgomery rounds: (E + 2^32 O) / 2^64 mod p for a sum below 3 * 2^289 held in nine even and nine odd limbs.
// After the first division the value is below 2^260, so the second round stays below 2^288 and its odd part needs eight
// limbs; the result before the subtraction is below 3 * 2^225 + p < 2p.
template <class P>
ZK_HD Fp<P> fixed_finish(uint32_t* E, uint32_t* O) {
  uint32_t m = E[0] * P::inv;
  row_even(O, O[8], P::mod(1), P::mod(3), P::mod(5), P::mod(7), m);
  row_even(E, E[8], P::mod(0), P::mod(2), P::mod(4), P::mod(6), m);
  m = redc_odd_shift(E, O, P::mod(1), P::mod(3), P::mod(5), P::mod(7), P::inv, E[8]);
  row_even(O, O[8], P::mod(0), P::mod(2), P::mod(4), P::mod(6), m);
  Fp<P> r;
  (void)add8(r.v, O + 1, E);
  final_sub<P>(r.v, 0);
  return r;
}

template <class P>
ZK_HD Fp<P> mul_fixed(const FixedMul<P>& t, const Fp<P>& d) {
  uint32_t E[9], O[9];
#pragma unroll
  for (int i = 0; i < 9; i++) E[i] = O[i] = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    row_even(E, E[8], t.c[j][0], t.c[j][2], t.c[j][4], t.c[j][6], d.v[j]);
    row_even(O, O[8], t.c[j][1], t.c[j][3], t.c[j][5], t.c[j][7], d.v[j]);
  }
  return fixed_finish<P>(E, O);
}

// t0 * d0 + t1 * d1 + t2 * d2 for three launch-constant multipliers in one accumulation: the
// three 291-bit row sums share the accumulators and one pair of Montgomery rounds, 210
// multiply-adds in all.  The d's may be any 256-bit values (unreduced differences).
template <class P>
ZK_HD Fp<P> mul_fixed3(const FixedMul<P>& t0, const uint32_t* d0, const FixedMul<P>& t1, const uint32_t* d1,
                       const FixedMul<P>& t2, const uint32_t* d2) {
  uint32_t E[9], O[9];
#pragma unroll
  for (int i = 0; i < 9; i++) E[i] = O[i] = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    row_even(E, E[8], t0.c[j][0], t0.c[j][2], t0.c[j][4], t0.c[j][6], d0[j]);
    row_even(O, O[8], t0.c[j][1], t0.c[j][3], t0.c[j][5], t0.c[j][7], d0[j]);
    row_even(E, E[8], t1.c[j][0], t1.c[j][2], t1.c[j][4], t1.c[j][6], d1[j]);
    row_even(O, O[8], t1.c[j][1], t1.c[j][3], t1.c[j][5], t1.c[j][7], d1[j]);
    row_even(E, E[8], t2.c[j][0], t2.c[j][2], t2.c[j][4], t2.c[j][6], d2[j]);
    row_even(O, O[8], t2.c[j][1], t2.c[j][3], t2.c[j][5], t2.c[j][7], d2[j]);
  }
  return fixed_finish<P>(E, O);
}

// a + p - b without the conditional correction: any value congruent to a - b below 2p.
template <class P>
ZK_HD void sub_lazy(uint32_t* out, const Fp<P>& a, const Fp<P>& b) {
  uint32_t m[8], t[8];
#pragma unroll
  for (int i = 0; i < 8; i++) m[i] = P::mod(i);
  (void)add8(t, a.v, m);
  (void)sub8(out, t, b.v);
}

// 512-bit integer used for lazily reduced sums of products.
struct Wide {
  uint32_t v[16];
};

// Full 512-bit product of two 256-bit integers (no reduction).
// Even/odd column accumulators over 16 limbs; rows in increasing order so the limb that
// receives a row's carry has not been written before.
ZK_HD void mul_wide(Wide& out, const uint32_t* a, const uint32_t* b) {
  uint32_t E[16], O[16];  // O[k] sits at limb position k+1
#pragma unroll
  for (int i = 0; i < 16; i++) E[i] = O[i] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if ((i & 1) == 0) {
      E[i + 8] = madwide4_c(E + i, a[0], a[2], a[4], a[6], b[i]);
      madwide4(O + i, a[1], a[3], a[5], a[7], b[i]);  // top carry is zero: value < 2^(32(i+9))
    } else {
      O[i + 7] = madwide4_c(O + i - 1, a[0], a[2], a[4], a[6], b[i]);
      madwide4(E + i + 1, a[1], a[3], a[5], a[7], b[i]);
    }
  }
  // out = E + (O << 32); the product fits 512 bits
  uint32_t S[16];
  S[0] = 0;
#pragma unroll
  for (int k = 0; k < 16; k++) out.v[k] = E[k];
#pragma unroll
  for (int k = 1; k < 16; k++) S[k] = O[k - 1];
  add16(out.v, S);
}

// (acc[2k+1]:acc[2k]) += x_k * y for k < N as one chain, its carry added to acc[2N].
template <int N>
ZK_HD void madwide_n(uint32_t* acc, const uint32_t* x, uint32_t y) {  // x_k = x[2k]
  if constexpr (N == 4) {
    row_even(acc, acc[8], x[0], x[2], x[4], x[6], y);
  } else if constexpr (N == 3) {
#ifdef __CUDA_ARCH__
    asm("mad.lo.cc.u32   %0, %7, %10, %0;\n\t"
        "madc.hi.cc.u32  %1, %7, %10, %1;\n\t"
        "madc.lo.cc.u32  %2, %8, %10, %2;\n\t"
        "madc.hi.cc.u32  %3, %8, %10, %3;\n\t"
        "madc.lo.cc.u32  %4, %9, %10, %4;\n\t"
        "madc.hi.cc.u32  %5, %9, %10, %5;\n\t"
        "addc.u32        %6, %6, 0;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6])
        : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(y));
#endif
  } else if constexpr (N == 2) {
#ifdef __CUDA_ARCH__
    asm("mad.lo.cc.u32   %0, %5, %7, %0;\n\t"
        "madc.hi.cc.u32  %1, %5, %7, %1;\n\t"
        "madc.lo.cc.u32  %2, %6, %7, %2;\n\t"
        "madc.hi.cc.u32  %3, %6, %7, %3;\n\t"
        "addc.u32        %4, %4, 0;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4])
        : "r"(x[0]), "r"(x[2]), "r"(y));
#endif
  } else if constexpr (N == 1) {
#ifdef __CUDA_ARCH__
    asm("mad.lo.cc.u32   %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32  %1, %3, %4, %1;\n\t"
        "addc.u32        %2, %2, 0;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2])
        : "r"(x[0]), "r"(y));
#endif
  }
#ifndef __CUDA_ARCH__
  if constexpr (N < 4) {
    uint64_t c = 0;
    for (int k = 0; k < N; k++) {
      const uint64_t p = (uint64_t)x[2 * k] * y;
      c += (uint64_t)acc[2 * k] + (uint32_t)p;
      acc[2 * k] = (uint32_t)c;
      c >>= 32;
      c += (uint64_t)acc[2 * k + 1] + (p >> 32);
      acc[2 * k + 1] = (uint32_t)c;
      c >>= 32;
    }
    acc[2 * N] += (uint32_t)c;
  }
#endif
}

// (acc[2k+1]:acc[2k]) += x[k]^2 for k < 8 as one chain; the caller has proved no carry out.
ZK_HD void add_squares(uint32_t* acc, const uint32_t* x) {
#ifdef __CUDA_ARCH__
  asm("mad.lo.cc.u32   %0, %16, %16, %0;\n\t"
      "madc.hi.cc.u32  %1, %16, %16, %1;\n\t"
      "madc.lo.cc.u32  %2, %17, %17, %2;\n\t"
      "madc.hi.cc.u32  %3, %17, %17, %3;\n\t"
      "madc.lo.cc.u32  %4, %18, %18, %4;\n\t"
      "madc.hi.cc.u32  %5, %18, %18, %5;\n\t"
      "madc.lo.cc.u32  %6, %19, %19, %6;\n\t"
      "madc.hi.cc.u32  %7, %19, %19, %7;\n\t"
      "madc.lo.cc.u32  %8, %20, %20, %8;\n\t"
      "madc.hi.cc.u32  %9, %20, %20, %9;\n\t"
      "madc.lo.cc.u32  %10, %21, %21, %10;\n\t"
      "madc.hi.cc.u32  %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32  %12, %22, %22, %12;\n\t"
      "madc.hi.cc.u32  %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32  %14, %23, %23, %14;\n\t"
      "madc.hi.u32     %15, %23, %23, %15;"
      : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]), "+r"(acc[7]),
        "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]), "+r"(acc[14]), "+r"(acc[15])
      : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]));
#else
  uint64_t c = 0;
  for (int k = 0; k < 8; k++) {
    const uint64_t p = (uint64_t)x[k] * x[k];
    c += (uint64_t)acc[2 * k] + (uint32_t)p;
    acc[2 * k] = (uint32_t)c;
    c >>= 32;
    c += (uint64_t)acc[2 * k + 1] + (p >> 32);
    acc[2 * k + 1] = (uint32_t)c;
    c >>= 32;
  }
#endif
}

// a^2 over 512 bits: the 28 products of unequal limbs once, doubled, and the eight squares: 36 multiply-adds for 64.
// Even / odd columns as in mul_wide; a row's carry lands in a limb that holds nothing but carries so far.
ZK_HD void sqr_wide(Wide& out, const uint32_t* a) {
  uint32_t E[18], O[18];  // O[k] sits at limb position k+1
#pragma unroll
  for (int i = 0; i < 18; i++) E[i] = O[i] = 0;
  madwide_n<4>(O + 0, a + 1, a[0]);   // columns 1 3 5 7
  madwide_n<3>(E + 2, a + 2, a[0]);   // 2 4 6
  madwide_n<3>(O + 2, a + 2, a[1]);   // 3 5 7
  madwide_n<3>(E + 4, a + 3, a[1]);   // 4 6 8
  madwide_n<3>(O + 4, a + 3, a[2]);   // 5 7 9
  madwide_n<2>(E + 6, a + 4, a[2]);   // 6 8
  madwide_n<2>(O + 6, a + 4, a[3]);   // 7 9
  madwide_n<2>(E + 8, a + 5, a[3]);   // 8 10
  madwide_n<2>(O + 8, a + 5, a[4]);   // 9 11
  madwide_n<1>(E + 10, a + 6, a[4]);  // 10
  madwide_n<1>(O + 10, a + 6, a[5]);  // 11
  madwide_n<1>(E + 12, a + 7, a[5]);  // 12
  madwide_n<1>(O + 12, a + 7, a[6]);  // 13
  uint32_t S[16];
  S[0] = 0;
#pragma unroll
  for (int k = 0; k < 16; k++) out.v[k] = E[k];
#pragma unroll
  for (int k = 1; k < 16; k++) S[k] = O[k - 1];
  add16(out.v, S);
#pragma unroll
  for (int k = 0; k < 16; k++) S[k] = out.v[k];
  add16(out.v, S);
  add_squares(out.v, a);
}

// acc += w over 16 limbs (caller keeps acc below 2^512).
ZK_HD void wide_add(Wide& acc, const Wide& w) { add16(acc.v, w.v); }

// Keep acc < p * 2^256 by subtracting p from the upper half when it is >= p.
// Valid while acc < 2 * p * 2^256, i.e. after adding at most 5 products of reduced operands
// to an accumulator that was below p * 2^256 (5 p^2 < p * 2^256 for both BN254 fields).
template <class P>
ZK_HD void wide_trim(Wide& acc) {
  final_sub<P>(acc.v + 8, 0);
}
constexpr int kLazyProducts = 5;

// Montgomery reduction of T < p * 2^256: returns T / 2^256 mod p, fully reduced.
// Only the low half goes through the reduction rows: (T_lo + M p) / 2^256 <= p, and the
// upper half (< p) is added afterwards, so one conditional subtraction finishes.
template <class P>
ZK_HD Fp<P> redc(const Wide& t) {
  uint32_t X[8], Y[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    X[i] = t.v[i];
    Y[i] = 0;
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t* E = (i & 1) ? Y : X;
    uint32_t* O = (i & 1) ? X : Y;
    uint32_t m;
    if (i == 0) {
      m = E[0] * P::inv;
      madwide4(O, P::mod(1), P::mod(3), P::mod(5), P::mod(7), m);
    } else {
      m = redc_odd_shift(O, E, P::mod(1), P::mod(3), P::mod(5), P::mod(7), P::inv);
    }
    row_even(E, O[7], P::mod(0), P::mod(2), P::mod(4), P::mod(6), m);
  }
  Fp<P> r;
  uint32_t lo[8];
  row_finish(lo, Y, X);                   // <= p
  uint32_t c = add8(r.v, lo, t.v + 8);    // < 2p < 2^256
  final_sub<P>(r.v, c);
  return r;
}

// Montgomery square: 108 multiply-adds for the 136 of a product (with the reduction alone in from_mont, 1.9 % of a KZH2 commitment
// of 2^24 values).
template <class P>
ZK_HD Fp<P> sqr(const Fp<P>& a) {
#ifdef __CUDA_ARCH__
  Wide t;
  sqr_wide(t, a.v);
  return redc<P>(t);
#else
  return mul(a, a);
#endif
}

// Into / out of Montgomery form.
template <class P>
ZK_HD Fp<P> to_mont(const Fp<P>& canonical) {
  return mul(Fp<P>::r2(), canonical);
}
template <class P>
ZK_HD Fp<P> from_mont(const Fp<P>& a) {
#ifdef __CUDA_ARCH__
  Wide t;  // the reduction alone: half the multiply-adds of a product by one (k_msm_bits: 297 -> 208 us)
#pragma unroll
  for (int i = 0; i < 8; i++) {
    t.v[i] = a.v[i];
    t.v[i + 8] = 0;
  }
  return redc<P>(t);
#else
  Fp<P> one = Fp<P>::zero();  // four 64-bit limbs beat the 32-bit reduction: 25 ns against 68
  one.v[0] = 1;
  return mul_host(a, one);
#endif
}

// Small unsigned integer as a field element (Montgomery form).
template <class P>
ZK_HD Fp<P> from_u32(uint32_t x) {
  Fp<P> c = Fp<P>::zero();
  c.v[0] = x;
  return to_mont(c);
}

// Multiplicative inverse (0 maps to 0) by the division steps of Bernstein and Yang, "Fast constant-time gcd computation
// and modular inversion" (2019), with the counter delta started at 1/2 as P. Wuille and G. Maxwell proposed ("Bounds on
// divsteps iterations in safegcd", 2021: 590 steps suffice for 256-bit inputs, 741 as in the paper).  Fermat's power is a chain of some 380 dependent
// products; here the low words alone decide thirty steps, which are collected in a 2x2 matrix and then applied to the
// whole numbers, so an inversion is about 18 batches of thirty 32-bit steps and two matrix products over nine limbs.
// k_normalize on 4096 points (an inversion per thread): 22 us against 173 us.
//
// Numbers are nine limbs of 30 bits, the lower eight in [0, 2^30), the top one signed.  f and g stay within (-p, p].
// d and e satisfy d a = f and e a = g (mod p); a batch takes each to (u d + v e + m p) / 2^30 with |u| + |v| <= 2^30 and
// m in [-2^29, 2^29) chosen to make the division exact, so they grow by at most p/2 a batch and stay below 13 p in
// absolute value: no reduction is needed before the end.  25 batches (750 steps) are more than either bound;
// the loop ends as soon as g is zero.
template <class P>
ZK_HD int32_t mod30(int i) {  // limb i of p in base 2^30; a constant after unrolling
  const int bit = 30 * i, k = bit >> 5, sh = bit & 31;
  uint32_t v = P::mod(k) >> sh;
  if (sh > 2 && k < 7) v |= P::mod(k + 1) << (32 - sh);
  return (int32_t)(v & 0x3fffffffu);
}

template <class P>
#if defined(__CUDACC__)
static __host__ __device__ __noinline__ Fp<P> inverse(const Fp<P> a) {
#else
inline Fp<P> inverse(const Fp<P> a) {
#endif
  constexpr uint32_t kMask = 0x3fffffffu;
  int32_t f[9], g[9], d[9], e[9];
#pragma unroll
  for (int i = 0; i < 9; i++) {
    const int bit = 30 * i, k = bit >> 5, sh = bit & 31;
    uint32_t v = a.v[k] >> sh;
    if (sh > 2 && k < 7) v |= a.v[k + 1] << (32 - sh);
    g[i] = (int32_t)(v & kMask);
    f[i] = mod30<P>(i);
    d[i] = 0;
    e[i] = i == 0;
  }
  int32_t z = 0;  // delta - 1/2
#pragma unroll 1
  for (int batch = 0; batch < 25; batch++) {
    int32_t any = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) any |= g[i];
    if (any == 0) break;
    // thirty steps on the low words: (f, g) <- (f, g + c f) / (1, 2) with c = 0 for even g, and for odd g c = 1, or
    // c = -1 with f replaced by the old g when delta is positive
    uint32_t fl = (uint32_t)f[0] | ((uint32_t)f[1] << 30), gl = (uint32_t)g[0] | ((uint32_t)g[1] << 30);
    int32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 6
    for (int i = 0; i < 30; i++) {
      const bool odd = gl & 1u, swap = odd && z >= 0;
      const int32_t c = odd ? (swap ? -1 : 1) : 0;
      const uint32_t fn = swap ? gl : fl;
      const int32_t un = swap ? q : u, vn = swap ? r : v;
      gl = (gl + (uint32_t)c * fl) >> 1;
      q += c * u;
      r += c * v;
      fl = fn;
      u = un * 2;
      v = vn * 2;
      z = swap ? -z : z + 1;
    }
    // apply the matrix to f, g (exact) and to d, e (exact after adding a multiple of p)
    int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0], cg = (int64_t)q * f[0] + (int64_t)r * g[0];
    int64_t cd = (int64_t)u * d[0] + (int64_t)v * e[0], ce = (int64_t)q * d[0] + (int64_t)r * e[0];
    const int32_t md = (int32_t)(((uint32_t)cd * P::inv) << 2) >> 2, me = (int32_t)(((uint32_t)ce * P::inv) << 2) >> 2;
    cd += (int64_t)md * mod30<P>(0);
    ce += (int64_t)me * mod30<P>(0);
    cf >>= 30;
    cg >>= 30;
    cd >>= 30;
    ce >>= 30;
#pragma unroll
    for (int i = 1; i < 9; i++) {
      cf += (int64_t)u * f[i] + (int64_t)v * g[i];
      cg += (int64_t)q * f[i] + (int64_t)r * g[i];
      cd += (int64_t)u * d[i] + (int64_t)v * e[i] + (int64_t)md * mod30<P>(i);
      ce += (int64_t)q * d[i] + (int64_t)r * e[i] + (int64_t)me * mod30<P>(i);
      f[i - 1] = (int32_t)((uint32_t)cf & kMask);
      g[i - 1] = (int32_t)((uint32_t)cg & kMask);
      d[i - 1] = (int32_t)((uint32_t)cd & kMask);
      e[i - 1] = (int32_t)((uint32_t)ce & kMask);
      cf >>= 30;
      cg >>= 30;
      cd >>= 30;
      ce >>= 30;
    }
    f[8] = (int32_t)cf;
    g[8] = (int32_t)cg;
    d[8] = (int32_t)cd;
    e[8] = (int32_t)ce;
  }
  // f = +-1 (f = p and d = 0 for a = 0): the inverse is f d.  16 p + f d lies in (3 p, 29 p); conditional subtractions
  // of 16 p, 8 p and 4 p bring it below 4 p < 2^256, which the product accepts as its second operand.
  const int32_t sign = f[8] < 0 ? -1 : 1;
  int64_t carry = 0;
#pragma unroll
  for (int i = 0; i < 9; i++) {
    carry += (int64_t)sign * d[i] + ((int64_t)mod30<P>(i) << 4);
    d[i] = (int32_t)((uint32_t)carry & (i < 8 ? kMask : 0xffffffffu));
    carry >>= 30;
  }
#pragma unroll
  for (int k = 4; k >= 2; k--) {
    int64_t borrow = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) {
      borrow += (int64_t)d[i] - ((int64_t)mod30<P>(i) << k);
      e[i] = (int32_t)((uint32_t)borrow & (i < 8 ? kMask : 0xffffffffu));
      borrow >>= 30;
    }
    const bool keep = e[8] >= 0;
#pragma unroll
    for (int i = 0; i < 9; i++) d[i] = keep ? e[i] : d[i];
  }
  Fp<P> y;
#pragma unroll
  for (int k = 0; k < 8; k++) {  // 32 bits from bit 32 k of the 30-bit limbs
    const int bit = 32 * k, i = bit / 30, sh = bit % 30;
    uint32_t v = (uint32_t)d[i] >> sh;
    v |= (uint32_t)d[i + 1] << (30 - sh);
    if (sh > 28 && i + 2 < 9) v |= (uint32_t)d[i + 2] << (60 - sh);
    y.v[k] = v;
  }
  return mul(Fp<P>::r3(), y);  // (a R)^-1 R^3 / R = a^-1 R
}

using Fr = Fp<FrParams>;
using Fq = Fp<FqParams>;

}  // namespace zk
