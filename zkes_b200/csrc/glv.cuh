// The endomorphism of the curve: BN254's G1 has phi(x, y) = (beta x, y) = lambda (x, y) with beta^3 = 1 mod q, lambda^3 = 1 mod r, and the
// lattice of (u, v) with u + v lambda = 0 mod r has a basis v1 = (a1, b1), v2 = (a2, b2) of vectors of length about sqrt(r).  A scalar
// k = k1 + k2 lambda with k1, k2 of 126 bits (kEndoMagnitude): (k1, k2) = (k, 0) - c1 v1 - c2 v2, c1 and c2 the nearest integers to b2 k / r and
// -b1 k / r (Gallant, Lambert and Vanstone, "Faster point multiplication on elliptic curves with efficient endomorphisms", 2001; the
// basis by the extended Euclidean algorithm on r and lambda, as there).  The rounded quotients come from products with 2^256 b2 / r and
// 2^256 |b1| / r, whose own rounding adds k / 2^257 < 2^-4 to the half.
#pragma once
#include "ff.cuh"

namespace zk {

struct Glv {
  static ZK_HD constexpr uint32_t a1(int i) {  // = b2
    constexpr uint32_t m[2] = {0x94d213e3u, 0x89d32568u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t nb1(int i) {  // -b1
    constexpr uint32_t m[4] = {0x7d4f1128u, 0x8211bbebu, 0xeeb859fcu, 0x6f4d8248u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t a2(int i) {
    constexpr uint32_t m[4] = {0x1221250bu, 0x0be4e154u, 0xeeb859fdu, 0x6f4d8248u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t g1(int i) {  // round(2^256 b2 / r)
    constexpr uint32_t m[3] = {0xc7e0b3d7u, 0xd91d232eu, 0x00000002u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t g2(int i) {  // round(-2^256 b1 / r)
    constexpr uint32_t m[5] = {0x391eb18eu, 0x7a7bd9d4u, 0xa773d2cfu, 0x4ccef014u, 0x00000002u};
    return m[i];
  }
  static ZK_HD constexpr uint32_t beta(int i) {  // in Montgomery form
    constexpr uint32_t m[8] = {0xd782e155u, 0x71930c11u, 0xffbe3323u, 0xa6bb947cu, 0xd4741444u, 0xaa303344u, 0x26594943u, 0x2c3b3f0du};
    return m[i];
  }
};

// out = the NO low words of a b
template <int NA, int NB, int NO>
ZK_HD void mul_words(uint32_t* out, const uint32_t* a, const uint32_t* b) {
#pragma unroll
  for (int i = 0; i < NO; i++) out[i] = 0;
#pragma unroll
  for (int i = 0; i < NA; i++) {
    uint64_t c = 0;
#pragma unroll
    for (int j = 0; j < NB; j++) {
      if (i + j < NO) {
        c += (uint64_t)a[i] * b[j] + out[i + j];
        out[i + j] = (uint32_t)c;
        c >>= 32;
      }
    }
    if (i + NB < NO) out[i + NB] = (uint32_t)c;
  }
}

// r -= a over N words; returns nothing: the caller works modulo 2^(32 N)
template <int N>
ZK_HD void sub_words(uint32_t* r, const uint32_t* a) {
  uint64_t borrow = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const uint64_t d = (uint64_t)r[i] - a[i] - borrow;
    r[i] = (uint32_t)d;
    borrow = (d >> 32) & 1u;
  }
}

// |v| of a two's complement number of five words below 2^128 in absolute value; returns the sign.
ZK_HD bool magnitude(const uint32_t (&v)[5], uint32_t (&m)[4]) {
  const bool negative = (v[4] >> 31) != 0;
  const uint32_t flip = negative ? 0xffffffffu : 0u;
  uint64_t c = negative ? 1 : 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    c += (uint64_t)(v[i] ^ flip);
    m[i] = (uint32_t)c;
    c >>= 32;
  }
  return negative;
}

// k (below r / 2) = +-m1 +- m2 lambda
ZK_HD void glv_split(const uint32_t (&k)[8], uint32_t (&m1)[4], bool* n1, uint32_t (&m2)[4], bool* n2) {
  uint32_t g1[3], g2[5], a1[2], nb1[4], a2[4], t1[11], t2[13];
#pragma unroll
  for (int i = 0; i < 3; i++) g1[i] = Glv::g1(i);
#pragma unroll
  for (int i = 0; i < 5; i++) g2[i] = Glv::g2(i);
#pragma unroll
  for (int i = 0; i < 2; i++) a1[i] = Glv::a1(i);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    nb1[i] = Glv::nb1(i);
    a2[i] = Glv::a2(i);
  }
  mul_words<8, 3, 11>(t1, k, g1);
  mul_words<8, 5, 13>(t2, k, g2);
  // c1 (below 2^64) and c2 (below 2^127): the words from 2^256 on, rounded
  uint32_t c1[2], c2[4];
  uint64_t c = t1[7] >> 31;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    c += t1[8 + i];
    c1[i] = (uint32_t)c;
    c >>= 32;
  }
  c = t2[7] >> 31;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    c += t2[8 + i];
    c2[i] = (uint32_t)c;
    c >>= 32;
  }
  uint32_t k1[5], k2[5], p[5];
#pragma unroll
  for (int i = 0; i < 5; i++) k1[i] = k[i];
  mul_words<2, 2, 4>(p, c1, a1);
  p[4] = 0;
  sub_words<5>(k1, p);
  mul_words<4, 4, 5>(p, c2, a2);
  sub_words<5>(k1, p);
  mul_words<2, 4, 5>(k2, c1, nb1);
  mul_words<4, 2, 5>(p, c2, a1);
  sub_words<5>(k2, p);
  *n1 = magnitude(k1, m1);
  *n2 = magnitude(k2, m2);
}

}  // namespace zk
