// Sums of products of field elements as byte products on the tensor cores: the pieces common to the kernels that contract a
// table with fixed factors (k_fold2, k_from_right).
//
// A 256-bit number is 32 bytes, and mma.sync.m16n8k32 multiplies 16 x 32 by 32 x 8 unsigned bytes into exact 32-bit sums.  The
// multiply-adds of a contraction then cost the integer pipe nothing; what is left for it is to put 32 columns of byte products
// back together, some 60 additions, shifts and shuffles an element where a product takes 64 wide multiply-adds.
#pragma once
#include "ff.cuh"
#include <cuda_runtime.h>

namespace zk {

// d += a b.  Lane 4 g + t: a[0], a[1] are bytes 4t .. 4t + 3 of rows g and g + 8, a[2], a[3] the same rows' bytes 16 + 4t ..;
// b0, b1 are bytes 4t .. and 16 + 4t .. of column g; d[0], d[1] are columns 2t, 2t + 1 of row g, d[2], d[3] of row g + 8.
__device__ __forceinline__ void mma_bytes(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// w = c[0] + 2^8 c[1] + ... + 2^56 c[7] for sums below 2^23 (128 products of bytes): three words, the last below 2^16.
__device__ __forceinline__ void join_columns(uint32_t (&w)[3], const uint32_t (&c)[8]) {
  uint32_t p[4];  // two columns each: below 2^23 + 2^31
#pragma unroll
  for (int j = 0; j < 4; j++) p[j] = c[2 * j] + (c[2 * j + 1] << 8);
  const uint32_t s0 = p[1] << 16, s1 = __funnelshift_l(p[1], p[3], 16), s2 = p[3] >> 16;
  asm("add.cc.u32  %0, %3, %5;\n\t"
      "addc.cc.u32 %1, %4, %6;\n\t"
      "addc.u32    %2, %7, 0;"
      : "=r"(w[0]), "=r"(w[1]), "=r"(w[2])
      : "r"(p[0]), "r"(p[2]), "r"(s0), "r"(s1), "r"(s2));
}

// A quad holds four rows, 64 bits of columns a lane: x[r] is row r's share.  Lane t leaves with the four shares of row t.
__device__ __forceinline__ void quad_transpose(uint32_t (&x)[4][3], int t) {
#pragma unroll
  for (int step = 1; step <= 2; step <<= 1) {
    const bool up = (t & step) != 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      if (r & step) continue;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const uint32_t lo = x[r][k], hi = x[r + step][k];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, step);
        x[r][k] = up ? got : lo;
        x[r + step][k] = up ? hi : got;
      }
    }
  }
}

// (sum_t 2^(64 t) x[t]) / 2^32 mod p, for a sum below 2^269.  One Montgomery round leaves it below 2^237 + p < 2p.
template <class P>
__device__ __forceinline__ Fp<P> reduce_shares(const uint32_t (&x)[4][3]) {
  uint32_t v[9], m;
  v[0] = x[0][0];
  v[1] = x[0][1];
  asm("add.cc.u32  %0, %7,  %14;\n\t"
      "addc.cc.u32 %1, %8,  0;\n\t"
      "addc.cc.u32 %2, %9,  %15;\n\t"
      "addc.cc.u32 %3, %10, 0;\n\t"
      "addc.cc.u32 %4, %11, %16;\n\t"
      "addc.cc.u32 %5, %12, 0;\n\t"
      "addc.u32    %6, %13, 0;"
      : "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8])
      : "r"(x[1][0]), "r"(x[1][1]), "r"(x[2][0]), "r"(x[2][1]), "r"(x[3][0]), "r"(x[3][1]), "r"(x[3][2]), "r"(x[0][2]),
        "r"(x[1][2]), "r"(x[2][2]));
  m = v[0] * P::inv;
  row_even(v, v[8], P::mod(0), P::mod(2), P::mod(4), P::mod(6), m);
  madwide4(v + 1, P::mod(1), P::mod(3), P::mod(5), P::mod(7), m);  // the value stays below 2^269 + 2^32 p < 2^288
  Fp<P> r;
#pragma unroll
  for (int k = 0; k < 8; k++) r.v[k] = v[k + 1];
  final_sub<P>(r.v, 0);
  return r;
}

}  // namespace zk
