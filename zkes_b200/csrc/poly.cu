// Multilinear helpers of src/util/poly.rs on the device:
//   eq table   evaluate_lagrange_basis / precompute_eq (poly.rs:573-618, 657-699)
//   fix from right   out[lo] = sum_hi eq[hi] * f[hi * 2^rem + lo]   (poly.rs:705-758)
#include "internal.hpp"
#include "reduce.cuh"
#include "byte_mma.cuh"
#include "from_right_plan.hpp"

namespace zk {
namespace {

__device__ __forceinline__ Fr ldg_fr(const Fr* p) {
  const uint4 lo = __ldg(reinterpret_cast<const uint4*>(p));
  const uint4 hi = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  return fr_from_chunks(lo, hi);
}
__device__ __forceinline__ Fr ld_fr_plain(const Fr* p) {
  const uint4 lo = reinterpret_cast<const uint4*>(p)[0];
  const uint4 hi = reinterpret_cast<const uint4*>(p)[1];
  return fr_from_chunks(lo, hi);
}
__device__ __forceinline__ void st_fr_plain(Fr* p, const Fr& x) {
  uint4 lo, hi;
  fr_to_chunks(x, lo, hi);
  reinterpret_cast<uint4*>(p)[0] = lo;
  reinterpret_cast<uint4*>(p)[1] = hi;
}

// The eq table in one launch, in stretches of 2^kEqBits consecutive entries that share their high bits.  A stretch is the outer
// product of two half tables over its low variables, the upper half times the factor of the high bits (a product over the variables
// above kEqBits), so that an entry is some six dependent products deep, where doubling the table variable by variable is thirteen:
// the products are few, and below 2^18 entries their latency is the whole time.
//   One stretch a block (up to kEqWave blocks per SM): the seeded halves are multiplied out straight into global memory.
//   More: the halves make the low table in shared memory, and a block multiplies it by the factors of its stretches, one product
//   an entry instead of halves for every stretch (2^21 entries: 54 us against 79 us with a doubling for every stretch).
// 2^12 entries take 6.8 us of kernel time, with a doubling 10.3; 2^17 7.3 and 12.4.
// The point travels as a kernel argument: as a copy it was a call of its own before every table.
constexpr int kEqBits = 10, kEqThreads = 512, kEqWave = 2;

__device__ __forceinline__ Fr eq_factor(const EqPoint& point, uint64_t x, int j) {  // x: the entry's bits from variable 0 on
  const Fr r = point.r[j];
  return ((x >> j) & 1u) ? r : sub(Fr::one(), r);
}
// The factor of `bits` variables from `from` on for an entry with those bits `x`: two interleaved chains of products.
__device__ __forceinline__ Fr eq_product(const EqPoint& point, int from, int bits, uint64_t x) {
  Fr f = Fr::one(), g = Fr::one();
  if (bits > 0) f = eq_factor(point, x << from, from);
  if (bits > 1) g = eq_factor(point, x << from, from + 1);
#pragma unroll 1
  for (int j = 2; j < bits; j += 2) {
    f = mul(f, eq_factor(point, x << from, from + j));
    if (j + 1 < bits) g = mul(g, eq_factor(point, x << from, from + j + 1));
  }
  return bits > 1 ? mul(f, g) : f;
}

__global__ void __launch_bounds__(kEqThreads) k_eq_table(Fr* out, const EqPoint point, int k) {
  __shared__ Fr sh[1 << kEqBits];
  __shared__ Fr seeds[kEqThreads];  // the half tables, later the factors of the stretches
  const int low = k < kEqBits ? k : kEqBits, high = k - low, low_a = low >> 1, low_b = low - low_a;
  const uint64_t n_hi = 1ull << high;
  const bool seeded = n_hi <= gridDim.x;  // one stretch per block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Fr* half_a = seeds;
  Fr* half_b = seeds + 32;
  if (warp == 0 && lane < (1 << low_a)) half_a[lane] = eq_product(point, 0, low_a, lane);
  if (warp == 1 && lane < (1 << low_b)) half_b[lane] = eq_product(point, low_a, low_b, lane);
  if (warp == 2 && seeded) {
    Fr f = Fr::one();
    if (lane < high) f = eq_factor(point, (uint64_t)blockIdx.x << low, low + lane);
    int width = 1;
    while (width < high) width <<= 1;
#pragma unroll 1
    for (int off = width >> 1; off > 0; off >>= 1) {
      Fr o;
#pragma unroll
      for (int i = 0; i < 8; i++) o.v[i] = __shfl_down_sync(0xffffffffu, f.v[i], off);
      f = mul(f, o);
    }
    if (lane == 0) seeds[64] = f;
  }
  __syncthreads();
  if (seeded) {
    if (threadIdx.x < (1u << low_b)) half_b[threadIdx.x] = mul(half_b[threadIdx.x], seeds[64]);
    __syncthreads();
  }
  Fr* dst = seeded ? out + ((uint64_t)blockIdx.x << low) : sh;
#pragma unroll 1
  for (uint32_t x = threadIdx.x; x < (1u << low); x += kEqThreads) st_fr_plain(dst + x, mul(half_a[x & ((1u << low_a) - 1u)], half_b[x >> low_a]));
  if (seeded) return;
  __syncthreads();
  // this block's stretches are blockIdx.x, blockIdx.x + gridDim.x, ...: their factors kEqThreads at a time, then the products
  for (uint64_t first = blockIdx.x; first < n_hi; first += (uint64_t)kEqThreads * gridDim.x) {
    const uint64_t mine = first + (uint64_t)threadIdx.x * gridDim.x;
    if (mine < n_hi) seeds[threadIdx.x] = eq_product(point, low, high, mine);
    __syncthreads();
    for (uint32_t t = 0; t < kEqThreads; t++) {
      const uint64_t hi = first + (uint64_t)t * gridDim.x;
      if (hi >= n_hi) break;
      const Fr f = seeds[t];
#pragma unroll 1
      for (uint32_t x = threadIdx.x; x < (1u << kEqBits); x += kEqThreads) st_fr_plain(out + (hi << kEqBits) + x, mul(f, sh[x]));
    }
    __syncthreads();
  }
}

// Partial column sums: block (bx, by) covers 256 columns and the hi range of split by.
__global__ void __launch_bounds__(256) k_from_right(const Fr* __restrict__ f, const Fr* __restrict__ eq, uint64_t lo_n,
                                                    uint64_t hi_n, uint64_t hi_per_split, Fr* partial) {
  const uint64_t lo = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (lo >= lo_n) return;
  const uint64_t h0 = (uint64_t)blockIdx.y * hi_per_split;
  const uint64_t h1 = (h0 + hi_per_split < hi_n) ? h0 + hi_per_split : hi_n;
  Wide acc;
#pragma unroll
  for (int k = 0; k < 16; k++) acc.v[k] = 0;
  int pending = 0;
  for (uint64_t h = h0; h < h1; h++) {
    const Fr e = ldg_fr(eq + h);
    const Fr v = ldg_fr(f + h * lo_n + lo);
    Wide w;
    mul_wide(w, v.v, e.v);
    wide_add(acc, w);
    if (++pending == kLazyProducts) {
      wide_trim<FrParams>(acc);
      pending = 0;
    }
  }
  wide_trim<FrParams>(acc);
  st_fr_plain(partial + (uint64_t)blockIdx.y * lo_n + lo, redc<FrParams>(acc));
}

// The same sums on the tensor cores (byte_mma.cuh): for a column, D[j][i] = sum_hi (byte j of eq[hi]) (byte i of f[hi][lo]) is a
// product of matrices of bytes, 32 x hi_n by hi_n x 32, and the column's sum is sum_ij 2^(8 (i + j)) D[i][j].
// A warp takes two columns and 32 rows a step: 2 KiB of f, streamed through kCtStages slots of its own in shared memory, which the
// lanes read back as eight bytes of eight rows each and transpose to four rows of a byte in a word, as the instruction wants its
// second operand.  The 2 x 32 x 32 sums stay in registers from step to step.  eq is brought into the order of the first operand once
// per kCtChunk rows for the block's eight warps.
// The steps of all columns form one line that is cut into equal pieces, one for each block that fits the GPU, so that no place idles
// whatever the shape; where a piece ends inside a column, or a column inside a piece, the block puts its sums together (some ten
// steps' worth) and leaves them in a slot of the column's own, and k_sum_splits adds the slots.
// 2^12 rows of 2^12 columns take 102 us (5.3 TB/s of the table's bytes), where the integer pipe took 171 with 64 multiply-adds an
// element; cut by columns alone, 256 blocks for 296 places, it was 112 us.  What bounds it now is issue: some 100 instructions a warp
// and step beside 16 of the tensor cores.
constexpr int kCtThreads = 32 * kCtWarps, kCtStages = 4, kCtChunk = 256;
constexpr size_t kCtShared = (size_t)kCtWarps * kCtStages * 2048 + (size_t)kCtChunk * 32;

// out[b] = bytes b of a0, a1, a2, a3
__device__ __forceinline__ void transpose_bytes(uint32_t (&out)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
  const uint32_t l0 = __byte_perm(a0, a1, 0x5140), h0 = __byte_perm(a0, a1, 0x7362);
  const uint32_t l1 = __byte_perm(a2, a3, 0x5140), h1 = __byte_perm(a2, a3, 0x7362);
  out[0] = __byte_perm(l0, l1, 0x5410);
  out[1] = __byte_perm(l0, l1, 0x7632);
  out[2] = __byte_perm(h0, h1, 0x5410);
  out[3] = __byte_perm(h0, h1, 0x7632);
}

// v / 2^256 mod p for a number of 17 words
__device__ __forceinline__ Fr reduce_words(const uint32_t (&v)[17]) {
  Wide low;
  Fr mid, top = Fr::zero();
#pragma unroll
  for (int k = 0; k < 8; k++) {
    low.v[k] = v[k];
    low.v[k + 8] = 0;
    mid.v[k] = v[k + 8];
  }
  top.v[0] = v[16];
  return add(redc<FrParams>(low), add(mul(Fr::one(), mid), mul(Fr::r2(), top)));
}

// per: steps of a block; col_steps: steps of a column group, ceil(hi_n / 32); slots: as many as a column can have.
__global__ void __launch_bounds__(kCtThreads, 2) k_from_right_bytes(const Fr* __restrict__ f, const Fr* __restrict__ eq, uint64_t lo_n,
                                                                    uint64_t hi_n, uint32_t col_groups, uint32_t col_steps, uint64_t per,
                                                                    uint32_t slots, Fr* partial) {
  extern __shared__ uint4 ct_shared[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  uint4* stage = ct_shared + warp * kCtStages * 128;                                      // [slot][row][4 chunks], swizzled
  uint32_t* frag = reinterpret_cast<uint32_t*>(ct_shared + kCtWarps * kCtStages * 128);   // [step of the chunk][lane][8]
  const uint64_t all = (uint64_t)col_groups * col_steps, line0 = blockIdx.x * per, line1 = line0 + per < all ? line0 + per : all;
  // this lane's part of a copy: chunk lane & 3 of rows lane / 4 + 8 i; a row's chunks sit permuted by its bit 1, so that the lanes'
  // reads below meet no bank twice
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(stage + (lane >> 2) * 4 + ((lane & 3) ^ ((lane >> 2) & 2)));
  const uint64_t row8 = lo_n * 8 * sizeof(Fr);
  const int last_rows = (int)(hi_n - (uint64_t)(col_steps - 1) * kCtStep);
  for (uint64_t line = line0; line < line1;) {
    const uint32_t group = (uint32_t)(line / col_steps), step0 = (uint32_t)(line - (uint64_t)group * col_steps);
    const uint32_t steps = (uint32_t)(line1 - line < col_steps - step0 ? line1 - line : col_steps - step0);
    const uint64_t lo0 = ((uint64_t)group * kCtWarps + warp) * 2;
    const bool in_columns = lo0 + ((lane & 3) >> 1) < lo_n;
    const char* src = reinterpret_cast<const char*>(f + ((uint64_t)step0 * kCtStep + (lane >> 2)) * lo_n + lo0) + 16 * (lane & 3);
    auto issue = [&](uint32_t step) {  // called for step 0, 1, ... in turn
      if (step < steps) {
        const uint32_t dst = to + (step % kCtStages) * 2048;
        const int rows = step0 + step + 1 < col_steps ? kCtStep : last_rows;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const bool live = in_columns && (lane >> 2) + 8 * i < rows;
          const uint32_t bytes = live ? 16u : 0u;  // 0: nothing is read, zeros are written
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 512 * i), "l"(live ? src : (const char*)f), "r"(bytes) : "memory");
          src += row8;
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // d[4 w + b][M]: byte b of word w of the lane columns' eight bytes against bytes 16 M .. 16 M + 15 of eq
    uint32_t d[8][2][4];
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int m = 0; m < 2; m++)
#pragma unroll
        for (int q = 0; q < 4; q++) d[k][m][q] = 0;
#pragma unroll
    for (int k = 0; k < kCtStages - 1; k++) issue(k);
    for (uint32_t step = 0; step < steps; step++) {
      const uint32_t in_chunk = step % (kCtChunk / kCtStep);
      if (in_chunk == 0) {
        // the order of the rows of a step is free as long as both operands have the same: row 16 h + 4 q + t is byte q of word h of
        // the lanes with that t
        __syncthreads();
        for (int k = threadIdx.x; k < kCtChunk * 2; k += kCtThreads) {
          const int word = k & 7, ft = (k >> 3) & 3, fh = (k >> 5) & 1, fs = k >> 6;
          uint32_t a[4], o[4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const uint64_t h = (uint64_t)(step0 + step + fs) * kCtStep + 16 * fh + 4 * q + ft;
            a[q] = h < hi_n ? __ldg(reinterpret_cast<const uint32_t*>(eq + h) + word) : 0u;
          }
          transpose_bytes(o, a[0], a[1], a[2], a[3]);
#pragma unroll
          for (int b = 0; b < 4; b++) {
            const int j = 4 * word + b;
            frag[(fs * 32 + 4 * (j & 7) + ft) * 8 + (j >> 3) * 2 + fh] = o[b];
          }
        }
        __syncthreads();
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(kCtStages - 2) : "memory");
      __syncwarp();
      issue(step + kCtStages - 1);  // into the slot that the warp read a step ago
      const uint4* slot = stage + (step % kCtStages) * 128;
      uint2 x[8];
#pragma unroll
      for (int r = 0; r < 8; r++) x[r] = reinterpret_cast<const uint2*>(slot + (4 * r + t) * 4 + ((g >> 1) ^ (t & 2)))[g & 1];
      const uint4* fr = reinterpret_cast<const uint4*>(frag + (in_chunk * 32 + lane) * 8);
      const uint4 e0 = fr[0], e1 = fr[1];  // bytes of eq: rows g and g + 8 of the first tile, then of the second
#pragma unroll
      for (int w = 0; w < 2; w++) {
        uint32_t b0[4], b1[4];
        if (w == 0) {
          transpose_bytes(b0, x[0].x, x[1].x, x[2].x, x[3].x);
          transpose_bytes(b1, x[4].x, x[5].x, x[6].x, x[7].x);
        } else {
          transpose_bytes(b0, x[0].y, x[1].y, x[2].y, x[3].y);
          transpose_bytes(b1, x[4].y, x[5].y, x[6].y, x[7].y);
        }
#pragma unroll
        for (int b = 0; b < 4; b++) {
          mma_bytes(d[4 * w + b][0], e0.x, e0.z, e0.y, e0.w, b0[b], b1[b]);
          mma_bytes(d[4 * w + b][1], e1.x, e1.z, e1.y, e1.w, b0[b], b1[b]);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // The lane's sums: eight bytes each of columns n = 2 t and 2 t + 1 (n counts eight bytes along the two columns of f), against
    // bytes g + 8 m of eq: u = sum over the column bytes, n - 2 t and m; it belongs at bytes g + 16 (t & 1) of column lo0 + (t >> 1).
    unsigned long long u[11];
#pragma unroll
    for (int k = 0; k < 11; k++) u[k] = 0;
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
      for (int c = 0; c < 2; c++)
#pragma unroll
        for (int w = 0; w < 2; w++) {
          unsigned long long s = 0;
#pragma unroll
          for (int b = 3; b >= 0; b--) s = (s << 8) + d[4 * w + b][m >> 1][2 * (m & 1) + c];
          u[2 * (c + m) + w] += (uint32_t)s;
          u[2 * (c + m) + w + 1] += s >> 32;
        }
    uint32_t v[12], z[17];
    unsigned long long carry = 0;
#pragma unroll
    for (int k = 0; k < 11; k++) {
      carry += u[k];
      v[k] = (uint32_t)carry;
      carry >>= 32;
    }
    v[11] = 0;  // below 2^(256 + 90)
#pragma unroll
    for (int k = 11; k > 0; k--) v[k] = __funnelshift_l(v[k - 1], v[k], 8 * (g & 3));
    v[0] <<= 8 * (g & 3);
#pragma unroll
    for (int k = 0; k < 17; k++) z[k] = (k < 12) ? ((g & 4) ? (k > 0 ? v[k - 1] : 0u) : v[k]) : (k == 12 && (g & 4)) ? v[11] : 0u;
    if (t & 1) {
#pragma unroll
      for (int k = 16; k >= 0; k--) z[k] = k >= 4 ? z[k - 4] : 0u;
    }
#pragma unroll
    for (int off = 16; off > 0; off = off == 4 ? 1 : off >> 1) {  // the eight g, and the two t of a column
      carry = 0;
#pragma unroll
      for (int k = 0; k < 17; k++) {
        carry += (unsigned long long)z[k] + __shfl_xor_sync(0xffffffffu, z[k], off);
        z[k] = (uint32_t)carry;
        carry >>= 32;
      }
    }
    const Fr r = reduce_words(z);
    const uint64_t lo = lo0 + (t >> 1);
    if (g == 0 && (t & 1) == 0 && lo < lo_n) {
      uint32_t at = bytes_slot(blockIdx.x, group, col_steps, per);
      st_fr_plain(partial + (uint64_t)at * lo_n + lo, r);
      if (step0 + steps == col_steps)  // the column's last piece clears the slots that are left over
        for (at++; at < slots; at++) st_fr_plain(partial + (uint64_t)at * lo_n + lo, Fr::zero());
    }
    line += steps;
  }
}

// out[lo] = sum_k partial[k * lo_n + lo].  A block takes 32 columns; its eight warps share the splits (warp g
// sums splits g, g + 8, ...: a warp reads 1 KiB of one split at a time, and the loads of a thread do not wait
// for one another), then the eight partial sums of a column are added through shared memory.
__global__ void __launch_bounds__(256) k_sum_splits(const Fr* __restrict__ partial, uint64_t lo_n, uint32_t splits, Fr* out) {
  __shared__ Fr sh[8][32];
  const int col = threadIdx.x & 31, g = threadIdx.x >> 5;
  const uint64_t lo = (uint64_t)blockIdx.x * 32 + col;
  Fr s = Fr::zero();
  if (lo < lo_n) {
    uint32_t k = g;
    for (; k + 24 < splits; k += 32) {  // four loads in flight
      const Fr a = ld_fr_plain(partial + (uint64_t)k * lo_n + lo), b = ld_fr_plain(partial + (uint64_t)(k + 8) * lo_n + lo);
      const Fr c = ld_fr_plain(partial + (uint64_t)(k + 16) * lo_n + lo), d = ld_fr_plain(partial + (uint64_t)(k + 24) * lo_n + lo);
      s = add(add(s, add(a, b)), add(c, d));
    }
    for (; k < splits; k += 8) s = add(s, ld_fr_plain(partial + (uint64_t)k * lo_n + lo));
  }
  sh[g][col] = s;
  __syncthreads();
  if (g == 0 && lo < lo_n) {
#pragma unroll
    for (int w = 1; w < 8; w++) s = add(s, sh[w][col]);
    st_fr_plain(out + lo, s);
  }
}

// sum_i a[i] * b[i] with lazily reduced products (evaluate_multilinear_extension's final sum, poly.rs:635-647).
__global__ void __launch_bounds__(256) k_dot(const Fr* __restrict__ a, const Fr* __restrict__ b, uint64_t n, const MsgSink sink) {
  Wide acc;
#pragma unroll
  for (int k = 0; k < 16; k++) acc.v[k] = 0;
  int pending = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const Fr x = ldg_fr(a + i), y = ldg_fr(b + i);
    Wide w;
    mul_wide(w, x.v, y.v);
    wide_add(acc, w);
    if (++pending == kLazyProducts) {
      wide_trim<FrParams>(acc);
      pending = 0;
    }
  }
  wide_trim<FrParams>(acc);
  Fr s[1] = {redc<FrParams>(acc)};
  grid_sum<1, 8>(s, sink);
}

}  // namespace

// sink.msg[0] = sum_i a[i] b[i]
void launch_dot(const Fr* a, const Fr* b, uint64_t n, const RoundScratch& sc, cudaStream_t s) {
  uint64_t blocks = (n + 255) / 256;
  const uint64_t cap = (uint64_t)sc.sm_count * 4 < (uint64_t)sc.max_blocks ? sc.sm_count * 4 : sc.max_blocks;
  if (blocks < 1) blocks = 1;
  if (blocks > cap) blocks = cap;
  k_dot<<<(unsigned)blocks, 256, 0, s>>>(a, b, n, sc.sink);
}

// out[0 .. 2^k) = eq(., point), k at most kEqMax.  Returns launches.
int launch_eq_table(const EqPoint& point, uint32_t k, Fr* out, int sm_count, cudaStream_t s) {
  const uint64_t stretches = k > (uint32_t)kEqBits ? 1ull << (k - kEqBits) : 1, wave = (uint64_t)sm_count * kEqWave;
  k_eq_table<<<(unsigned)(stretches < wave ? stretches : wave), kEqThreads, 0, s>>>(out, point, (int)k);
  return 1;
}

uint32_t from_right_splits(uint64_t lo_n, uint64_t hi_n, int sm_count) {
  if (hi_n >= kCtRows) return bytes_plan(lo_n, hi_n, sm_count).slots;
  const uint64_t col_blocks = (lo_n + 255) / 256;
  uint64_t want = ((uint64_t)sm_count * 8 + col_blocks - 1) / col_blocks;  // about 8 blocks per SM
  if (want > hi_n) want = hi_n;
  if (want < 1) want = 1;
  if (want > 65535) want = 65535;
  return (uint32_t)want;
}

// out[lo] = sum_hi eq[hi] * f[hi * lo_n + lo]; partial needs from_right_splits() * lo_n elements.
int launch_from_right(const Fr* f, const Fr* eq, uint64_t lo_n, uint64_t hi_n, Fr* partial, Fr* out, int sm_count,
                      cudaStream_t s) {
  const uint32_t splits = from_right_splits(lo_n, hi_n, sm_count);
  Fr* dst = splits == 1 ? out : partial;
  if (hi_n >= kCtRows) {
    const BytesPlan p = bytes_plan(lo_n, hi_n, sm_count);
    (void)resident_blocks((const void*)k_from_right_bytes, kCtThreads, kCtShared);
    k_from_right_bytes<<<(unsigned)p.blocks, kCtThreads, kCtShared, s>>>(f, eq, lo_n, hi_n, (uint32_t)p.groups, (uint32_t)p.steps, p.per, p.slots, dst);
  } else {
    const uint64_t per = (hi_n + splits - 1) / splits;
    k_from_right<<<dim3((unsigned)((lo_n + 255) / 256), splits), 256, 0, s>>>(f, eq, lo_n, hi_n, per, dst);
  }
  if (splits == 1) return 1;
  k_sum_splits<<<(unsigned)((lo_n + 31) / 32), 256, 0, s>>>(partial, lo_n, splits, out);
  return 2;
}

}  // namespace zk
