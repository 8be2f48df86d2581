// Multilinear helpers of src/util/poly.rs on the device:
//   eq table   evaluate_lagrange_basis / precompute_eq (poly.rs:573-618, 657-699)
//   fix from right   out[lo] = sum_hi eq[hi] * f[hi * 2^rem + lo]   (poly.rs:705-758)
#include "internal.hpp"
#include "reduce.cuh"

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

// The eq table in one launch, in stretches of 2^kEqBits consecutive entries that share their high bits; the factor of the
// high bits is a product over the variables above kEqBits.  Launches and the multiplier tables that the host made for every
// level were most of the time of a doubling level by level (2^17 entries: a head launch of 11 us and seven level launches of
// 2.5 us each, with some 4 us of host work before each).
//   One stretch a block (up to kEqWave blocks per SM): the factor seeds a doubling over the low variables in shared memory,
//   a[x + cur] = r a[x], a[x] -= a[x + cur], whose last level goes to global memory; a chain of some twelve products.
//   More: the doubling starts from one and makes the low table, and a block multiplies it by the factors of its stretches,
//   one product an entry instead of a chain per stretch (2^21 entries: 54 us against 79 us with a chain for every stretch).
constexpr int kEqBits = 10, kEqThreads = 512, kEqWave = 2;

__device__ __forceinline__ Fr eq_factor(const Fr* __restrict__ point, uint64_t hi, int j) {
  const Fr r = ldg_fr(point + j);
  return ((hi >> j) & 1u) ? r : sub(Fr::one(), r);
}

__global__ void __launch_bounds__(kEqThreads) k_eq_table(Fr* out, const Fr* __restrict__ point, int k) {
  __shared__ Fr sh[1 << kEqBits];
  __shared__ Fr seeds[kEqThreads];
  const int low = k < kEqBits ? k : kEqBits, high = k - low;
  const uint64_t n_hi = 1ull << high;
  const bool seeded = n_hi <= gridDim.x;  // one stretch per block
  if (threadIdx.x < 32) {
    Fr f = Fr::one();
    if (seeded) {
      if ((int)threadIdx.x < high) f = eq_factor(point + low, blockIdx.x, threadIdx.x);
      int width = 1;
      while (width < high) width <<= 1;
#pragma unroll 1
      for (int off = width >> 1; off > 0; off >>= 1) {
        Fr o;
#pragma unroll
        for (int i = 0; i < 8; i++) o.v[i] = __shfl_down_sync(0xffffffffu, f.v[i], off);
        f = mul(f, o);
      }
    }
    if (threadIdx.x == 0) {
      if (low == 0) st_fr_plain(out, f); else sh[0] = f;
    }
  }
  __syncthreads();
  Fr* dst = out + ((uint64_t)blockIdx.x << low);
#pragma unroll 1
  for (int i = 0; i < low; i++) {
    const uint32_t cur = 1u << i;
    if (threadIdx.x < cur) {
      const Fr r = ldg_fr(point + i);
      const Fr v = sh[threadIdx.x];
      const Fr hi = mul(r, v), lo = sub(v, hi);
      if (seeded && i == low - 1) {
        st_fr_plain(dst + threadIdx.x + cur, hi);
        st_fr_plain(dst + threadIdx.x, lo);
      } else {
        sh[threadIdx.x + cur] = hi;
        sh[threadIdx.x] = lo;
      }
    }
    __syncthreads();
  }
  if (seeded) return;
  // this block's stretches are blockIdx.x, blockIdx.x + gridDim.x, ...: their factors kEqThreads at a time, then the products
  for (uint64_t first = blockIdx.x; first < n_hi; first += (uint64_t)kEqThreads * gridDim.x) {
    const uint64_t mine = first + (uint64_t)threadIdx.x * gridDim.x;
    if (mine < n_hi) {
      Fr f = eq_factor(point + low, mine, 0);
#pragma unroll 1
      for (int j = 1; j < high; j++) f = mul(f, eq_factor(point + low, mine, j));
      seeds[threadIdx.x] = f;
    }
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

// out[0 .. 2^k) = eq(., point); point_dev holds the k coordinates on the device.  Returns launches.
int launch_eq_table(const Fr* point_dev, uint32_t k, Fr* out, int sm_count, cudaStream_t s) {
  const uint64_t stretches = k > (uint32_t)kEqBits ? 1ull << (k - kEqBits) : 1, wave = (uint64_t)sm_count * kEqWave;
  k_eq_table<<<(unsigned)(stretches < wave ? stretches : wave), kEqThreads, 0, s>>>(out, point_dev, (int)k);
  return 1;
}

uint32_t from_right_splits(uint64_t lo_n, uint64_t hi_n, int sm_count) {
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
  const uint64_t per = (hi_n + splits - 1) / splits;
  dim3 grid((unsigned)((lo_n + 255) / 256), splits);
  if (splits == 1) {
    k_from_right<<<grid, 256, 0, s>>>(f, eq, lo_n, hi_n, per, out);
    return 1;
  }
  k_from_right<<<grid, 256, 0, s>>>(f, eq, lo_n, hi_n, per, partial);
  k_sum_splits<<<(unsigned)((lo_n + 31) / 32), 256, 0, s>>>(partial, lo_n, splits, out);
  return 2;
}

}  // namespace zk
