// Dense sumcheck round kernels over BN254 Fr.
//
// One launch per round.  k_round<L, FOLD> binds the previous round's challenge (FOLD) and
// computes this round's message in the same pass, so every live table entry is read once
// per round and the folded half is written once:
//   fold     u[j]  = t[2j] + r (t[2j+1] - t[2j])                    linear_prover.rs:151-178
//   message  s(c)  = sum_y prod_i (u_i[2y] + c (u_i[2y+1] - u_i[2y])),  c = 0..L   :82-140
// Sums of products are kept as unreduced 512-bit integers per thread (one Montgomery
// reduction per thread per evaluation point), then reduced over the warp by shuffles, over
// the block through shared memory and over the grid by the last block to finish.
#include "internal.hpp"
#include "reduce.cuh"
#include "round_pass.cuh"
#include "byte_mma.cuh"

namespace zk {

namespace {

constexpr int kThreads = kRoundThreads;
constexpr int kWarps = kRoundWarps;

template <int L>
struct RoundParams {
  const Fr* src[L];
  Fr* dst[L];
  FixedMul<FrParams> r;  // multiplier table of the challenge being bound
  uint64_t pairs;  // (even, odd) pairs of the table the message is computed over
  MsgSink sink;
};

template <int L, bool FOLD>
__global__ void __launch_bounds__(kThreads, (L <= 1 ? 3 : 2)) k_round(const RoundParams<L> p) {
  __shared__ uint4 stage[kWarps][WarpTile<8>::kChunks];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Fr s[L + 1];
  round_pass<L, FOLD>(p.src, p.dst, p.r, p.pairs, (uint64_t)blockIdx.x * kWarps + warp, (uint64_t)gridDim.x * kWarps,
                      stage[warp], lane, s);
  grid_sum<L + 1, kWarps>(s, p.sink);
}

// Last step of the protocol: bind the final challenge on the two remaining entries of each
// table and multiply the results (linear_prover.rs:181-190).  With bind == 0 the tables
// already hold one entry each (num_var == 0).
struct FinalParams {
  const Fr* src[kMaxPolys];
  int num_poly;
  int bind;
  Fr r;
  Fr* out;  // out[0..num_poly) = a_arrays[i][0], out[num_poly] = product
};

__global__ void k_final(const FinalParams p) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Fr prod = Fr::one();
  for (int i = 0; i < p.num_poly; i++) {
    Fr a = p.src[i][0];
    if (p.bind) a = add(a, mul(p.r, sub(p.src[i][1], a)));
    p.out[i] = a;
    prod = mul(prod, a);
  }
  p.out[p.num_poly] = prod;
}

// Plain fold of the lowest variable (no message): util/poly.rs:852-884.
struct FoldParams {
  const Fr* src;
  Fr* dst;
  FixedMul<FrParams> r;
  uint64_t out_len;
};

__global__ void __launch_bounds__(kThreads) k_fold(const FoldParams p) {
  __shared__ uint4 stage[kWarps][WarpTile<4>::kChunks];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* sw = stage[warp];
  const uint64_t tiles = (p.out_len + 31) >> 5;
  for (uint64_t tile = (uint64_t)blockIdx.x * kWarps + warp; tile < tiles; tile += (uint64_t)gridDim.x * kWarps) {
    const uint64_t e0 = tile << 5;
    const uint32_t valid = (uint32_t)((p.out_len - e0) < 32 ? (p.out_len - e0) : 32);
    uint4 raw[4], q[4];
    WarpTile<4>::issue(reinterpret_cast<const uint4*>(p.src) + e0 * 4, valid * 4, lane, raw);
    WarpTile<4>::transpose_in(sw, lane, raw, q);
    const Fr a = fr_from_chunks(q[0], q[1]), b = fr_from_chunks(q[2], q[3]);
    const Fr u = add(a, mul_fixed(p.r, sub(b, a)));
    uint4 o[2];
    fr_to_chunks(u, o[0], o[1]);
    WarpTile<2>::store(reinterpret_cast<uint4*>(p.dst) + e0 * 2, valid * 2, sw, lane, o);
  }
}

// Two folds in one pass (challenges r0 then r1): dst[y] from src[4y .. 4y+3].  Used when the
// first of the two folds could be postponed, so the table is read once for both.
//
// dst[y] = sum_i w_i src[4y + i] with the four weights (1 - r0)(1 - r1), r0 (1 - r1), (1 - r0) r1, r0 r1 fixed for the launch, and
// byte j of src[4y + i] contributes itself times w_i 2^(8j) mod p: the fold is the product of the table, read as rows of 128
// bytes, with a 128 x 32 matrix of bytes, and runs on the tensor cores (byte_mma.cuh).  The matrix carries a factor 2^32, which
// the one Montgomery round over a row's 32 columns takes off again.
// What bounds it is HBM: the two launches of a prove over 2^26 entries move 3.36 GB in 503 us, 6.7 TB/s, as fast as a plain copy;
// with 210 multiply-adds an element on the integer pipe they took 665 us at 77 % of that pipe.  16 instructions of 7.5 cycles per 16
// elements leave the tensor cores a fifth busy.
struct Fold2Params {
  const Fr* src;
  Fr* dst;
  Fr w[4];  // the weights times 2^32, in Montgomery form
  uint64_t out_len;
};

// A warp takes 32 rows, two tiles of 16.  Lane 4 g + t reads 16 bytes each of the two halves of rows 4 g .. 4 g + 3 (a quad reads
// whole lines, nothing goes through shared memory), and the order of a row's bytes in the product is the one in which they sit in
// the lanes.  The columns are dealt so that a lane's eight of a row are neighbours.  The next 32 rows are read ahead.
__global__ void __launch_bounds__(kThreads, 4) k_fold2(const Fold2Params p) {
  __shared__ Fr table[128];  // row i * 32 + j: w_i 2^(32 + 8 j)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  for (int k = threadIdx.x; k < 128; k += kThreads) {
    Fr shift = Fr::zero();
#pragma unroll
    for (int i = 0; i < 8; i++) shift.v[i] = i == ((k & 31) >> 2) ? 1u << (8 * (k & 3)) : 0u;
    table[k] = mul(p.w[k >> 5], shift);
  }
  __syncthreads();
  // step s, tile j of eight columns: words 2 s and 2 s + 1 of the row's eight words of lane t; column g of the tile
  uint32_t c[4][4][2];
  const uint8_t* bytes = reinterpret_cast<const uint8_t*>(table);
#pragma unroll
  for (int s = 0; s < 4; s++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int q = 2 * s + h, at = (q >> 2) * 64 + 16 * t + 4 * (q & 3), col = 8 * (g >> 1) + 2 * j + (g & 1);
        uint32_t v = 0;
#pragma unroll
        for (int b = 0; b < 4; b++) v |= (uint32_t)bytes[(at + b) * 32 + col] << (8 * b);
        c[s][j][h] = v;
      }
  const uint64_t tiles = (p.out_len + 31) >> 5, stride = (uint64_t)gridDim.x * kWarps;
  const uint4* src = reinterpret_cast<const uint4*>(p.src);
  uint64_t tile = (uint64_t)blockIdx.x * kWarps + warp;
  uint4 x[4][2];
  auto fetch = [&](uint64_t at) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const uint64_t row = (at << 5) + 4 * g + r;
#pragma unroll
      for (int h = 0; h < 2; h++) x[r][h] = row < p.out_len ? __ldg(src + row * 8 + 4 * h + t) : make_uint4(0, 0, 0, 0);
    }
  };
  if (tile < tiles) fetch(tile);
  for (; tile < tiles; tile += stride) {
    uint32_t d[2][4][4];
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int k = 0; k < 4; k++) d[u][j][k] = 0;
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint4 a = x[2 * u][h], b = x[2 * u + 1][h];
#pragma unroll
        for (int j = 0; j < 4; j++) mma_bytes(d[u][j], a.x, b.x, a.y, b.y, c[2 * h][j][0], c[2 * h][j][1]);
#pragma unroll
        for (int j = 0; j < 4; j++) mma_bytes(d[u][j], a.z, b.z, a.w, b.w, c[2 * h + 1][j][0], c[2 * h + 1][j][1]);
      }
    if (tile + stride < tiles) fetch(tile + stride);
    uint32_t share[4][3];  // of rows 4 g .. 4 g + 3
#pragma unroll
    for (int r = 0; r < 4; r++) {
      uint32_t cols[8];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        cols[2 * j] = d[r >> 1][j][2 * (r & 1)];
        cols[2 * j + 1] = d[r >> 1][j][2 * (r & 1) + 1];
      }
      join_columns(share[r], cols);
    }
    quad_transpose(share, t);
    const Fr y = reduce_shares<FrParams>(share);
    const uint64_t out = (tile << 5) + lane;
    if (out < p.out_len) {
      uint4 lo, hi;
      fr_to_chunks(y, lo, hi);
      reinterpret_cast<uint4*>(p.dst + out)[0] = lo;
      reinterpret_cast<uint4*>(p.dst + out)[1] = hi;
    }
  }
}

int grid_for(uint64_t tiles, int max_blocks) {
  uint64_t blocks = (tiles + kWarps - 1) / kWarps;
  if (blocks < 1) blocks = 1;
  if (blocks > (uint64_t)max_blocks) blocks = max_blocks;
  return (int)blocks;
}

template <int L>
void launch_round_t(bool fold, const Fr* const* src, Fr* const* dst, const Fr& r, uint64_t pairs,
                    const RoundScratch& sc, cudaStream_t stream) {
  RoundParams<L> p;
  for (int i = 0; i < L; i++) {
    p.src[i] = src[i];
    p.dst[i] = fold ? dst[i] : nullptr;
  }
  p.r = make_fixed_mul(r);
  p.pairs = pairs;
  p.sink = sc.sink;
  static int occ[2] = {0, 0};  // resident blocks per SM, per variant
  if (!occ[fold]) {
    int o = 0;
    if (fold)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_round<L, true>, kThreads, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_round<L, false>, kThreads, 0);
    occ[fold] = o > 0 ? o : 1;
  }
  int cap = sc.sm_count * occ[fold];
  if (cap > sc.max_blocks) cap = sc.max_blocks;
  const int grid = grid_for((pairs + 31) / 32, cap);
  if (fold)
    k_round<L, true><<<grid, kThreads, 0, stream>>>(p);
  else
    k_round<L, false><<<grid, kThreads, 0, stream>>>(p);
}

}  // namespace

void launch_round(int num_poly, bool fold, const Fr* const* src, Fr* const* dst, const Fr& r, uint64_t pairs,
                  const RoundScratch& sc, cudaStream_t stream) {
  switch (num_poly) {
    case 1: launch_round_t<1>(fold, src, dst, r, pairs, sc, stream); break;
    case 2: launch_round_t<2>(fold, src, dst, r, pairs, sc, stream); break;
    case 3: launch_round_t<3>(fold, src, dst, r, pairs, sc, stream); break;
    case 4: launch_round_t<4>(fold, src, dst, r, pairs, sc, stream); break;
    default: break;  // callers check 1 <= num_poly <= kMaxPolys
  }
}

void launch_final(int num_poly, bool bind, const Fr* const* src, const Fr& r, Fr* out, cudaStream_t stream) {
  FinalParams p;
  for (int i = 0; i < kMaxPolys; i++) p.src[i] = i < num_poly ? src[i] : nullptr;
  p.num_poly = num_poly;
  p.bind = bind ? 1 : 0;
  p.r = r;
  p.out = out;
  k_final<<<1, 32, 0, stream>>>(p);
}

void launch_fold(const Fr* src, Fr* dst, const Fr& r, uint64_t out_len, int max_blocks, cudaStream_t stream) {
  FoldParams p{src, dst, make_fixed_mul(r), out_len};
  k_fold<<<grid_for((out_len + 31) / 32, max_blocks), kThreads, 0, stream>>>(p);
}

void launch_fold2(const Fr* src, Fr* dst, const Fr& r0, const Fr& r1, uint64_t out_len, int max_blocks,
                  cudaStream_t stream) {
  Fold2Params p;
  p.src = src;
  p.dst = dst;
  p.out_len = out_len;
  Fr two32 = Fr::zero();
  two32.v[1] = 1;
  two32 = to_mont(two32);
  const Fr both = mul(r0, r1);
  const Fr w[4] = {add(sub(sub(Fr::one(), r0), r1), both), sub(r0, both), sub(r1, both), both};
  for (int i = 0; i < 4; i++) p.w[i] = mul(w[i], two32);
  k_fold2<<<grid_for((out_len + 31) / 32, max_blocks / 2), kThreads, 0, stream>>>(p);  // four blocks per SM of the eight
}

}  // namespace zk
