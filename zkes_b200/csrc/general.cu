// The two remaining provers of src/crypto/sumcheck/linear_prover.rs:
//   SparseBoolSumcheckProver (:455-656)   sum_x eq(r,x) sum_j w_j s_j(x)(s_j(x) - 1), s_j sparse
//   GeneralLinearSumcheckProver (:193-438) sum_x eq(x) sum_j a_j prod_i p_ji(x)
// Both reuse the plain fold kernel for their dense tables; the sparse one reuses the entry fold
// and compaction of sparse.cu with keys = term * 2^(remaining variables) + index, so entries of
// different terms never pair up.
#include "internal.hpp"
#include "reduce.cuh"

namespace zk {
namespace {

constexpr int kGThreads = 256;

__device__ __forceinline__ Fr g_ld(const Fr* p) {
  const uint4 lo = __ldg(reinterpret_cast<const uint4*>(p));
  const uint4 hi = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  return fr_from_chunks(lo, hi);
}

// The round message (compute_round_message, :529-591) is s(c) = sum_y eq(c, y) sum_j w_j aux(aux - 1), c = 0..3, with aux(c) =
// v0 + c (v1 - v0) for the pair (v0, v1) of an even / odd position.  The variable of the round has the factor K eq(tau, c) in eq to itself,
// K the same factor of the variables bound before, so that s(c) = K eq(tau, c) t(c) with t of degree two in c: the kernel sums
//   t(0) = sum_y E (v0^2 - v0),   t(1) = sum_y E (v1^2 - v1),   and t's leading coefficient   sum_y E (v1 - v0)^2
// (weights and terms understood), E the eq table of the variables still to come, and the host makes the four values of them
// (bool_message).  E needs no folding: it is the sum over the lowest variable of the table before (k_eq_sums), whatever the challenges.
//
// Entry by entry instead of pair by pair: an entry alone (value v) is two products, u = E v and u v; a pair's cross term -2 E v0 v1
// exists only where both sides are present, one entry in sixteen for the selection polynomials of the lookups; those entries are queued
// per warp and worked off thirty-two at a time, so that the rare case does not cost every warp its products.
// (With four values straight from records {eq(c), c = 0..3} of every position it was a square and three products an entry and 96 bytes
// gathered for 32: 20 rounds over 16 x 2^17 entries in 1 242 us, now 789.)
//
// The entries are ordered by (term, position), so a warp that walks a contiguous span of them stays inside one term
// for thousands of entries: the weight is taken out of the inner sum and multiplied in when a lane's term changes.
// The gather of E depends on the position: the entry after the next is looked up, and the next one's value and E are on their way,
// while an entry is computed.
//
// ONES: the first round, where every value is one (the selection polynomials are 0/1): t(0) = t(1) = 0, and an entry alone adds E to the
// leading coefficient, a pair nothing; no value is read and nothing is multiplied but the weights.
constexpr int kPairQueue = 64;  // per warp: a batch of 32 plus what one more sweep can add

template <bool ONES>
__global__ void __launch_bounds__(kGThreads, 2) k_sbool_msg(const uint32_t* __restrict__ keys, const Fr* __restrict__ val,
                                                            const uint32_t* __restrict__ count, const Fr* __restrict__ eq,
                                                            const Fr* __restrict__ weights, uint32_t vars_left,
                                                            const MsgSink sink) {
  __shared__ uint32_t queue[ONES ? 1 : kGThreads / 32][ONES ? 1 : kPairQueue];
  const uint32_t n = *count;
  const uint32_t mask = (vars_left >= 32) ? 0xffffffffu : ((1u << vars_left) - 1u);
  // the weighted sums over all terms are touched once per term: they live in shared memory
  __shared__ Fr s_sm[3][kGThreads];
  auto s_add = [&](int c, const Fr& x, bool negate) {
    const Fr cur = s_sm[c][threadIdx.x];
    s_sm[c][threadIdx.x] = negate ? sub(cur, x) : add(cur, x);
  };
#pragma unroll
  for (int c = 0; c < 3; c++) s_sm[c][threadIdx.x] = Fr::zero();
  // the sums over the term this lane is in, without its weight.  ONES: a field element.  Otherwise, for either parity, an unreduced
  // 512-bit sum of the products u v and the sum of the u; picked by the entry's parity, so they live in shared memory (16-byte words
  // kGThreads apart, conflict free), the products trimmed below p 2^256 one by one.
  Fr inner = Fr::zero();
  extern __shared__ uint4 s_sums[];  // [2][6][kGThreads]
  auto wide_ld = [&](int b, Wide& w) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 x = s_sums[(b * 6 + k) * kGThreads + threadIdx.x];
      w.v[4 * k] = x.x;
      w.v[4 * k + 1] = x.y;
      w.v[4 * k + 2] = x.z;
      w.v[4 * k + 3] = x.w;
    }
  };
  auto wide_st = [&](int b, const Wide& w) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      s_sums[(b * 6 + k) * kGThreads + threadIdx.x] = make_uint4(w.v[4 * k], w.v[4 * k + 1], w.v[4 * k + 2], w.v[4 * k + 3]);
  };
  auto lin_ld = [&](int b) { return fr_from_chunks(s_sums[(b * 6 + 4) * kGThreads + threadIdx.x], s_sums[(b * 6 + 5) * kGThreads + threadIdx.x]); };
  auto lin_st = [&](int b, const Fr& x) {
    uint4 lo, hi;
    fr_to_chunks(x, lo, hi);
    s_sums[(b * 6 + 4) * kGThreads + threadIdx.x] = lo;
    s_sums[(b * 6 + 5) * kGThreads + threadIdx.x] = hi;
  };
  if constexpr (!ONES) {
#pragma unroll
    for (int k = 0; k < 12; k++) s_sums[k * kGThreads + threadIdx.x] = make_uint4(0, 0, 0, 0);
  }
  uint32_t cur_term = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint64_t warp = (uint64_t)blockIdx.x * (kGThreads / 32) + wib;
  const uint64_t warps = (uint64_t)gridDim.x * (kGThreads / 32);
  const uint64_t span = (((uint64_t)n + warps - 1) / warps + 31) & ~31ull;  // entries per warp, a multiple of the warp width
  const uint64_t begin = warp * span, end = begin + span < n ? begin + span : n;
  uint32_t queued = 0;  // the same in every lane of the warp
  auto flush = [&](uint32_t term) {
    const Fr w = g_ld(weights + term);
    if constexpr (ONES) {
      s_add(2, mul(w, inner), false);
      inner = Fr::zero();
    } else {
      Wide zero;
#pragma unroll
      for (int k = 0; k < 16; k++) zero.v[k] = 0;
      Fr all = Fr::zero();
#pragma unroll 1
      for (int b = 0; b < 2; b++) {
        Wide sum;
        wide_ld(b, sum);
        const Fr x = redc<FrParams>(sum);
        s_add(b, mul(w, sub(x, lin_ld(b))), false);
        all = add(all, x);
        wide_st(b, zero);
        lin_st(b, Fr::zero());
      }
      s_add(2, mul(w, all), false);
    }
  };
  // the cross terms of 32 queued pairs (or of what is left, at the end)
  auto work_off = [&](uint32_t cnt) {
    if (lane < cnt) {
      const uint32_t i = queue[ONES ? 0 : wib][ONES ? 0 : lane];
      const uint32_t key = keys[i];
      const Fr w = g_ld(weights + (vars_left >= 32 ? 0 : (key >> vars_left)));
      const Fr wx = mul(w, mul(g_ld(val + i), g_ld(val + i + 1)));
      const Fr a = mul(wx, g_ld(eq + ((key & mask) >> 1)));
      s_add(2, add(a, a), true);
    }
  };
  auto key_at = [&](uint64_t i) { return i < end ? keys[i] : 0u; };
  uint32_t key = key_at(begin + lane), key_n = key_at(begin + lane + 32);
  Fr v = Fr::zero(), ev = Fr::zero();
  if (begin + lane < end) {
    if (!ONES) v = g_ld(val + begin + lane);
    ev = g_ld(eq + ((key & mask) >> 1));
  }
  for (uint64_t base = begin; base < end; base += 32) {
    const uint64_t i = base + lane;
    const bool valid = i < end;
    const uint32_t key_nn = key_at(i + 64);
    Fr v_n = v, e_n = ev;
    if (i + 32 < end) {
      if (!ONES) v_n = g_ld(val + i + 32);
      e_n = g_ld(eq + ((key_n & mask) >> 1));
    }
    const bool odd = key & 1u;
    const uint32_t term = vars_left >= 32 ? 0 : (key >> vars_left);
    if (valid && term != cur_term) {
      if (cur_term != 0xffffffffu) flush(cur_term);
      cur_term = term;
    }
    if constexpr (ONES) {
      // alone unless the neighbour of the same pair is the next (previous) entry
      const bool lone = valid && (odd ? !(i > 0 && keys[i - 1] == key - 1) : !(i + 1 < n && keys[i + 1] == key + 1));
      if (lone) inner = add(inner, ev);
    } else {
      if (valid) {
        const Fr u = mul(ev, v);
        const int b = odd ? 1 : 0;
        Wide x, sum;
        mul_wide(x, u.v, v.v);
        wide_ld(b, sum);
        wide_add(sum, x);
        wide_trim<FrParams>(sum);
        wide_st(b, sum);
        lin_st(b, add(lin_ld(b), u));
      }
      // an even entry whose odd neighbour is present: queue the pair's cross term
      const bool pair = valid && !odd && i + 1 < n && keys[i + 1] == key + 1;
      const uint32_t m = __ballot_sync(0xffffffffu, pair);
      if (pair) queue[wib][queued + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i;
      queued += __popc(m);
      __syncwarp();
      if (queued >= 32) {
        work_off(32);
        __syncwarp();
        if (lane + 32 < queued) queue[wib][lane] = queue[wib][lane + 32];  // at most 16 are left over
        queued -= 32;
        __syncwarp();
      }
    }
    key = key_n;
    key_n = key_nn;
    v = v_n;
    ev = e_n;
  }
  if constexpr (!ONES) {
    if (queued) work_off(queued);
  }
  if (cur_term != 0xffffffffu) flush(cur_term);
  Fr s[3];
#pragma unroll
  for (int c = 0; c < 3; c++) s[c] = s_sm[c][threadIdx.x];
  grid_sum<3, kGThreads / 32>(s, sink);
}

// The eq tables of fewer and fewer variables: level l of a table of n entries (a power of two), at tab + 2 n - (2 n >> l), sums the
// pairs of the level before (eq(tau, 0) + eq(tau, 1) = 1).  A block takes kSumBlock entries and the levels up to one entry of its own.
constexpr uint32_t kSumBlock = 1024;
__global__ void __launch_bounds__(256) k_eq_sums(Fr* tab, uint64_t n) {
  __shared__ Fr sh[kSumBlock / 2];
  uint32_t m = n < kSumBlock ? (uint32_t)n : kSumBlock;
  const Fr* src = tab + (uint64_t)blockIdx.x * m;
  for (int level = 1; m > 1; level++) {
    m >>= 1;
    Fr* out = tab + 2 * n - ((2 * n) >> level) + (uint64_t)blockIdx.x * m;
    Fr r[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t t = threadIdx.x + 256 * k;
      if (t < m) r[k] = add(src[2 * t], src[2 * t + 1]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t t = threadIdx.x + 256 * k;
      if (t < m) {
        sh[t] = r[k];
        out[t] = r[k];
      }
    }
    __syncthreads();
    src = sh;
  }
}

// final_evaluation (:644-655): eq * sum_j w_j v_j (v_j - 1), v_j = the entry with key j, eq at the challenges.
__global__ void k_sbool_final(const uint32_t* keys, const Fr* val, const uint32_t* count, const Fr eq,
                              const Fr* weights, uint32_t n_terms, Fr* out) {
  const uint32_t n = *count;
  const Fr one = Fr::one();
  Fr inner = Fr::zero();
  for (uint32_t i = threadIdx.x; i < n; i += 32) {  // one warp: the terms share the chain of products
    const uint32_t j = keys[i];
    if (j >= n_terms) continue;
    const Fr v = val[i];
    inner = add(inner, mul(weights[j], mul(v, sub(v, one))));
  }
  inner = warp_sum(inner);
  if (threadIdx.x == 0) out[0] = mul(eq, inner);
}

__global__ void k_fill_ones(Fr* out, uint32_t n) {
  const Fr one = Fr::one();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = one;
}

struct GeneralParams {
  const Fr* const* tables;  // device array: n_terms * n_factors pointers
  const Fr* scalars;        // n_terms
  const Fr* eq;
  uint32_t n_terms, n_factors;
  uint64_t pairs;
  MsgSink sink;
};

// s(c) = sum_y eq_c(y) sum_j a_j prod_i p_ji,c(y) for c = 0 .. n_factors + 1 (compute_g_value, :298-357).
__global__ void __launch_bounds__(kGThreads) k_general_msg(const GeneralParams p) {
  constexpr int kMaxEval = kMaxPolys + 2;
  Fr s[kMaxEval];
#pragma unroll
  for (int c = 0; c < kMaxEval; c++) s[c] = Fr::zero();
  const int n_eval = (int)p.n_factors + 2;
  for (uint64_t y = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; y < p.pairs; y += (uint64_t)gridDim.x * blockDim.x) {
    const Fr e0 = g_ld(p.eq + 2 * y), e1 = g_ld(p.eq + 2 * y + 1);
    const Fr de = sub(e1, e0);
    Fr inner[kMaxEval];
#pragma unroll
    for (int c = 0; c < kMaxEval; c++) inner[c] = Fr::zero();
    for (uint32_t j = 0; j < p.n_terms; j++) {
      Fr prod[kMaxEval];
      const Fr a = g_ld(p.scalars + j);
#pragma unroll
      for (int c = 0; c < kMaxEval; c++) prod[c] = a;
      for (uint32_t i = 0; i < p.n_factors; i++) {
        const Fr* t = p.tables[j * p.n_factors + i];
        const Fr v0 = g_ld(t + 2 * y), v1 = g_ld(t + 2 * y + 1);
        const Fr dv = sub(v1, v0);
        Fr v = v0;
#pragma unroll
        for (int c = 0; c < kMaxEval; c++) {
          if (c < n_eval) prod[c] = mul(prod[c], v);
          v = add(v, dv);
        }
      }
#pragma unroll
      for (int c = 0; c < kMaxEval; c++) inner[c] = add(inner[c], prod[c]);
    }
    Fr e = e0;
#pragma unroll
    for (int c = 0; c < kMaxEval; c++) {
      if (c < n_eval) s[c] = add(s[c], mul(inner[c], e));
      e = add(e, de);
    }
  }
  grid_sum<kMaxEval, kGThreads / 32>(s, p.sink);
}

// final_evaluation (:420-437): eq[0] * sum_j a_j prod_i p_ji[0]; also writes every table's value.
__global__ void k_general_final(const Fr* const* tables, const Fr* scalars, const Fr* eq, uint32_t n_terms,
                                uint32_t n_factors, Fr* table_vals, Fr* out) {
  if (threadIdx.x || blockIdx.x) return;
  Fr inner = Fr::zero();
  for (uint32_t j = 0; j < n_terms; j++) {
    Fr prod = scalars[j];
    for (uint32_t i = 0; i < n_factors; i++) {
      const Fr v = tables[j * n_factors + i][0];
      if (table_vals) table_vals[j * n_factors + i] = v;
      prod = mul(prod, v);
    }
    inner = add(inner, prod);
  }
  out[0] = mul(inner, eq[0]);
}

inline int g_blocks(uint64_t n, const RoundScratch& sc) {
  uint64_t b = (n + kGThreads - 1) / kGThreads;
  const uint64_t cap = (uint64_t)sc.sm_count * 2 < (uint64_t)sc.max_blocks ? sc.sm_count * 2 : sc.max_blocks;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (int)b;
}

}  // namespace

// The sums of k_sbool_msg<false>: 48 KB beside its 27 KB of static shared memory, two blocks per SM.
constexpr int kSumBytes = 12 * kGThreads * (int)sizeof(uint4);

void launch_sbool_msg(const uint32_t* keys, const Fr* val, const uint32_t* count, uint32_t upper, const Fr* eq,
                      const Fr* weights, uint32_t vars_left, bool ones, const RoundScratch& sc, cudaStream_t s) {
  if (ones) {
    k_sbool_msg<true><<<g_blocks(upper, sc), kGThreads, 0, s>>>(keys, val, count, eq, weights, vars_left, sc.sink);
  } else {
    (void)resident_blocks((const void*)k_sbool_msg<false>, kGThreads, kSumBytes);
    k_sbool_msg<false><<<g_blocks(upper, sc), kGThreads, kSumBytes, s>>>(keys, val, count, eq, weights, vars_left, sc.sink);
  }
}
int launch_eq_sums(Fr* tab, uint64_t n, cudaStream_t s) {
  int launches = 0;
  while (n > 1) {
    const uint64_t blocks = n > kSumBlock ? n / kSumBlock : 1;
    k_eq_sums<<<(unsigned)blocks, 256, 0, s>>>(tab, n);
    launches++;
    tab += 2 * n - 2 * blocks;  // the level of one entry a block
    n = blocks;
  }
  return launches;
}
void launch_sbool_final(const uint32_t* keys, const Fr* val, const uint32_t* count, const Fr& eq, const Fr* weights,
                        uint32_t n_terms, Fr* out, cudaStream_t s) {
  k_sbool_final<<<1, 32, 0, s>>>(keys, val, count, eq, weights, n_terms, out);
}
void launch_fill_ones(Fr* out, uint32_t n, int sm_count, cudaStream_t s) {
  k_fill_ones<<<sm_count * 2, 256, 0, s>>>(out, n);
}
void launch_general_msg(const Fr* const* tables_dev, const Fr* scalars, const Fr* eq, uint32_t n_terms, uint32_t n_factors,
                        uint64_t pairs, const RoundScratch& sc, cudaStream_t s) {
  GeneralParams p{tables_dev, scalars, eq, n_terms, n_factors, pairs, sc.sink};
  k_general_msg<<<g_blocks(pairs, sc), kGThreads, 0, s>>>(p);
}
void launch_general_final(const Fr* const* tables_dev, const Fr* scalars, const Fr* eq, uint32_t n_terms,
                          uint32_t n_factors, Fr* table_vals, Fr* out, cudaStream_t s) {
  k_general_final<<<1, 32, 0, s>>>(tables_dev, scalars, eq, n_terms, n_factors, table_vals, out);
}

}  // namespace zk
