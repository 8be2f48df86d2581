// Range-proof preprocessing of Dag::prove_range (src/dag/mod.rs:1314-1337), per auxiliary
// selection polynomial:
//   part[t]  = sum over the selection pairs (input_idx, table_idx = t) of eq(point)[input_idx]
//   middle   = sum_t part[t] * t
//   acc[t]  += beta_gamma * part[t]          (the running sum of the aux polynomials, :1339)
// and the table polynomial range_dense(n).add_by_scalar(alpha) (util/poly.rs:1359-1366, 915-927).
//
// The scatter-add has many pairs per table index and no order among them.  A field element has no
// atomic add, but a sum of Montgomery representations is linear: every 32-bit limb is added into
// its own 64-bit counter with one native atomic (2^32 addends cannot overflow it), and one pass
// afterwards carries the eight counters of an index into a 288-bit integer and reduces it.
#include "../../include/zkb200.h"
#include "ctx.hpp"
#include "reduce.cuh"

using namespace zk;

namespace zk {
int eq_table_device(zk_ctx* ctx, const uint64_t* point_host, uint32_t k, Fr* table, cudaStream_t on = nullptr);
}

namespace {

__global__ void __launch_bounds__(256) k_range_scatter(const uint64_t* __restrict__ input_idx,
                                                       const uint64_t* __restrict__ table_idx, uint64_t n_sel,
                                                       const Fr* __restrict__ eq, uint64_t n_inputs, uint64_t n_table,
                                                       unsigned long long* limbs, unsigned int* bad) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n_sel; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = input_idx[e], t = table_idx[e];
    if (i >= n_inputs || t >= n_table) {
      atomicExch(bad, 1u);
      continue;
    }
    const uint4 lo = __ldg(reinterpret_cast<const uint4*>(eq + i));
    const uint4 hi = __ldg(reinterpret_cast<const uint4*>(eq + i) + 1);
    unsigned long long* L = limbs + t * 8;
    atomicAdd(L + 0, (unsigned long long)lo.x);
    atomicAdd(L + 1, (unsigned long long)lo.y);
    atomicAdd(L + 2, (unsigned long long)lo.z);
    atomicAdd(L + 3, (unsigned long long)lo.w);
    atomicAdd(L + 4, (unsigned long long)hi.x);
    atomicAdd(L + 5, (unsigned long long)hi.y);
    atomicAdd(L + 6, (unsigned long long)hi.z);
    atomicAdd(L + 7, (unsigned long long)hi.w);
  }
}

// The same for a small table (at most kSmallTable entries: lookup blocks of a few bits): with so few counters
// every global atomic would meet thousands of others on its address, so a block first adds into its own copy
// of the counters in shared memory and then flushes each non-zero counter with one global atomic.
constexpr uint32_t kSmallTable = 512;
__global__ void __launch_bounds__(256) k_range_scatter_small(const uint64_t* __restrict__ input_idx,
                                                             const uint64_t* __restrict__ table_idx, uint64_t n_sel,
                                                             const Fr* __restrict__ eq, uint64_t n_inputs, uint32_t n_table,
                                                             unsigned long long* limbs, unsigned int* bad) {
  extern __shared__ unsigned long long sh_limbs[];
  for (uint32_t k = threadIdx.x; k < n_table * 8; k += blockDim.x) sh_limbs[k] = 0;
  __syncthreads();
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n_sel; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = input_idx[e], t = table_idx[e];
    if (i >= n_inputs || t >= n_table) {
      atomicExch(bad, 1u);
      continue;
    }
    const uint4 lo = __ldg(reinterpret_cast<const uint4*>(eq + i));
    const uint4 hi = __ldg(reinterpret_cast<const uint4*>(eq + i) + 1);
    unsigned long long* L = sh_limbs + t * 8;
    atomicAdd(L + 0, (unsigned long long)lo.x);
    atomicAdd(L + 1, (unsigned long long)lo.y);
    atomicAdd(L + 2, (unsigned long long)lo.z);
    atomicAdd(L + 3, (unsigned long long)lo.w);
    atomicAdd(L + 4, (unsigned long long)hi.x);
    atomicAdd(L + 5, (unsigned long long)hi.y);
    atomicAdd(L + 6, (unsigned long long)hi.z);
    atomicAdd(L + 7, (unsigned long long)hi.w);
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < n_table * 8; k += blockDim.x) {
    const unsigned long long v = sh_limbs[k];
    if (v) atomicAdd(limbs + k, v);
  }
}

// And for a table of at most kCopiesTable entries, where 32 lanes would meet on 16 counters: eight lanes take a pair, a limb each,
// and add it into counters of their own, so that no addition is atomic before the block's copies are added up.  2^17 pairs on 16
// entries take 6.9 us, by atomics on a block's one copy 21.6.  The line is where a block of 256 threads fills 32 KB of shared memory with
// its copies.  Above it the lanes of a warp meet half as often with every doubling, and a block that keeps the 32 KB has half as many threads:
// whole calls by copies in such blocks and by atomics take 40 and 50 us for 2^17 pairs on 32 entries, 46 and 50 on 64 (40 and 55 on 16),
// 67 and 100, 70 and 93 (71 and 109) for 2^19, 36 and 40, 37 and 40 (36 and 42) for 2^12.  Blocks of other sizes are not built.
constexpr uint32_t kCopiesTable = 16;
constexpr int kCopiesThreads = 256, kCopies = kCopiesThreads / 8;
__global__ void __launch_bounds__(kCopiesThreads) k_range_scatter_copies(const uint64_t* __restrict__ input_idx,
                                                                         const uint64_t* __restrict__ table_idx, uint64_t n_sel,
                                                                         const Fr* __restrict__ eq, uint64_t n_inputs, uint32_t n_table,
                                                                         unsigned long long* limbs, unsigned int* bad) {
  __shared__ unsigned long long copies[kCopies][kCopiesTable * 8];
  const uint32_t lane = threadIdx.x & 31, limb = threadIdx.x & 7;
  unsigned long long* mine = copies[threadIdx.x >> 3] + limb;
#pragma unroll
  for (uint32_t t = 0; t < kCopiesTable; t++) mine[t * 8] = 0;
  const uint64_t warps = (uint64_t)gridDim.x * (kCopiesThreads / 32), warp = (uint64_t)blockIdx.x * (kCopiesThreads / 32) + (threadIdx.x >> 5);
  for (uint64_t first = warp * 32; first < n_sel; first += warps * 32) {
    uint32_t i = 0, t = kCopiesTable;  // kCopiesTable: no pair
    if (first + lane < n_sel) {
      const uint64_t in = input_idx[first + lane], to = table_idx[first + lane];
      if (in < n_inputs && to < n_table) {
        i = (uint32_t)in;
        t = (uint32_t)to;
      } else {
        atomicExch(bad, 1u);
      }
    }
    uint32_t word[8], at[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {  // the eight lanes of a copy take their eight pairs one after the other
      const int from = (int)(lane & 24u) + k;
      at[k] = __shfl_sync(0xffffffffu, t, from);
      const uint32_t src = __shfl_sync(0xffffffffu, i, from);
      word[k] = at[k] < kCopiesTable ? __ldg(reinterpret_cast<const uint32_t*>(eq + src) + limb) : 0u;
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (at[k] < kCopiesTable) mine[at[k] * 8] += word[k];
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < n_table * 8; k += kCopiesThreads) {
    unsigned long long v = 0;
#pragma unroll 8
    for (int c = 0; c < kCopies; c++) v += copies[c][k];
    if (v) atomicAdd(limbs + k, v);
  }
}

// part[t] from its limb counters; acc[t] += beta_gamma * part[t]; sink.msg[0] = sum_t part[t] * t, sink.msg[1] zero unless *bad is not.
__global__ void __launch_bounds__(256) k_range_finish(const unsigned long long* __restrict__ limbs, uint64_t n_table,
                                                      const unsigned int* __restrict__ bad, const FixedMul<FrParams> bg, Fr* acc,
                                                      const MsgSink sink) {
  Fr mid = Fr::zero();
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_table; t += (uint64_t)gridDim.x * blockDim.x) {
    // X = sum_j limbs[j] * 2^(32 j) < 2^288, as sixteen 32-bit limbs
    Wide x;
#pragma unroll
    for (int k = 0; k < 16; k++) x.v[k] = 0;
    unsigned long long carry = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const unsigned long long v = limbs[t * 8 + j];
      const unsigned long long s = (v & 0xffffffffull) + (carry & 0xffffffffull);
      x.v[j] = (uint32_t)s;
      carry = (v >> 32) + (carry >> 32) + (s >> 32);
    }
    x.v[8] = (uint32_t)carry;
    x.v[9] = (uint32_t)(carry >> 32);
    // X mod r in Montgomery form: redc gives X / R, one more Montgomery product by R^2 restores the factor
    const Fr part = to_mont(redc<FrParams>(x));
    Fr tt = Fr::zero();
    tt.v[0] = (uint32_t)t;
    tt.v[1] = (uint32_t)(t >> 32);
    mid = add(mid, mul(part, to_mont(tt)));
    acc[t] = add(acc[t], mul_fixed(bg, part));
  }
  Fr s[2] = {mid, Fr::zero()};
  if (blockIdx.x == 0 && threadIdx.x == 0) s[1].v[0] = *bad != 0;
  grid_sum<2, 8>(s, sink);
}

// out[i] = i + alpha
__global__ void k_range_table(uint64_t n, const Fr alpha, Fr* out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    Fr v = Fr::zero();
    v.v[0] = (uint32_t)i;
    v.v[1] = (uint32_t)(i >> 32);
    out[i] = add(to_mont(v), alpha);
  }
}

inline size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

extern "C" {

int zk_range_aux_accumulate(zk_ctx* ctx, uint32_t k, const uint64_t* point, uint64_t n_sel, const uint64_t* input_idx,
                            const uint64_t* table_idx, zk_mem idx_mem, const uint64_t* beta_gamma, uint32_t table_log,
                            uint64_t* acc, zk_mem acc_mem, uint64_t* middle_claim_out) {
  if (!ctx || !beta_gamma || !acc || !middle_claim_out || (k && !point) || (n_sel && (!input_idx || !table_idx)))
    return fail(ZK_ERR_ARG, "range_aux_accumulate: NULL argument");
  if (k > 30 || table_log > 30) return fail(ZK_ERR_ARG, "range_aux_accumulate: k %u or table_log %u too large", k, table_log);
  if (n_sel >= (1ull << 32)) return fail(ZK_ERR_ARG, "range_aux_accumulate: at most 2^32 - 1 selection pairs");
  CtxLock lk(ctx);
  ctx = lk.lane;
  cudaStream_t s = ctx->stream;
  const uint64_t n_inputs = 1ull << k, n_table = 1ull << table_log;
  const bool host_idx = idx_mem == ZK_MEM_HOST, host_acc = acc_mem == ZK_MEM_HOST;
  char* base = nullptr;
  size_t need = al(n_inputs * sizeof(Fr)) + al(n_table * 64 + 8) + 1024;
  if (host_idx) need += 2 * al(n_sel * 8 + 8);
  if (host_acc) need += al(n_table * sizeof(Fr));
  int rc = ctx->reserve_work(need, (void**)&base);
  if (rc) return rc;
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += al(bytes); return p; };
  Fr* eq = reinterpret_cast<Fr*>(take(n_inputs * sizeof(Fr)));
  unsigned long long* limbs = reinterpret_cast<unsigned long long*>(take(n_table * 64 + 8));
  unsigned int* bad = reinterpret_cast<unsigned int*>(limbs + n_table * 8);  // cleared together with the counters
  const uint64_t *d_in = input_idx, *d_tab = table_idx;
  if (host_idx && n_sel) {
    uint64_t* a = reinterpret_cast<uint64_t*>(take(n_sel * 8 + 8));
    uint64_t* b = reinterpret_cast<uint64_t*>(take(n_sel * 8 + 8));
    ZK_CUDA(cudaMemcpyAsync(a, input_idx, n_sel * 8, cudaMemcpyHostToDevice, s));
    ZK_CUDA(cudaMemcpyAsync(b, table_idx, n_sel * 8, cudaMemcpyHostToDevice, s));
    d_in = a;
    d_tab = b;
  }
  Fr* d_acc = reinterpret_cast<Fr*>(acc);
  if (host_acc) {
    d_acc = reinterpret_cast<Fr*>(take(n_table * sizeof(Fr)));
    ZK_CUDA(cudaMemcpyAsync(d_acc, acc, n_table * sizeof(Fr), cudaMemcpyHostToDevice, s));
  }
  rc = eq_table_device(ctx, point, k, eq);
  if (rc) return rc;
  ZK_CUDA(cudaMemsetAsync(limbs, 0, n_table * 64 + 8, s));
  if (n_sel) {
    uint64_t blocks = (n_sel + 255) / 256;
    if (blocks > (uint64_t)ctx->sm_count * 8) blocks = ctx->sm_count * 8;
    if (n_table <= kCopiesTable) {
      if (blocks > (uint64_t)ctx->sm_count) blocks = ctx->sm_count;
      k_range_scatter_copies<<<(unsigned)blocks, kCopiesThreads, 0, s>>>(d_in, d_tab, n_sel, eq, n_inputs, (uint32_t)n_table, limbs, bad);
    } else if (n_table <= kSmallTable) {
      if (blocks > (uint64_t)ctx->sm_count * 4) blocks = ctx->sm_count * 4;
      k_range_scatter_small<<<(unsigned)blocks, 256, n_table * 64, s>>>(d_in, d_tab, n_sel, eq, n_inputs, (uint32_t)n_table, limbs, bad);
    } else {
      k_range_scatter<<<(unsigned)blocks, 256, 0, s>>>(d_in, d_tab, n_sel, eq, n_inputs, n_table, limbs, bad);
    }
    ctx->launches++;
  }
  const RoundScratch sc = ctx->next_msg_scratch(false);  // published to the polling host: no copy, no synchronisation
  uint64_t blocks = (n_table + 255) / 256;
  const uint64_t cap = (uint64_t)ctx->sm_count * 4 < (uint64_t)sc.max_blocks ? ctx->sm_count * 4 : sc.max_blocks;
  if (blocks > cap) blocks = cap;
  k_range_finish<<<(unsigned)blocks, 256, 0, s>>>(limbs, n_table, bad, make_fixed_mul(fr_load(beta_gamma)), d_acc, sc.sink);
  ctx->launches++;
  ZK_CUDA(cudaGetLastError());
  if (host_acc) {
    ZK_CUDA(cudaMemcpyAsync(acc, d_acc, n_table * sizeof(Fr), cudaMemcpyDeviceToHost, s));
    ZK_CUDA(cudaStreamSynchronize(s));
  }
  rc = wait_result(ctx);  // every block's sums are in memory before the last one publishes
  if (rc) return rc;
  const Fr* found = reinterpret_cast<const Fr*>(ctx->mailbox);
  if (!found[1].is_zero()) return fail(ZK_ERR_ARG, "range_aux_accumulate: a selection index is out of range");
  memcpy(middle_claim_out, found, sizeof(Fr));
  return ZK_OK;
}

int zk_range_table(zk_ctx* ctx, uint32_t n, const uint64_t* alpha, uint64_t* out, zk_mem out_mem) {
  if (!ctx || !alpha || !out) return fail(ZK_ERR_ARG, "range_table: NULL argument");
  if (n > 32) return fail(ZK_ERR_ARG, "range_table: n %u too large (the reference's entries are u32)", n);
  CtxLock lk(ctx);
  ctx = lk.lane;
  cudaStream_t s = ctx->stream;
  const uint64_t size = 1ull << n;
  Fr* d_out = reinterpret_cast<Fr*>(out);
  if (out_mem == ZK_MEM_HOST) {
    int rc = ctx->reserve_work(size * sizeof(Fr) + 256, (void**)&d_out);
    if (rc) return rc;
  }
  uint64_t blocks = (size + 255) / 256;
  if (blocks > (uint64_t)ctx->sm_count * 8) blocks = ctx->sm_count * 8;
  k_range_table<<<(unsigned)blocks, 256, 0, s>>>(size, fr_load(alpha), d_out);
  ctx->launches++;
  ZK_CUDA(cudaGetLastError());
  if (out_mem == ZK_MEM_HOST) ZK_CUDA(cudaMemcpyAsync(out, d_out, size * sizeof(Fr), cudaMemcpyDeviceToHost, s));
  ZK_CUDA(cudaStreamSynchronize(s));
  return ZK_OK;
}

}  // extern "C"
