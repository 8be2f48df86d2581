// Host build of the MSM's shape rules (csrc/msm_plan.hpp) for the CPU unit tests.
#include "../../zkes_b200/csrc/msm_plan.hpp"
using namespace zk;

// out: buckets, scratch bytes
extern "C" void zkp_buckets(uint64_t total, uint32_t rows, int w, int k_windows, int sm, uint64_t* out) {
  const BucketPlan b = bucket_plan(total, rows, w, k_windows, sm);
  out[0] = b.n_buckets;
  out[1] = b.scratch;
}
// out: window bits, windows (of scalars below 2^30 with the largest magnitude max_mag)
extern "C" void zkp_windows(uint64_t n, uint32_t rows, uint32_t max_mag, uint64_t* out) {
  int bits = 0;
  while (max_mag >> bits) bits++;
  const int w = pick_window(n, rows, bits);
  out[0] = (uint64_t)w;
  out[1] = (uint64_t)windows_for(max_mag, w);
}
// out: group, planes, groups, seg, parts, scratch bytes, partial sums, chains held at a time
extern "C" void zkp_rows(uint64_t n, uint32_t rows, uint32_t max_span, uint64_t nonzero, int w, int k_windows, int sm, uint64_t max_scratch,
                         uint64_t* out) {
  const RowsPlan p = rows_plan(n, rows, max_span, nonzero, bucket_plan(n * rows, rows, w, k_windows, sm), sm, max_scratch);
  out[0] = (uint64_t)p.group;
  out[1] = (uint64_t)p.planes;
  out[2] = p.groups;
  out[3] = p.seg;
  out[4] = p.parts;
  out[5] = p.scratch();
  out[6] = (uint64_t)p.parts * rows * p.planes;
  out[7] = p.slab;
}
// out: window bits, windows, most points a row, most points a row of a split scalar
extern "C" void zkp_merged(uint64_t n, uint64_t* out) {
  const int w = merged_window(n);
  out[0] = (uint64_t)w;
  out[1] = (uint64_t)((kEndoMagnitude + 1 + w - 1) / w);
  out[2] = kMergedMost;
  out[3] = kEndoMost;
}
extern "C" int zkp_merged_rows(uint64_t n, uint32_t rows) { return merged_rows(n, rows); }
extern "C" uint32_t zkp_reduce_lanes(uint32_t n_items, uint32_t half, int sm) { return reduce_lanes(n_items, half, sm); }
extern "C" int zkp_combine_by(uint32_t rows, int w, int k_windows, int sm) { return (int)combine_by(rows, w, k_windows, sm); }
extern "C" uint32_t zkp_fixup_groups(uint32_t n_buckets, uint32_t n_chunks, uint64_t longest, uint32_t seg) {
  return fixup_groups(n_buckets, n_chunks, longest, seg);
}
extern "C" uint32_t zkp_chunk_entries(uint32_t n_entries, int sm) { return chunk_entries(n_entries, sm); }
