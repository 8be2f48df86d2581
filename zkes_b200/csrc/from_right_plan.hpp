// How a contraction of a table's high variables is cut among the blocks of k_from_right_bytes (poly.cu): plain arithmetic, so that the CPU
// tests can go through every piece.
#pragma once
#include <cstdint>

namespace zk {

// Contractions of at least kCtRows rows go through the tensor cores.  A column's sums cost the same to put together whatever its rows:
// 2^22 values take 212 us in 2^5 rows, 121 in 2^6, 73 in 2^7, 54 in 2^8, 43 in 2^10; on the integer pipe 60, 56, 54, 52 and 54.  Few
// columns leave warps of a block without any, and the integer kernel's threads too: a call over 2^18 values takes 49 us in one column, 34 in
// four, 32 in sixteen and 26 in 256; on the integer pipe 269, 119, 63 and 43.  Over 2^16 values 34, 30, 24 in 1, 4, 16 against 98, 60, 49.
constexpr uint64_t kCtRows = 512;
constexpr int kCtWarps = 8, kCtStep = 32, kCtCols = 2 * kCtWarps;  // a warp takes two columns, kCtStep rows a step

struct BytesPlan {
  uint64_t groups, steps, per, blocks;  // groups of kCtCols columns, steps of a column, steps of a block
  uint32_t slots;                       // partial sums of a column, at most
};
inline BytesPlan bytes_plan(uint64_t lo_n, uint64_t hi_n, int sm_count) {
  BytesPlan p;
  p.groups = (lo_n + kCtCols - 1) / kCtCols;
  p.steps = (hi_n + kCtStep - 1) / kCtStep;
  const uint64_t all = p.groups * p.steps, places = 2 * (uint64_t)sm_count;
  p.per = (all + places - 1) / places;
  // sums of 2^15 products of bytes stay below 2^31
  if (p.per > 1024) p.per = 1024;
  p.blocks = (all + p.per - 1) / p.per;
  // a column that begins where a piece does has ceil(steps / per) of them; where all columns do, that is all
  p.slots = (uint32_t)((p.steps + p.per - 1) / p.per + (p.per % p.steps == 0 || p.steps % p.per == 0 ? 0 : 1));
  return p;
}

// The slot of the piece that block `block` has of a column group: the blocks that share a column are neighbours.
constexpr uint32_t bytes_slot(uint64_t block, uint64_t group, uint64_t col_steps, uint64_t per) {
  return (uint32_t)(block - group * col_steps / per);
}

}  // namespace zk
