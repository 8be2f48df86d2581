// Host build of the cut of k_from_right_bytes (csrc/from_right_plan.hpp): every block's walk, as the kernel goes it.
#include "../../zkes_b200/csrc/from_right_plan.hpp"

#include <vector>
using namespace zk;

// 0: every step of every column group is in one piece, every slot of a column is written once and none beyond; otherwise what is not.
extern "C" int zkf_walk(uint64_t lo_n, uint64_t hi_n, int sm, uint64_t* out) {
  const BytesPlan p = bytes_plan(lo_n, hi_n, sm);
  out[0] = p.groups;
  out[1] = p.steps;
  out[2] = p.per;
  out[3] = p.blocks;
  out[4] = p.slots;
  const uint64_t all = p.groups * p.steps;
  if (p.per * 32 * 255 * 255 >= 1ull << 31) return 1;  // the exact sums of a piece
  std::vector<uint8_t> written(p.groups * p.slots, 0);
  uint64_t expect = 0;
  for (uint64_t block = 0; block < p.blocks; block++) {
    const uint64_t line1 = (block + 1) * p.per < all ? (block + 1) * p.per : all;
    if (block * p.per >= line1) return 2;
    for (uint64_t line = block * p.per; line < line1;) {
      const uint64_t group = line / p.steps, step0 = line - group * p.steps;
      const uint64_t steps = line1 - line < p.steps - step0 ? line1 - line : p.steps - step0;
      if (line != expect) return 3;
      uint64_t at = bytes_slot(block, group, p.steps, p.per);
      if (at >= p.slots || written[group * p.slots + at]++) return 4;
      if (step0 + steps == p.steps)
        for (at++; at < p.slots; at++)
          if (written[group * p.slots + at]++) return 5;
      line += steps;
      expect = line;
    }
  }
  if (expect != all) return 6;
  for (uint8_t w : written)
    if (w != 1) return 7;
  return 0;
}
