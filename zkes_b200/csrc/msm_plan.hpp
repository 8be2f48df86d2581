// Shapes of the MSM pipeline (msm.cu): which route a call takes, how its work is cut, and the scratch that this needs.  Host
// arithmetic on sizes alone, without CUDA, so that it can be checked on a machine without a GPU.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>

namespace zk {

constexpr unsigned kEndoBits = 160;  // scalars of more bits are split by the endomorphism (glv.cuh)
// Points a row of a split scalar, at most.  What the split saves is in the buckets, and they are few beside many points: 2^16 points take
// 662 us split and 726 whole, 2^20 3 869 and 4 124, 2^22 13 086 and 13 489, 2^24 49 622 and 50 258, 2^25 99 429 and 99 749.  Above 2^24
// that is less than a two-hundredth of the call for images of the bases of a gigabyte and more.
constexpr uint64_t kEndoMost = 1ull << 24;
constexpr int kEndoMagnitude = 126;  // into magnitudes of as many bits: (1/2 + 2^-4) (a1 + a2) of glv.cuh is below 2^126
constexpr int kCompactBits = 30;  // magnitudes below 2^30 have a compact form (k_msm_bits)
constexpr int kAccBlocks = 4;     // blocks of 128 threads per SM of the kernels that add points in chains (126 and 122 registers)
constexpr uint32_t kReduceThreads = 128;   // threads of a block of the bucket reduction
constexpr int kRowsGroupMax = 12;          // bases a group of the subset-sum tables has at most (k_rows_*)
constexpr size_t kAffineBytes = 64, kXyzzBytes = 128;

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Window width for n points per row whose scalars have at most max_bits magnitude bits.
inline int pick_window(uint64_t n, uint32_t rows, int max_bits) {
  int lg = 0;
  while ((1ull << (lg + 1)) <= n) lg++;
  // a row costs windows * (n + 2 * 2^(w-1)) additions; with many rows the buckets (128 bytes each, per
  // row and window) also have to fit in memory, so rows use a narrower window
  int w = rows > 1 ? lg - 4 : lg - 2;
  if (w > 16) w = 16;
  if (w < 3) w = 3;
  if (w > max_bits + 1) w = max_bits + 1;
  if (w < 2) w = 2;
  // A top window of one to three bits has a handful of buckets that between them take every point, and joining their pieces is
  // a chain of its own; one bit less per window then costs at most one window more.  Of full-width scalars (254 bits with the
  // sign) this is the width 14, 2^16 to 2^17 - 1 points: it leaves two bits for the nineteenth window, 13 leaves seven for the
  // twentieth (100003 points: 1 140 us against 941).  15 and 16 bits leave fourteen (262143 points: 1 623 us with 15, 1 872 us
  // with 14).  Narrower windows stay as they are: 12 bits (2^14 points on) leave two bits, but 11 would leave one; and 11 bits
  // take 12000 points in 548 us where 10, which leave four, take 583.
  if (rows == 1 && w >= 14 && max_bits > kCompactBits && (max_bits + 1) - w * ((max_bits + w) / w - 1) < 4) w--;
  return w;
}

// Rows over the same bases whose windows share their buckets (k_multiples): from kMergedRows rows on.  Window width: a row adds
// 2 n points a window and some three points a bucket.  Below 32 rows the multiples (a chain of 126 doublings, 0.2 to 0.6 ms) cost what
// the shared buckets save.
// The tables of the multiples stay in the lane's scratch, so the route is bounded by their bytes: 2^18 points a row, 470 MB.  It
// gains less with the points, too: 32 rows of 2^14 full-width scalars take 2.76 ms with shared buckets and 3.31 without, of 2^18 32.8 and
// 34.4, of 2^19 63.9 and 59.1 (128 rows of 2^18: 111 and 137).
constexpr uint32_t kMergedRows = 32;
constexpr uint64_t kMergedMost = 1ull << 20;  // points a row whose multiples' indices fit beside an entry's flags whatever the window
constexpr size_t kMergedBytes = 512u << 20;
constexpr size_t kMultipleBytes = 64 + 128 + 32;  // of a multiple: affine, XYZZ while they are made, the x of its image
inline int merged_window(uint64_t n) {
  int best = 4;
  double least = 1e300;
  for (int w = 4; w <= 16; w++) {
    const double cost = 2.0 * (double)n * ((kEndoMagnitude + w) / w) + 3.0 * (double)(1u << (w - 1));
    if (cost < least) {
      least = cost;
      best = w;
    }
  }
  return best;
}
inline bool merged_rows(uint64_t n, uint32_t rows) {
  if (rows < kMergedRows || n > kMergedMost) return false;
  const int w = merged_window(n);
  return n * (uint64_t)((kEndoMagnitude + w) / w) * kMultipleBytes <= kMergedBytes;
}

// Signed-digit windows needed for magnitudes up to max_mag: k digits in (-half, half] reach
// half * (1 + 2^w + ... + 2^(w (k - 1))).
inline int windows_for(uint32_t max_mag, int w) {
  const uint64_t half = 1ull << (w - 1);
  uint64_t reach = 0;
  int k = 0;
  do {
    reach = (reach << w) + half;
    k++;
  } while (reach < max_mag);
  return k;
}

// Entries per chunk of the accumulation (a chunk is a thread's): whole waves of resident threads, of some 64 to 96 entries each
// where there are that many.  Shorter chunks mean more pieces of buckets to join afterwards, a last wave that is nearly
// empty costs as much as a full one: 2^24 entries in chunks of 32 left 2^19 pieces, whose sums took 286 us against 142 us for a
// third of them; 1.9 M entries in one full wave instead of four fifths of one take 345 us against 436 us.
constexpr uint32_t kChunkMin = 16, kChunkWaves = 12;
inline uint32_t chunk_entries(uint32_t n_entries, int sm) {
  const uint64_t resident = (uint64_t)sm * kAccBlocks * 128;
  uint64_t seg = (n_entries + resident - 1) / resident;
  if (seg < kChunkMin) return kChunkMin;
  if (seg > 96) {
    uint64_t waves = seg / 64;
    if (waves > kChunkWaves) waves = kChunkWaves;
    seg = (n_entries + resident * waves - 1) / (resident * waves);
  }
  return (uint32_t)seg;
}

// Up to kFixupBuckets buckets, the pieces of a bucket that was cut by the chunks are added by up to kFixupGroups blocks, one per
// kFixupShare pieces (k_msm_fixup_block).  How many a bucket can keep busy is bounded by the digits that a (row, window) has:
// `longest` of them may all be the same one, and then a single block adds its pieces one after the other.
constexpr uint32_t kFixupBuckets = 8192, kFixupGroups = 128, kFixupShare = 256;
constexpr uint32_t kFixupPartials = 16384;  // partial sums (buckets x blocks)
inline uint32_t fixup_groups(uint32_t n_buckets, uint32_t n_chunks, uint64_t longest, uint32_t seg) {
  const uint64_t pieces = std::min<uint64_t>(n_chunks, longest / seg + 2);
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({(pieces + kFixupShare - 1) / kFixupShare, kFixupGroups, kFixupPartials / n_buckets}));
}

// Lanes per item for k_msm_bucket_reduce_rows, 0 where an item is worth a block or more of its own.  More lanes shorten the
// chain and add work (a scan and a tree over them), so they double only until half of the threads that fit the GPU (three
// blocks of 128 per SM) have work: 4096 items of 128 buckets lost 2 % of their commitment with sixteen lanes instead of eight.
// An item of two or four buckets (rows of fewer than 256 bases, scalars of one bit) is one thread's: a block has nothing to
// share out (2048 rows of 128 full-width scalars, 174080 items: 28.8 ms with a block each, 5.6 with a thread, 5.9 with two and
// 6.4 with four lanes; 16 rows, 1360 items: 1.22 and 1.05 ms; 4 rows, 340 items: 0.87 and 0.85 ms).  With fewer items the blocks
// cost nothing, and most buckets may be empty, which a thread skips, but not a warp that has 32 items (one point, 85 items: 407 us
// with a thread each, 337 with a block).
inline uint32_t reduce_lanes(uint32_t n_items, uint32_t half, int sm) {
  if (half < 8) return n_items < 512 ? 0 : 1;
  if (n_items < 1024) return 0;
  uint32_t lanes = 8;
  while (lanes < 32 && lanes * 2 <= half && (uint64_t)n_items * lanes < (uint64_t)sm * 3 * 64) lanes *= 2;
  return lanes;
}

// Buckets per thread and blocks per item of the bucket reduction.  Longer runs cost fewer additions in all (2 + 4 / per a
// bucket), shorter ones a shorter chain: the runs double while the launch still fills the GPU with threads, and an item has at
// most kReduceThreads blocks (the second launch joins them in one block).
inline void reduce_shape(uint32_t n_items, uint32_t half, uint32_t* per, uint32_t* parts) {
  uint32_t p = 1;
  while (p < half && (p < 32 && (uint64_t)n_items * (half / (2 * p)) >= 40000)) p *= 2;
  if (p < 4) p = half < 4 ? half : 4;
  while (half / p > kReduceThreads * kReduceThreads) p *= 2;
  *per = p;
  const uint32_t n = half / p;
  *parts = n > kReduceThreads ? n / kReduceThreads : 1;
}

// Who combines the windows of a row (sum_k 2^(W k) window k, a chain of W (windows - 1) dependent doublings).
//   the host: up to four rows, from a few dozen doublings on.  A doubling takes a CPU core 0.3 us with 64-bit limbs, a GPU thread
//   4.5 us and a warp 2.2 us, against which the two small copies and the synchronisation (some 20 us) count little.
//   a warp per row: up to a few rows per SM, where the combination is one such chain (40 rows of two windows of three bits: 284 us
//   by threads, 275 by warps; of 16 bits in six windows: 361 and 308).
//   a thread per row: more rows, whose chains overlap while a thread does an eighth of a warp's work; and a single window, where
//   there is no chain and a warp's tree only adds to the time (one row 169 us by a warp, 156 by a thread; 592 rows 268 and 257).
enum class Combine { kHost, kWarps, kThreads };
constexpr uint32_t kHostCombineRows = 4, kHostCombineChain = 24;
inline Combine combine_by(uint32_t rows, int w, int k_windows, int sm) {
  const uint32_t chain = (uint32_t)w * (uint32_t)(k_windows - 1);
  if (chain == 0 || rows > 4u * (uint32_t)sm) return Combine::kThreads;
  return rows <= kHostCombineRows && chain >= kHostCombineChain ? Combine::kHost : Combine::kWarps;
}

// Buckets of a call and the scratch of their route, laid out for the worst case: every scalar has a non-zero digit in every
// window.  Small scalars have fewer, and the real total is checked after the count pass (entry slots are 32-bit).
struct BucketPlan {
  int w = 0, k_windows = 0;
  uint32_t half = 0;            // buckets per (row, window)
  uint64_t n_buckets = 0;       // 2^31 or more: not representable, nothing below is set
  uint64_t max_entries = 0;
  uint64_t chunks = 0;          // of the accumulation, at most
  uint32_t red_per = 0, red_parts = 0;
  uint64_t n_runs = 0;
  size_t scratch = 0;           // bytes, without the scan's own
};

inline BucketPlan bucket_plan(uint64_t total, uint32_t rows, int w, int k_windows, int sm) {
  BucketPlan b;
  b.w = w;
  b.k_windows = k_windows;
  b.half = 1u << (w - 1);
  b.n_buckets = (uint64_t)rows * k_windows * b.half;
  if (b.n_buckets >= (1ull << 31)) return b;
  b.max_entries = std::min<uint64_t>(total * (uint64_t)k_windows, 0xffffffffull);
  b.chunks = std::min<uint64_t>(b.max_entries / kChunkMin + 1, (uint64_t)sm * kAccBlocks * 128 * kChunkWaves);
  reduce_shape(rows * (uint32_t)k_windows, b.half, &b.red_per, &b.red_parts);
  b.n_runs = b.red_parts > 1 ? 2ull * rows * k_windows * b.red_parts : 0;
  b.scratch = align256(b.n_runs * kXyzzBytes) + 2 * align256((b.n_buckets + 2) * 4) + align256(b.n_buckets * kXyzzBytes) +
              align256((size_t)rows * k_windows * kXyzzBytes) + align256(b.max_entries * 4) + 2 * align256((b.chunks + 1) * kXyzzBytes) +
              align256((size_t)kFixupPartials * kXyzzBytes) + 4096;
  return b;
}

// Shape of the subset-sum method for `rows` dense rows of n small scalars, group = 0 when buckets are taken instead.
struct RowsPlan {
  int group = 0;  // bases per group
  int planes = 0;
  uint32_t groups = 0;
  uint32_t seg = 0, parts = 0;  // a unit's groups are cut into `parts` chains of `seg`, a thread each
  uint32_t slab = 0;            // chains whose tables are held at a time
  size_t idx_bytes = 0, halves_bytes = 0, table_bytes = 0, pieces_bytes = 0;
  uint32_t slab_groups() const { return (uint32_t)std::min<uint64_t>(groups, (uint64_t)slab * seg); }
  size_t scratch() const { return align256(idx_bytes) + align256(halves_bytes) + align256(table_bytes) + align256(pieces_bytes) + 1024; }
};

// The time is the waves of threads that the chains take times a chain's length, plus the additions that join the chains
// (14 products to 10, at half the efficiency): 32768 units of 342 groups in three parts are 1.3 waves, which cost two, and took
// 2.17 ms; nine parts are 3.9.
inline void rows_chains(RowsPlan* p, uint32_t rows, int sm) {
  const uint64_t units = (uint64_t)rows * p->planes, resident = (uint64_t)sm * kAccBlocks * 128;
  uint64_t parts = 1;
  double least = 1e300;
  for (uint64_t c = 1; c <= 64 && c <= p->groups; c++) {
    const uint64_t waves = (units * c + resident - 1) / resident;
    const double cost = (double)waves * (double)((p->groups + c - 1) / c) + 2.8 * (double)(units * c) / (double)resident;
    if (cost < least) {
      least = cost;
      parts = c;
    }
  }
  p->seg = (uint32_t)((p->groups + parts - 1) / parts);
  p->parts = (p->groups + p->seg - 1) / p->seg;
}

// Sizes with the tables of `slab` chains held at a time.
inline void rows_sizes(RowsPlan* p, uint32_t rows, uint32_t slab) {
  const uint64_t units = (uint64_t)rows * p->planes;
  const int s = p->group, lo_bits = (s + 1) / 2;
  p->slab = slab;
  const uint64_t held = p->slab_groups();
  p->idx_bytes = units * held * 2;
  p->halves_bytes = held * ((1u << lo_bits) + (1u << (s - lo_bits))) * kAffineBytes;
  p->table_bytes = (held << s) * kAffineBytes;
  p->pieces_bytes = p->parts * units * kXyzzBytes;
}

// max_scratch: what the buckets' route would take.  Above kRowsScratch the tables never take more than that: they are made for
// as many chains at a time as fit (2^20 columns in 1024 rows of int8 values: 9 GB at once, 4.6 GB of buckets).
constexpr size_t kRowsScratch = 256ull << 20;

// Microseconds of the two routes beyond what they share (the pass over the scalars and its read-back), from the times of their
// kernels at 148 SMs.  Both have parts that are rates and parts that are chains of dependent additions, 4.8 us each, which small
// calls and few rows never get below: counting additions alone sent 16 rows of 16384 bits to the sums (613 us, 385 by buckets)
// and took no account of zeros, which have no digits (4096 rows of 4096 int8 values, nine in ten of them zero: 2609 and 1786 us).
// Over 4366 shapes (2 to 16384 rows of 8 to 65536 values of 1 to 24 bits, none to 99.5 % of them zero) the route taken is 0.7 %
// slower than the better one on average (geometric mean), where the count of additions was 12 % slower and up to ten times.
inline double buckets_us(const BucketPlan& b, uint32_t rows, uint64_t nonzero, uint64_t total, int sm) {
  const double resident = (double)sm * kAccBlocks * 128, items = (double)rows * b.k_windows, nb = (double)b.n_buckets;
  const double entries = std::max(1.0, (double)nonzero * b.k_windows), seg = std::max((double)kChunkMin, entries / resident);
  double t = 60 + 24e-6 * (double)total * b.k_windows;  // counting, scan, scatter, a second read-back
  // accumulation: chains of seg entries, on which a thread also passes over the empty buckets between its entries
  const double chunks = std::max(1.0, entries / kChunkMin);
  const double walk = nb > entries ? 0.15 * nb / chunks * (1 + std::log(std::min(32.0, chunks))) : 0;
  t += std::max(4.8 * std::min(seg, entries) + walk, 0.166e-3 * entries);
  t += b.n_buckets <= kFixupBuckets ? 6 + 0.014 * std::min(nb, entries / 8) : 30 + 0.5e-3 * std::min(nb, 8 * entries / seg);
  const uint32_t lanes = reduce_lanes((uint32_t)items, b.half, sm);
  if (lanes) {
    const double per = (double)b.half / lanes, steps = 2 * per + 2 * std::log2(lanes) + (lanes > 1 ? std::log2(per) + 1 : 0);
    t += steps * std::max(lanes > 1 ? 5.0 : 8.0, 0.3e-3 * items * lanes);
  } else {
    t += std::max(60 + 0.1 * items + 4 * std::log2(b.half), 0.75e-3 * nb);
  }
  const double chain = b.w * (b.k_windows - 1);
  if (chain > 0) t += rows <= 4u * (uint32_t)sm ? 20 + 1.6 * chain + 0.03 * rows : 15 + 5 * chain;
  return t;
}

inline double sums_us(const RowsPlan& p, uint32_t rows, uint64_t nonzero, uint64_t total) {
  const int s = p.group;
  const double units = (double)rows * p.planes, groups = p.groups, table = std::ldexp(groups, s);
  const double halves = groups * (std::ldexp(1.0, (s + 1) / 2) + std::ldexp(1.0, s / 2));
  // a warp adds where any of the rows that its 32 units belong to has a scalar that is not zero
  const double busy = 1 - std::pow(1 - (double)nonzero / (double)total, s * std::max(1.0, 32.0 / p.planes));
  double t = 0.004e-3 * (double)total + std::max(21 + 2.2 * s, 1.4e-3 * halves) + std::max(50.0, 0.174e-3 * table);
  t += std::max(4.8 * p.seg * busy, 0.156e-3 * units * groups * busy) + 0.004e-3 * units * groups;
  if (p.parts > 1) t += std::max(8 + 1.85 * p.parts, 0.3e-3 * p.parts * units);
  return t + 11.3 * (p.planes - 1);
}

// The shape with the fewest additions whose scratch fits, if it is faster than the buckets b.
inline RowsPlan rows_plan(uint64_t n, uint32_t rows, uint32_t max_span, uint64_t nonzero, const BucketPlan& b, int sm, size_t max_scratch) {
  RowsPlan best;
  int planes = 1;
  while (planes < 32 && (max_span >> (planes - 1))) planes++;
  double least = 1e300;
  const uint64_t units = (uint64_t)rows * planes;
  if (units >= (1ull << 31)) return best;
  for (int s = 2; s <= kRowsGroupMax; s++) {
    const uint64_t groups = (n + s - 1) / s;
    if ((groups << s) >= (1ull << 31) || units * groups >= (1ull << 40)) continue;
    const double cost = (double)(units * groups) + (double)(groups << s);
    if (cost >= least) continue;
    RowsPlan p;
    p.group = s;
    p.planes = planes;
    p.groups = (uint32_t)groups;
    rows_chains(&p, rows, sm);
    if (p.parts * units >= (1ull << 31)) continue;
    const size_t limit = std::max(max_scratch, kRowsScratch);
    uint32_t slab = p.parts;
    rows_sizes(&p, rows, slab);
    while (p.scratch() > limit && slab > 1) {
      slab = (slab + 1) / 2;
      rows_sizes(&p, rows, slab);
    }
    if (p.scratch() > limit) continue;
    least = cost;
    best = p;
  }
  if (best.group && b.n_buckets < (1ull << 31) && sums_us(best, rows, nonzero, n * rows) >= buckets_us(b, rows, nonzero, n * rows, sm))
    return RowsPlan();
  return best;
}

}  // namespace zk
