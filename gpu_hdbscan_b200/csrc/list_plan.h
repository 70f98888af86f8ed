// How large the joins' candidate list is, from the number of rows and of warps that
// append to it: what is allocated (knn.cu) and what a batch is budgeted for
// (capi.cu).  Host code without CUDA.
#pragma once
#include <algorithm>
#include <cstdint>

namespace hdb {
namespace knn {

// Slots that a warp takes from the list at a time.  The tail that it leaves unused in
// its last chunk is sorted along as sentinels, so the chunk follows the work: about
// a quarter of what a warp will append, between kListChunkMin (one append's most) and
// 768 slots.  (With 1,024 always, the list of 1,500 rows held 1.5 M slots for some
// 50 k candidates.)
constexpr uint32_t kListChunkMin = 96, kListChunkMax = 768;
inline uint32_t list_chunk(int64_t n, int64_t warps) {
  const int64_t candidates_per_warp = 40 * n / warps;
  uint32_t c = kListChunkMin;
  while (c < kListChunkMax && 8 * (int64_t)c <= candidates_per_warp) c *= 2;
  return c;
}

// Room for an iteration's candidates (about 42 per row where it was counted; a row's
// join offers at most 96, so a small list cannot fill up) and for the tails of the
// warps' last chunks.  Positions are 32-bit, and k_group_rows steps up to a block's
// 512 threads past a bucket's end: the list stays 4,096 short of 2^32.
inline int64_t list_slots(int64_t n, int64_t warps) {
  return std::min<int64_t>(std::max<int64_t>(64 * n, std::min<int64_t>(96 * n, int64_t(64) << 20)) +
                               warps * list_chunk(n, warps),
                           (int64_t(1) << 32) - 4096);
}

// Bytes of a list: target and candidate, with the second buffer of the grouping, and the
// grouping's digit counts and offsets (512 of each per 4,096 slots).
inline int64_t list_bytes(int64_t slots) { return slots * (2 * 12 + 1); }

constexpr int kBucketRows = 256;  // most rows of a bucket
// Rows per bucket of the candidate list's grouping, 2^shift: the fewest (from
// 8) whose buckets, and the one of the unused slots behind them, fit one digit
// of the radix passes (9 bits), so that one pass and k_group_rows group the list,
// as long as that is at most kBucketRows; beyond, 128 rows and two passes as long as
// these hold the buckets (2^25 - 128 rows), and past that 256 rows, which two passes
// hold up to 2^26 - 256 rows.  (NN-Descent of 2^25 x 4, k = 16: 624 ms with 128 rows
// and a third pass of one bit, 594 with 256; of 200 rows fewer 578.  Sorting the
// list by row took two and three passes.)
inline int bucket_shift(int64_t n) {
  int shift = 3;
  while ((n - 1) >> shift >= 511) shift++;
  if ((1 << shift) <= kBucketRows) return shift;
  return (n - 1) >> 7 >= (1 << 18) - 1 ? 8 : 7;
}

}  // namespace knn
}  // namespace hdb
