// Shared pieces of the NN-Descent kernels (knn.cu, join_tc.cu): packed
// (distance, id) keys and the candidate list that the joins append to.
#pragma once
#include "hdb_internal.cuh"

namespace hdb {
namespace knn {

constexpr int kMaxK = 32;

// Key of a candidate: distance bits (non-negative floats order as unsigned)
// above the id, so an unsigned compare orders by (distance, id).
__device__ __forceinline__ uint64_t pack(float d, int32_t id) {
  return ((uint64_t)__float_as_uint(d) << 32) | (uint32_t)id;
}
__device__ __forceinline__ float pk_dist(uint64_t k) { return __uint_as_float((uint32_t)(k >> 32)); }
__device__ __forceinline__ int32_t pk_id(uint64_t k) { return (int32_t)(uint32_t)k; }

// NNDElement::label(): "old" entries are stored as -id-1.
__device__ __forceinline__ int32_t decode(int32_t label) { return label >= 0 ? label : -label - 1; }

// Where the joins leave their candidates: one list of (target row, packed
// candidate), grouped by blocks of target rows between the join and the merge.
// Only when the list is full is a candidate dropped; the best dropped one per
// row is still kept in `best`.
struct CandList {
  unsigned long long *best;      // [n]
  uint32_t *tgt;                 // [cap] target row
  uint64_t *key;                 // [cap] packed candidate
  unsigned long long *counters;  // [0] dropped [1] rows gathered [2] candidates [3] list length
                                 // [4] distance pairs computed (FP32 join)
  int64_t cap;
  uint32_t chunk;                // slots that a warp takes at a time
  uint32_t none;                 // target of an unused slot: past every bucket of rows
};

// Space of the candidate list a warp writes into: [pos, end), taken from the
// list `chunk` slots at a time with one atomic on the list's counter, so that
// the warps of a join do not all queue on that one counter.  The tail that a
// warp leaves unused in its last chunk is sorted along as sentinels, so the
// chunk follows the work: about a quarter of what a warp will append, between
// kListChunkMin (one append's most) and 1,024 slots.  (With 1,024 always, the
// list of 1,500 rows held 1.5 M slots for some 50 k candidates.)
constexpr uint32_t kListChunkMin = 64, kListChunkMax = 1024;
inline uint32_t list_chunk(int64_t candidates_per_warp) {
  uint32_t c = kListChunkMin;
  while (c < kListChunkMax && 8 * (int64_t)c <= candidates_per_warp) c *= 2;
  return c;
}
struct ListCursor {
  unsigned long long pos = 0, end = 0;
};

// Writes the sentinel entry (target `none`, sorted after every row's; key ~0)
// at list positions [from, to).
__device__ __forceinline__ void list_fill(const CandList &cl, unsigned long long from,
                                          unsigned long long to) {
  for (unsigned long long p = from + (threadIdx.x & 31); p < to; p += 32)
    if ((int64_t)p < cl.cap) {
      cl.tgt[p] = cl.none;
      cl.key[p] = ~0ull;
    }
}

// Appends this lane's candidates (up to two: target row, packed key; the
// caller has checked each against its target's worst[]) to the list that is
// sorted by target before the next merge.  The warp writes them at its
// cursor; when they do not fit in the cursor's chunk, the rest of that chunk
// becomes sentinel entries and one lane takes a new chunk.  Past the list's
// capacity only the best dropped candidate of each target is kept.  Returns
// the lane's count.  Called by all 32 lanes of a warp.
__device__ __forceinline__ int append_candidates(const CandList &cl, ListCursor &cur, bool v0,
                                                 int32_t t0, uint64_t k0, bool v1,
                                                 int32_t t1, uint64_t k1) {
  const int lane = threadIdx.x & 31;
  uint32_t lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  const uint32_t b0 = __ballot_sync(0xffffffffu, v0), b1 = __ballot_sync(0xffffffffu, v1);
  const uint32_t tot = __popc(b0) + __popc(b1);
  if (tot == 0) return 0;
  if (cur.pos + tot > cur.end) {
    list_fill(cl, cur.pos, cur.end);
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&cl.counters[3], (unsigned long long)cl.chunk);
    base = __shfl_sync(0xffffffffu, base, 0);
    cur.pos = base;
    cur.end = base + cl.chunk;
  }
  const unsigned long long p0 = cur.pos + __popc(b0 & lt);
  const unsigned long long p1 = cur.pos + __popc(b0) + __popc(b1 & lt);
  cur.pos += tot;
  const int32_t tt[2] = {t0, t1};
  const uint64_t kk[2] = {k0, k1};
  const unsigned long long pp[2] = {p0, p1};
  const bool vv[2] = {v0, v1};
#pragma unroll
  for (int q = 0; q < 2; q++) {
    if (!vv[q]) continue;
    if ((int64_t)pp[q] < cl.cap) {
      cl.tgt[pp[q]] = (uint32_t)tt[q];
      cl.key[pp[q]] = kk[q];
    } else {
      atomicMin(&cl.best[tt[q]], (unsigned long long)kk[q]);
      atomicAdd(&cl.counters[0], 1ull);
    }
  }
  return (v0 ? 1 : 0) + (v1 ? 1 : 0);
}

}  // namespace knn
}  // namespace hdb
