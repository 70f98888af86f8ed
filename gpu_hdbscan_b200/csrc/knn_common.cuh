// Shared pieces of the NN-Descent kernels (knn.cu, join_tc.cu): packed
// (distance, id) keys and the candidate list that the joins append to.
#pragma once
#include "hdb_internal.cuh"
#include "list_plan.h"

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
// the warps of a join do not all queue on that one counter.
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

// Appends this lane's candidates (up to kMax: target row, packed key; the
// caller has checked each against its target's worst[]) to the list that is
// grouped by target before the next merge.  The warp writes them at its
// cursor; when they do not fit in the cursor's chunk, the rest of that chunk
// becomes sentinel entries and one lane takes a new chunk.  Past the list's
// capacity only the best dropped candidate of each target is kept.  Returns
// the lane's count.  Called by all 32 lanes of a warp.
template <int kMax>
__device__ __forceinline__ int append_candidates(const CandList &cl, ListCursor &cur,
                                                 const bool (&v)[kMax], const int32_t (&t)[kMax],
                                                 const uint64_t (&k)[kMax]) {
  static_assert(32 * kMax <= (int)kListChunkMin, "a chunk holds one append");
  const int lane = threadIdx.x & 31;
  uint32_t lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  uint32_t b[kMax], at[kMax], tot = 0;
#pragma unroll
  for (int q = 0; q < kMax; q++) {
    b[q] = __ballot_sync(0xffffffffu, v[q]);
    at[q] = tot + __popc(b[q] & lt);
    tot += __popc(b[q]);
  }
  if (tot == 0) return 0;
  if (cur.pos + tot > cur.end) {
    list_fill(cl, cur.pos, cur.end);
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&cl.counters[3], (unsigned long long)cl.chunk);
    base = __shfl_sync(0xffffffffu, base, 0);
    cur.pos = base;
    cur.end = base + cl.chunk;
  }
  const unsigned long long first = cur.pos;
  cur.pos += tot;
  int mine = 0;
#pragma unroll
  for (int q = 0; q < kMax; q++) {
    if (!v[q]) continue;
    mine++;
    const unsigned long long p = first + at[q];
    if ((int64_t)p < cl.cap) {
      cl.tgt[p] = (uint32_t)t[q];
      cl.key[p] = k[q];
    } else {
      atomicMin(&cl.best[t[q]], (unsigned long long)k[q]);
      atomicAdd(&cl.counters[0], 1ull);
    }
  }
  return mine;
}

// A row's counts and both sample lists in one memory round trip.  Lanes 0..15 hold
// the forward samples, lanes 16..31 the reverse ones.
struct SampleLists {
  int32_t nraw = 0, oraw = 0;
  int cnf = 0, cof = 0, cnr = 0, cor = 0;
  __device__ __forceinline__ void load(int64_t r, int64_t n, int S, const int32_t *__restrict__ newS,
                                       const int32_t *__restrict__ oldS, const int8_t *__restrict__ nf,
                                       const int8_t *__restrict__ of, const int32_t *nrev,
                                       const int32_t *orev) {
    if (r >= n) return;
    const int t = threadIdx.x & 15, half = (threadIdx.x >> 4) & 1;
    const int64_t at = r * (2 * S) + half * S + t;
    nraw = t < S ? newS[at] : 0;
    oraw = t < S ? oldS[at] : 0;
    cnf = nf[r];
    cof = of[r];
    cnr = nrev[r];
    cor = orev[r];
  }
  // The samples in use: new ones into ids[0..nn), old ones into ids[32..32+no),
  // forward before reverse, every id once (ShrinkGraph RemoveDuplicates,
  // nndescent.cu:285-291) and new \ old (:468-486).  The forward samples of a row
  // are distinct, as its list is, and so are the reverse ones, as a row samples an
  // id once: only a reverse sample can repeat a forward one.
  // So 16 comparisons find the repeats of both lists and 32 the new ids among the old,
  // against words that all lanes read together; two match_any take a turn per
  // distinct value (the lists of 1M rows: 485 us with them, 298 without).  The FP32
  // joins, bound by instructions and not by those turns, keep them (SlotLists: 2.03
  // ms at 1M x 12, 2.10 this way).  ids: 64 words, on 16 bytes.  Called by all 32
  // lanes of a warp.
  __device__ __forceinline__ void compact(int S, int32_t *ids, int &nn, int &no) const {
    const int lane = threadIdx.x & 31, t = lane & 15;
    const bool fwd = lane < 16;
    bool vn = t < (fwd ? min(cnf, S) : min(cnr, S));
    bool vo = t < (fwd ? min(cof, S) : min(cor, S));
    const int32_t nid = vn ? nraw : -1 - lane;  // no id, and no two the same
    const int32_t oid = vo ? oraw : -100 - lane;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    ids[lane] = nid;
    ids[32 + lane] = oid;
    const int32_t rnew = __shfl_xor_sync(0xffffffffu, nid, 16);
    __syncwarp();
    const int4 *words = reinterpret_cast<const int4 *>(ids);
    // lane l < 16: is reverse new sample l a forward one; lane 16 + l: old sample l
    const int32_t x = fwd ? rnew : oid;
    bool dup = false, in_old = false;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int4 v = words[(fwd ? 0 : 8) + q];
      dup = dup | (v.x == x) | (v.y == x) | (v.z == x) | (v.w == x);
    }
    if (cof | cor) {  // the same for the whole warp
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int4 v = words[8 + q];
        in_old = in_old | (v.x == nid) | (v.y == nid) | (v.z == nid) | (v.w == nid);
      }
    }
    const uint32_t rep = __ballot_sync(0xffffffffu, dup);
    if (!fwd) {
      vn = vn && !((rep >> t) & 1u);
      vo = vo && !dup;
    }
    vn = vn && !in_old;
    const uint32_t bn = __ballot_sync(0xffffffffu, vn), bo = __ballot_sync(0xffffffffu, vo);
    nn = __popc(bn);
    no = __popc(bo);
    __syncwarp();  // every lane has read the words
    if (vn) ids[__popc(bn & lt)] = nid;
    if (vo) ids[32 + __popc(bo & lt)] = oid;
    __syncwarp();
  }
};

}  // namespace knn
}  // namespace hdb
