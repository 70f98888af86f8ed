// NN-Descent kNN graph (gpuknn::NNDescent, gpuknn/nndescent.cu:2088-2199).
//
// Same algorithm as the reference -- hash-seeded random init, per iteration a
// sample of S new / S old neighbours plus reverse samples, a local join in
// which every new neighbour is offered its closest other new neighbour and
// its closest old neighbour and every old neighbour its closest new one --
// laid out for one B200:
//  * no per-row spin locks (InsertToGlobalGraph, nndescent.cu:969-1028): the
//    joins append their candidates (pre-filtered against the target row's
//    current k-th distance) to one list, which is grouped by target row, and
//    the next pass merges each row's part, one warp per row;
//  * the three sampling kernels, MarkAllToOld and the merge are one kernel
//    (k_sample);
//  * distances are the reference's sequential FP32 difference sum
//    (nndescent.cu:1086-1093, fmaf per element), so every pair has one exact
//    value wherever it is computed.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "hdb_internal.cuh"
#include "join_tc.cuh"
#include "knn.cuh"
#include "knn_common.cuh"

namespace hdb {

using namespace knn;

namespace {


__host__ __device__ __forceinline__ uint64_t xorshift64star(uint64_t x) {
  // gpuknn/knncuda_tools.cu:126-132
  x += 42;
  x ^= x >> 12;
  x ^= x << 25;
  x ^= x >> 27;
  return x * 0x2545F4914F6CDD1DULL;
}


// Ascending bitonic sort of one u64 per lane across the warp.
__device__ __forceinline__ uint64_t warp_sort32(uint64_t v) {
  const int lane = lane_id();
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      uint64_t o = __shfl_xor_sync(0xffffffffu, v, stride);
      bool up = ((lane & size) == 0);
      bool lower = (lane & stride) == 0;
      uint64_t mn = v < o ? v : o, mx = v < o ? o : v;
      v = (lower == up) ? mn : mx;
    }
  }
  return v;
}

// warp_sort32 with a 32-bit payload that moves with its key (keys distinct
// within the warp, or equal only where the payload does not matter).
__device__ __forceinline__ void warp_sort32_with(uint64_t &v, int32_t &pl) {
  const int lane = lane_id();
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const uint64_t o = __shfl_xor_sync(0xffffffffu, v, stride);
      const int32_t op = __shfl_xor_sync(0xffffffffu, pl, stride);
      const bool up = ((lane & size) == 0);
      const bool lower = (lane & stride) == 0;
      const bool take = (lower == up) ? o < v : v < o;  // the other lane's key is the min / max
      v = take ? o : v;
      pl = take ? op : pl;
    }
  }
}

// ---------------------------------------------------------------------------
// Two FP32 differences b - a with one packed instruction: b + (-a), per
// component the same rounding as __fsub_rn(b, a) = -__fsub_rn(a, b), so its
// square is the square of the reference's a - b, bit for bit.
__device__ __forceinline__ float2 neg_diff2(float2 b, float2 a) {
  return __fadd2_rn(b, make_float2(-a.x, -a.y));
}

// Exact sequential difference sums of one row against m <= 32 other rows, one per
// lane (its id): sum = fmaf(a_j - b_j, a_j - b_j, sum) for j = 0..d-1, the reference's
// FP32 difference sum (nndescent.cu:1086-1093).  The 33 rows are copied to shared
// memory whole (up to kStageCols dimensions at a time), all copies of a chunk in
// flight together, and each lane then walks its own row.  kV floats a copy: 4
// where every row is 16-byte aligned (d % 4 == 0), 2 where it is 8-byte aligned,
// else 1.  Rows take an odd number
// of copies, so the lanes' walks read distinct bank groups.
//
// Bound by the gather: at 20M x 128, k = 32, k_init takes 66 ms and k_rerank 47 (99
// and 74 with chunks of 32 dimensions in a ring of two), of 50 ms for 328 GB at the
// measured copy rate; at 10M x 12 k_init takes 10.4 ms (21), as the shared memory
// for a short row lets 32 warps run on an SM instead of 24.  64 dimensions, k_init
// and k_rerank at 20M x 128 and at 200k x 128 in L2: 65.5 + 46.8 ms, 0.44 + 0.38;
// 128: 67.3 + 48.1, 0.53 + 0.44 (half the warps); 32: 76.4 + 64.8, 0.46 + 0.40 (a row
// comes from memory in four visits).  Copies of single floats are bound by the
// instructions around them: whole groups of 32 go a row after the other without
// any index arithmetic, only the remainder is numbered through (k_init at 200k x 33, 65, 99, 201,
// 257: 0.28, 0.41, 0.64, 1.34, 1.73 ms; all numbered through 0.39, 0.69, 0.96, 1.84, 2.31; with
// loads through registers, 32 dimensions at a time, 0.36, 0.54, 0.89, 2.01, 2.61).
constexpr int kStageCols = 64;
constexpr int kStageWarps = 4;  // per block

inline int stage_floats(const float *X, int d) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(X) | 4 * (uintptr_t)d;
  return (a & 15) == 0 ? 4 : (a & 7) == 0 ? 2 : 1;
}
__host__ __device__ constexpr int stage_pitch(int d, int kV) {
  return ((d < kStageCols ? d : kStageCols) / kV) | 1;
}
__host__ __device__ constexpr size_t stage_bytes(int d, int kV) {
  return (size_t)33 * stage_pitch(d, kV) * kV * 4;
}
// A launch needs no opt-in, which would be an attribute of the whole process.
static_assert(kStageWarps * stage_bytes(kStageCols, 4) <= 48 * 1024 &&
                  kStageWarps * stage_bytes(kStageCols, 2) <= 48 * 1024 &&
                  kStageWarps * stage_bytes(kStageCols, 1) <= 48 * 1024,
              "staged rows within the default shared memory");

template <int kV>
__device__ __forceinline__ float diffsum_staged(const float *__restrict__ X, int d, int64_t row,
                                                int32_t id, int m, float *__restrict__ sm) {
  const int lane = lane_id();
  const int pitch = stage_pitch(d, kV);
  auto copy = [&](float *dst, const float *src) {
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    if (kV == 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to), "l"(src) : "memory");
    else if (kV == 2)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(to), "l"(src) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(to), "l"(src) : "memory");
  };
  float *own = sm + 32 * pitch * kV;
  float s = 0.0f;
  for (int c0 = 0; c0 < d; c0 += kStageCols) {
    const int w = min(d - c0, kStageCols) / kV;
    // copies [first, w) of the m rows, numbered through: lane l takes l, l + 32, ...
    auto numbered = [&](int first) {
      const int n = w - first, dr = 32 / n, dq = 32 - dr * n;
      int r = lane / n, q = lane - r * n;
#pragma unroll 4
      for (int i = 0; i < m * n; i += 32) {
        const int32_t rid = __shfl_sync(0xffffffffu, id, r & 31);
        if (r < m) copy(sm + (r * pitch + first + q) * kV, X + (int64_t)rid * d + c0 + (first + q) * kV);
        r += dr;
        q += dq;
        if (q >= n) {
          q -= n;
          r++;
        }
      }
    };
    __syncwarp();  // the rows before are no longer read
    for (int q = lane; q < w; q += 32) copy(own + q * kV, X + row * d + c0 + q * kV);
    if (kV == 1 && w >= 32) {  // whole groups of 32 floats a row after the other
#pragma unroll 8
      for (int r = 0; r < m; r++) {
        const float *src = X + (int64_t)__shfl_sync(0xffffffffu, id, r) * d + c0 + lane;
        float *dst = sm + r * pitch + lane;
        copy(dst, src);
        if (w == 64) copy(dst + 32, src + 32);
      }
      if (w & 31) numbered(32);
    } else {
      numbered(0);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();  // every lane's copies have landed
    if (lane < m) {
      const float *mine = sm + lane * pitch * kV;
      if (kV == 4) {
#pragma unroll 4
        for (int p = 0; p < w; p++) {
          const float4 b = reinterpret_cast<const float4 *>(mine)[p];
          const float4 a = reinterpret_cast<const float4 *>(own)[p];
          const float2 d01 = neg_diff2(make_float2(b.x, b.y), make_float2(a.x, a.y));
          const float2 d23 = neg_diff2(make_float2(b.z, b.w), make_float2(a.z, a.w));
          s = __fmaf_rn(d01.x, d01.x, s);
          s = __fmaf_rn(d01.y, d01.y, s);
          s = __fmaf_rn(d23.x, d23.x, s);
          s = __fmaf_rn(d23.y, d23.y, s);
        }
      } else {
#pragma unroll 4
        for (int p = 0; p < w; p++) {
          const float df = __fsub_rn(own[p * kV], mine[p * kV]);
          s = __fmaf_rn(df, df, s);
          if (kV == 2) {
            const float dg = __fsub_rn(own[p * kV + 1], mine[p * kV + 1]);
            s = __fmaf_rn(dg, dg, s);
          }
        }
      }
    }
  }
  __syncwarp();
  return s;
}

// With instances (seg.count > 0) every row draws from its own instance with
// the instance-local position and size, so an instance starts from the graph
// a run on that instance alone starts from.  With a renumbering (order: new
// row -> caller's row, inv: caller's row -> new row; X in the new numbering)
// the ids are drawn for the caller's row from the caller's numbering and then
// mapped, so the lists are exactly the caller-numbered initial graph
// renumbered (instances keep their ranges under the renumbering).
template <int kV>
__global__ void __launch_bounds__(32 * kStageWarps, 8) k_init(const float *__restrict__ X, int64_t n, int d, int k, Segments seg,
                       const uint32_t *__restrict__ order, const int32_t *__restrict__ inv,
                       int32_t *__restrict__ gid, float *__restrict__ gdist,
                       float *__restrict__ worst) {
  extern __shared__ float smem_stage[];
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  float *sm = smem_stage + (threadIdx.x >> 5) * 33 * stage_pitch(d, kV) * kV;
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    int64_t base = 0, cnt = n;
    if (seg.count > 0) {
      const int32_t t = seg.of_point(row);
      base = seg.off[t];
      cnt = seg.off[t + 1] - base;
    }
    const int64_t lrow = (order ? (int64_t)order[row] : row) - base;
    // InitKNNGraphIndexKernel (nndescent.cu:1673-1692): xorshift64star(pos) % n,
    // advanced past the row itself -- and here also past ids already taken:
    // slot t takes the first of its draw, draw + 1, ... (mod n) that is
    // neither the row nor taken by a slot before it.  All slots advance
    // together, each while it equals the row or an earlier slot's current id
    // (one match_any per round); a slot never steps over its final id that
    // way (the ids it steps over are the row or earlier slots' final ids), so
    // the fixed point is that sequential result.  A slot steps at most k
    // times, so k * (k + 1) / 2 rounds bound the loop.
    const int32_t lrow32 = (int32_t)lrow, cnt32 = (int32_t)cnt;
    int32_t label = (int32_t)(xorshift64star((uint64_t)(lrow * k + lane)) % (uint64_t)cnt);
    const uint32_t below = lanemask_lt();
    for (int round = 0; round <= kMaxK * (kMaxK + 1) / 2; round++) {
      // lanes past k carry values no id takes
      const uint32_t same = __match_any_sync(0xffffffffu, lane < k ? label : (int32_t)(0x80000000u | lane));
      const bool step = lane < k && (label == lrow32 || (same & below) != 0);
      if (__ballot_sync(0xffffffffu, step) == 0) break;
      if (step) label = label + 1 == cnt32 ? 0 : label + 1;
    }
    int64_t lab64 = (int64_t)label + base;
    if (order && lane < k) lab64 = inv[lab64];
    const float ds = diffsum_staged<kV>(X, d, row, (int32_t)lab64, k, sm);
    uint64_t key = ~0ull;
    if (lane < k) key = pack(ds, (int32_t)lab64);
    key = warp_sort32(key);
    if (lane < k) {
      gid[row * k + lane] = pk_id(key);  // all "new"
      gdist[row * k + lane] = pk_dist(key);
    }
    float w = __shfl_sync(0xffffffffu, pk_dist(key), k - 1);
    if (lane == 0) worst[row] = w;
  }
}

// Initial graph of the merge of two point sets A = [0, n1) and B = [n1, n)
// (InitRandomBlockedKNNGraph, knnmerge.cu:80-185, then the distance pass and
// per-row sort of InitRandomKNNGraph nndescent.cu:1800-1871 that
// NNDescentForMerge :2013 runs on it), one warp per row: the first k - k/2
// entries of the row's own subgraph row (ids shifted into the merged
// numbering, flagged old as after MarkAllToOld), then k/2 ids of the other
// set drawn as xorshift64star(local row * (k/2) + t) % |other set|, flagged
// new.  An id drawn twice is advanced to the next free one (the reference
// keeps repeats), and every distance is the sequential FP32 difference sum of
// the join (the reference's distance pass sums over a warp tree).  The rows
// are sorted by (distance, id); an entry's flag follows from its set: ids of
// the other set are the new ones.  Own-subgraph ids outside their set, self
// ids and repeats set DEVERR_ID_RANGE / SELF / DUP and are replaced by a
// valid id of the set so that no gather leaves X.
template <int kV>
__global__ void __launch_bounds__(32 * kStageWarps, 8) k_merge_init(const float *__restrict__ X, int64_t n, int d, int k, int64_t n1,
                             const hdb_nnd_element *__restrict__ G1,
                             const hdb_nnd_element *__restrict__ G2, int32_t *__restrict__ gid,
                             float *__restrict__ gdist, float *__restrict__ worst,
                             uint32_t *__restrict__ err) {
  extern __shared__ float smem_stage[];
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  float *sm = smem_stage + (threadIdx.x >> 5) * 33 * stage_pitch(d, kV) * kV;
  const int h = k - k / 2, r = k / 2;
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    const bool inb = row >= n1;
    const int64_t local = inb ? row - n1 : row;
    const int64_t own_n = inb ? n - n1 : n1, own_off = inb ? n1 : 0;
    const int64_t oth_n = inb ? n1 : n - n1, oth_off = inb ? 0 : n1;
    const hdb_nnd_element *own = inb ? G2 : G1;
    int64_t label = 0;
    uint32_t bad = 0;
    if (lane < h) {
      label = decode(own[local * k + lane].label_);
      if (label < 0 || label >= own_n) {
        bad |= DEVERR_ID_RANGE;
        label = (local + 1 + lane) % own_n;
      } else if (label == local) {
        bad |= DEVERR_SELF_ID;
        label = (local + 1 + lane) % own_n;
      }
    } else if (lane < k) {
      label = (int64_t)(xorshift64star((uint64_t)(local * r + (lane - h))) % (uint64_t)oth_n);
    }
    // repeats among the own entries (input error) and among the drawn ones
    const uint32_t same = __match_any_sync(0xffffffffu, lane < h ? label : -1 - (int64_t)lane);
    if (lane < h && (__ffs(same) - 1) != lane) bad |= DEVERR_DUP_ID;
    for (int t = 0; t < r; t++) {
      while (true) {
        const int64_t c = __shfl_sync(0xffffffffu, label, h + t);
        const bool dup = lane >= h && lane < h + t && label == c;
        if (__ballot_sync(0xffffffffu, dup) == 0) break;
        if (lane == h + t) label = (label + 1) % oth_n;
      }
    }
    const uint32_t anybad = __reduce_or_sync(0xffffffffu, bad);
    if (anybad && lane == 0) atomicOr(err, anybad);
    if (anybad & DEVERR_DUP_ID) {
      // keep the rows valid: the own half becomes the next h ids of its set
      if (lane < h) label = (local + 1 + lane) % own_n;
    }
    label += lane < h ? own_off : oth_off;
    const float ds = diffsum_staged<kV>(X, d, row, (int32_t)label, k, sm);
    uint64_t key = ~0ull;
    if (lane < k) key = pack(ds, (int32_t)label);
    key = warp_sort32(key);
    if (lane < k) {
      const int32_t id = pk_id(key);
      const bool isnew = (id >= n1) != inb;
      gid[row * k + lane] = isnew ? id : -id - 1;
      gdist[row * k + lane] = pk_dist(key);
    }
    const float w = __shfl_sync(0xffffffffu, pk_dist(key), k - 1);
    if (lane == 0) worst[row] = w;
  }
}

// Offers a chunk of up to 32 candidates (one per lane, ~0 for none) to the
// row held one sorted entry per lane (lane < k; key = (distance, id)).  Only
// candidates below the row's current k-th key can enter, and the k-th key
// never grows, so those are found with one ballot; each is then placed by
// rank (ballot of the keys below it) unless its id is already listed, the
// entries above it moving up one lane and the last one dropping out.  The
// result is the first k distinct ids of the union in key order, whatever the
// order of the candidates.  Inserted entries carry the "new" flag.
template <bool kCheckIds = true>
__device__ __forceinline__ void insert_chunk(int k, uint64_t &rkey, int32_t &lab, uint64_t cand) {
  const int lane = lane_id();
  const bool have = lane < k;
  const uint64_t kth = __shfl_sync(0xffffffffu, rkey, k - 1);
  uint32_t todo = __ballot_sync(0xffffffffu, cand < kth);
  while (todo) {
    const int t = __ffs(todo) - 1;
    todo &= todo - 1;
    const uint64_t c = __shfl_sync(0xffffffffu, cand, t);
    const int pos = __popc(__ballot_sync(0xffffffffu, have && rkey < c));
    if (pos >= k) continue;
    const int32_t cid = pk_id(c);
    if (kCheckIds && __any_sync(0xffffffffu, have && pk_id(rkey) == cid)) continue;
    const uint64_t up = __shfl_up_sync(0xffffffffu, rkey, 1);
    const int32_t uplab = __shfl_up_sync(0xffffffffu, lab, 1);
    if (lane == pos) {
      rkey = c;
      lab = cid;
    } else if (have && lane > pos) {
      rkey = up;
      lab = uplab;
    }
  }
}

// Rank of x among the sorted keys held by lanes 0..m-1 (number of keys
// below x), by binary search over shuffled lanes; every lane its own x.
__device__ __forceinline__ int rank_in_lanes(uint64_t sorted, int m, uint64_t x) {
  int lo = 0, hi = m;
#pragma unroll
  for (int it = 0; it < 6; it++) {  // 2^6 > 33 possible answers
    const int mid = (lo + hi) >> 1;
    const uint64_t v = __shfl_sync(0xffffffffu, sorted, mid & 31);
    if (lo < hi) {
      if (v < x) lo = mid + 1; else hi = mid;
    }
  }
  return lo;
}

// Per-warp shared memory of the merge: an open-addressing table of the ids
// seen (128 slots, -1 empty), the compacted survivors of a batch, and the
// merged row.
constexpr int kMergeTable = 128;
struct MergeSmem {
  int32_t tbl[kMergeTable];
  uint64_t stage[64];
  uint64_t sk[32];
  int32_t sl[32];
};

// Inserts id into the table; true if it was not there yet.  A batch puts at
// most 32 + 64 ids into the 128 slots, so a free slot is always found.
__device__ __forceinline__ bool table_insert(int32_t *tbl, int32_t id) {
  uint32_t h = ((uint32_t)id * 0x9E3779B1u) >> 25;
  for (int probe = 0; probe < kMergeTable; probe++) {
    const int32_t prev = atomicCAS(&tbl[h], -1, id);
    if (prev == -1) return true;
    if (prev == id) return false;
    h = (h + 1) & (kMergeTable - 1);
  }
  return false;
}

// Offers up to 64 candidates (c0, c1 per lane; ~0 for none) to the row held
// one sorted entry per lane (lane < k; key = (distance, id)), with the same
// result as insert_chunk on each of them.  Candidates at or above the row's
// k-th key cannot enter (the k-th key never grows).  The others go through a
// per-warp hash table holding the row's ids first, so a candidate whose id
// is listed or was already offered in the batch drops out (a pair's repeats
// carry equal keys, so which one stays does not matter); the survivors are
// compacted and either inserted one at a time (few) or sorted across the
// lanes and merged by rank -- each side finds its rank in the other by binary
// search -- with the first k entries placed through shared memory.
__device__ __forceinline__ void merge_batch(int k, uint64_t &rkey, int32_t &lab, uint64_t c0,
                                            uint64_t c1, MergeSmem &ms) {
  const int lane = lane_id();
  const bool have = lane < k;
  const uint64_t kth = __shfl_sync(0xffffffffu, rkey, k - 1);
  bool ok0 = c0 < kth, ok1 = c1 < kth;
  if (!__any_sync(0xffffffffu, ok0 || ok1)) return;
#pragma unroll
  for (int j = 0; j < kMergeTable / 32; j++) ms.tbl[lane + 32 * j] = -1;
  __syncwarp();
  if (have) table_insert(ms.tbl, pk_id(rkey));
  __syncwarp();
  if (ok0) ok0 = table_insert(ms.tbl, pk_id(c0));
  if (ok1) ok1 = table_insert(ms.tbl, pk_id(c1));
  const uint32_t b0 = __ballot_sync(0xffffffffu, ok0), b1 = __ballot_sync(0xffffffffu, ok1);
  const int nsurv = __popc(b0) + __popc(b1);
  if (nsurv == 0) return;
  const uint32_t lt = lanemask_lt();
  if (ok0) ms.stage[__popc(b0 & lt)] = c0;
  if (ok1) ms.stage[__popc(b0) + __popc(b1 & lt)] = c1;
  __syncwarp();
  for (int base = 0; base < nsurv; base += 32) {
    const int nc = min(32, nsurv - base);
    const uint64_t cand = lane < nc ? ms.stage[base + lane] : ~0ull;
    if (nc <= 12) {
      insert_chunk<false>(k, rkey, lab, cand);
      continue;
    }
    const uint64_t c = warp_sort32(cand);                // survivors in lanes 0..nc-1
    const int pos_r = lane + rank_in_lanes(c, nc, rkey);  // row entry: its merged rank
    const int pos_c = lane + rank_in_lanes(rkey, k, c);   // candidate: its merged rank
    __syncwarp();
    if (have && pos_r < k) {
      ms.sk[pos_r] = rkey;
      ms.sl[pos_r] = lab;
    }
    if (lane < nc && pos_c < k) {
      ms.sk[pos_c] = c;
      ms.sl[pos_c] = pk_id(c);  // inserted as "new"
    }
    __syncwarp();
    if (have) {
      rkey = ms.sk[lane];
      lab = ms.sl[lane];
    }
  }
}

// Sample (PrepareGraph :44-98 and reverse samples PrepareReverseGraph :293-346)
// and MarkAllToOld (:1398) of one row held one entry per lane.  split > 0 is
// the merge of two point sets [0, split) and [split, n) (PrepareGraphForMerge
// :100-166): old entries are sampled only from the row's own set; new entries
// and reverse samples are not filtered.
struct SampleOut {
  int32_t *newS, *oldS;  // [n][2S]: forward slots 0..S-1, reverse slots S..2S-1
  int8_t *nf, *of;       // [n] forward samples
  int32_t *nrev, *orev;  // [n] reverse samples offered
};
// The candidate list grouped by row.
struct RowList {
  const uint32_t *start;     // [n + 1]
  const uint64_t *key;
  unsigned long long *best;  // [n] the best candidate of each row that found no room in the list
};

__device__ __forceinline__ void sample_row(int64_t row, int k, int S, int64_t split, int32_t lab,
                                           float dist, int32_t *__restrict__ gid,
                                           float *__restrict__ gdist, float *__restrict__ worst,
                                           const SampleOut &so) {
  const int lane = lane_id();
  const bool have = lane < k;
  const int32_t id = decode(lab);
  const bool isnew = have && lab >= 0;
  const bool isold = have && lab < 0 && (split <= 0 || ((row < split) == (id < split)));
  const uint32_t nm = __ballot_sync(0xffffffffu, isnew), om = __ballot_sync(0xffffffffu, isold);
  const int rn = __popc(nm & lanemask_lt()), ro = __popc(om & lanemask_lt());
  const int64_t sb = row * (2 * S);
  if (isnew && rn < S) {
    so.newS[sb + rn] = id;
    const int p = atomicAdd(&so.nrev[id], 1);
    if (p < S) so.newS[(int64_t)id * (2 * S) + S + p] = (int32_t)row;
  }
  if (isold && ro < S) {
    so.oldS[sb + ro] = id;
    const int p = atomicAdd(&so.orev[id], 1);
    if (p < S) so.oldS[(int64_t)id * (2 * S) + S + p] = (int32_t)row;
  }
  if (lane == 0) {
    so.nf[row] = (int8_t)min(__popc(nm), S);
    so.of[row] = (int8_t)min(__popc(om), S);
  }
  if (have) {
    gid[row * k + lane] = isnew ? -id - 1 : lab;  // MarkAllToOld
    gdist[row * k + lane] = dist;
  }
  const float w = __shfl_sync(0xffffffffu, dist, k - 1);
  if (lane == 0) worst[row] = w;
}

// Merge of a row's part of the candidate list, and of the best candidate that
// found no room in it (normally none), into its sorted list (one warp), in
// batches of 64.  On return, lane j (< k) holds the j-th entry of the merged row.
__device__ __forceinline__ void merge_row(int64_t row, int k, int32_t &lab, float &dist,
                                          const RowList &rl, MergeSmem &ms) {
  const int lane = lane_id();
  const uint64_t ov = rl.best[row];
  const uint32_t o0 = rl.start[row], o1 = rl.start[row + 1];
  if (ov == ~0ull && o0 == o1) return;
  __syncwarp();
  if (lane == 0 && ov != ~0ull) rl.best[row] = ~0ull;
  const bool have = lane < k;
  uint64_t rkey = have ? pack(dist, decode(lab)) : ~0ull;
  const int64_t nov = ov != ~0ull ? 1 : 0;
  const int64_t m = nov + (int64_t)(o1 - o0);
  auto at = [&](int64_t i) -> uint64_t { return i < nov ? ov : rl.key[o0 + (i - nov)]; };
  for (int64_t base = 0; base < m; base += 64) {
    const uint64_t c0 = base + lane < m ? at(base + lane) : ~0ull;
    const uint64_t c1 = base + 32 + lane < m ? at(base + 32 + lane) : ~0ull;
    merge_batch(k, rkey, lab, c0, c1, ms);
  }
  if (have) dist = pk_dist(rkey);
}

// Merge (iterations >= 1), sample and MarkAllToOld, one warp per row.  The order
// in which rows arrive decides whose reverse samples are taken (a row keeps the
// first S).  It follows the blocks that are resident together -- the grid's
// first five per SM walk through all their rows before the others start -- so
// the shared memory's share of L1 (kSampleShare, 64 KB for 12 KB a block) keeps
// it at five blocks whatever the compiler makes of the registers: another order
// gives graphs as good, but other ones.
constexpr int kSampleShare = 28;  // per cent
__global__ void k_sample(int64_t n, int k, int S, int do_merge, int32_t *__restrict__ gid,
                         float *__restrict__ gdist, float *__restrict__ worst, RowList rl,
                         unsigned long long *counters, SampleOut so, int64_t split) {
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  __shared__ MergeSmem merge_smem[8];  // per-warp merge scratch (8 warps per block)
  MergeSmem &ms = merge_smem[threadIdx.x >> 5];
  if (blockIdx.x == 0 && threadIdx.x == 0) counters[3] = 0;  // the next join's list is empty
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    const bool have = lane < k;
    int32_t lab = have ? gid[row * k + lane] : 0;
    float dist = have ? gdist[row * k + lane] : 0.0f;
    if (do_merge) merge_row(row, k, lab, dist, rl, ms);
    sample_row(row, k, S, split, lab, dist, gid, gdist, worst, so);
  }
}

// Final merge after the last join; writes NNDElement rows with their flags.
__global__ void k_finalize(int64_t n, int k, const int32_t *__restrict__ gid,
                           const float *__restrict__ gdist, RowList rl,
                           hdb_nnd_element *__restrict__ out) {
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  __shared__ MergeSmem merge_smem[8];  // per-warp merge scratch (8 warps per block)
  MergeSmem &ms = merge_smem[threadIdx.x >> 5];
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    int32_t lab = lane < k ? gid[row * k + lane] : 0;
    float dist = lane < k ? gdist[row * k + lane] : 0.0f;
    merge_row(row, k, lab, dist, rl, ms);
    if (lane < k) out[row * k + lane] = hdb_nnd_element{dist, lab};
  }
}

// The candidate list grouped by bucket of 2^shift consecutive rows (bstart)
// -> grouped by row: one block per bucket counts its rows' candidates in shared
// memory, scans the counts (the rows' starts) and moves the keys to their
// rows.  A bucket's part is some 50 KB, so its scattered 8-byte stores meet in
// L2.  In place of a further pass of the radix sort and of the search for the
// rows' bounds in the sorted targets.
constexpr int kGroupThreads = 512;
__global__ void __launch_bounds__(kGroupThreads)
    k_group_rows(int64_t n, int shift, const uint32_t *__restrict__ tgt,
                 const uint64_t *__restrict__ key, const uint32_t *__restrict__ bstart,
                 uint32_t *__restrict__ start, uint64_t *__restrict__ out) {
  __shared__ uint32_t cnt[kBucketRows];
  __shared__ uint32_t wsum[kBucketRows / 32];
  const int lane = lane_id(), w = threadIdx.x >> 5, tid = threadIdx.x;
  const uint32_t row0 = (uint32_t)((int64_t)blockIdx.x << shift);
  const int rows = (int)min((int64_t)1 << shift, n - (int64_t)row0);
  const uint32_t b0 = bstart[blockIdx.x], b1 = bstart[blockIdx.x + 1];  // the unused slots lie behind
  if (tid < kBucketRows) cnt[tid] = 0;
  __syncthreads();
#pragma unroll 4
  for (uint32_t i = b0 + tid; i < b1; i += kGroupThreads) atomicAdd(&cnt[tgt[i] - row0], 1u);
  __syncthreads();
  const uint32_t c = tid < kBucketRows ? cnt[tid] : 0;
  uint32_t x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31 && w < kBucketRows / 32) wsum[w] = x;
  __syncthreads();
  uint32_t at = b0 + x - c;
  if (tid < kBucketRows) {
    for (int v = 0; v < w; v++) at += wsum[v];
    cnt[tid] = at;
  }
  if (tid < rows) start[row0 + tid] = at;
  if (tid == rows - 1 && (int64_t)row0 + rows == n) start[n] = at + c;
  __syncthreads();
#pragma unroll 4
  for (uint32_t i = b0 + tid; i < b1; i += kGroupThreads)
    out[atomicAdd(&cnt[tgt[i] - row0], 1u)] = key[i];
}

// Start of every bucket in the list grouped by bucket (tgt >> shift), and the
// end of the last one: bstart[0..buckets].  A warp searches one bucket's start, 32
// probes a step.  Six lists of 10M x 12: 0.37 ms, 4.35 with the list read through;
// 1M x 64: 0.07 and 0.39.
__global__ void k_bucket_bounds(const uint32_t *__restrict__ tgt,
                                const unsigned long long *__restrict__ count, int64_t cap, int shift,
                                int64_t buckets, uint32_t *__restrict__ bstart) {
  const int lane = lane_id();
  const int64_t c = min((int64_t)*count, cap);
  const int64_t stride = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b <= buckets; b += stride) {
    int64_t lo = 0, hi = c;  // the start lies in [lo, hi]
    while (lo < hi) {
      const int64_t step = (hi - lo + 31) / 32;
      const int64_t p = lo + (lane + 1) * step - 1;
      const bool less = p < hi && (int64_t)(tgt[p] >> shift) < b;
      lo += __popc(__ballot_sync(0xffffffffu, less)) * step;
      hi = min(hi, lo + step - 1);
    }
    if (lane == 0) bstart[b] = (uint32_t)min(lo, c);
  }
}

// ---- FP32 local join -----------------------------------------------------
constexpr int kJoinWarps = 8;

// A row's counts and both sample lists in one memory round trip, loaded one row
// ahead so that they are in flight while the previous row is joined.
struct SlotLists {
  int32_t nraw = 0, oraw = 0;
  int cnf = 0, cof = 0, cnr = 0, cor = 0;
  __device__ __forceinline__ void load(int64_t r, int64_t n, int S, const int32_t *__restrict__ newS,
                                       const int32_t *__restrict__ oldS, const int8_t *__restrict__ nf,
                                       const int8_t *__restrict__ of, const int32_t *nrev,
                                       const int32_t *orev) {
    if (r >= n) return;
    const int lane = lane_id();
    const int64_t sb = r * (2 * S);
    nraw = lane < 2 * S ? newS[sb + lane] : 0;
    oraw = lane < 2 * S ? oldS[sb + lane] : 0;
    cnf = nf[r];
    cof = of[r];
    cnr = nrev[r];
    cor = orev[r];
  }
  // The slots in use: new rows into ids[0..nn), old ones into ids[32..32+no).
  __device__ __forceinline__ void compact(int S, int32_t *ids, int &nn, int &no) const {
    const int lane = lane_id();
    const int nr = min(cnr, S), orv = min(cor, S);
    // slot t < S: forward sample t; slot S + t: reverse sample t
    bool vn = (lane < S) ? (lane < cnf) : (lane < 2 * S && lane - S < nr);
    bool vo = (lane < S) ? (lane < cof) : (lane < 2 * S && lane - S < orv);
    const int32_t nid = vn ? nraw : -1 - lane;
    const int32_t oid = vo ? oraw : -100 - lane;
    // de-duplicate (ShrinkGraph RemoveDuplicates, :285-291)
    const uint32_t pn = __match_any_sync(0xffffffffu, nid);
    vn = vn && (__ffs(pn) - 1 == lane);
    const uint32_t po = __match_any_sync(0xffffffffu, oid);
    vo = vo && (__ffs(po) - 1 == lane);
    const uint32_t bo = __ballot_sync(0xffffffffu, vo);
    no = __popc(bo);
    if (vo) ids[32 + __popc(bo & lanemask_lt())] = oid;
    __syncwarp();
    // new \ old (:468-486)
    bool in_old = false;  // independent reads, not a chain
#pragma unroll 8
    for (int t = 0; t < no; t++) in_old |= ids[32 + t] == nid;
    vn = vn && !in_old;
    const uint32_t bn = __ballot_sync(0xffffffffu, vn);
    nn = __popc(bn);
    if (vn) ids[__popc(bn & lanemask_lt())] = nid;
    __syncwarp();
  }
};

// floor(x / m) for 1 <= m <= 8 and 0 <= x < 1024: x * ceil(2^16 / m) >> 16.
__constant__ uint32_t kRecip[9] = {0, 65536, 32768, 21846, 16384, 13108, 10923, 9363, 8192};
__device__ __forceinline__ int div_small(int x, int m) { return (int)(((uint32_t)x * kRecip[m]) >> 16); }

// Shared memory of one warp: best candidates (distance bits, then ids: best
// other-new and best old per new row; best new per old row) | slot ids | a chunk
// of kJc dimensions of every staged row (new rows, then old ones).  A staged row
// takes nine 16-byte pieces of which eight hold data: rows that follow one another
// then start in different bank groups.
constexpr int kJc = 32;         // dimensions per staged chunk
constexpr int kJPitch = kJc / 4 + 1;
constexpr int kJCols = 8;       // most columns of a tile
struct JoinSmem {
  static constexpr int kBest = 96;   // distances and ids
  static constexpr int kIds = 64;
  static constexpr int kChunk = 64 * kJPitch;  // 16-byte pieces
  static constexpr size_t kBytes = kBest * 8 + kIds * 4 + (size_t)kChunk * 16;
};

// Copies dimensions [c0, c0 + 4 * nq) of the nn new and no old rows: 16-byte
// cp.async copies when every row piece is 16-byte aligned (d % 4 == 0; one
// group is committed), else scalar loads, zero padded to a multiple of four
// (adding fmaf(0, 0, s) = s leaves every sum unchanged).
__device__ __forceinline__ void stage_chunk(const float *__restrict__ X, int d, int c0, int nq,
                                            const int32_t *ids, int nn, int T, float4 *Xs, bool vec) {
  const int lane = lane_id();
  const int items = T * nq;
  for (int it = lane; it < items; it += 32) {
    const int r = nq == kJc / 4 ? it / (kJc / 4) : div_small(it, nq), q = it - r * nq;
    const float *src = X + (int64_t)ids[r < nn ? r : 32 + r - nn] * d + c0 + 4 * q;
    float4 *dst = Xs + r * kJPitch + q;
    if (vec) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(dst)),
                   "l"(src)
                   : "memory");
    } else {
      const int left = d - c0 - 4 * q;
      float4 v;
      v.x = left > 0 ? __ldg(src) : 0.0f;
      v.y = left > 1 ? __ldg(src + 1) : 0.0f;
      v.z = left > 2 ? __ldg(src + 2) : 0.0f;
      v.w = left > 3 ? __ldg(src + 3) : 0.0f;
      *dst = v;
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Adds a staged chunk's nq pieces to the sums of four rows (from piece `ra`)
// and cw columns (from piece `cb`, `step` pieces apart, none past `last`).  One
// loop with a way out after each column: a loop for every width runs 1.5x slower,
// as the warps of an SM, each at another width, then miss the instruction cache.
__device__ __forceinline__ void tile_sums(float (&acc)[4][kJCols], const float4 *Xs, int ra, int cb,
                                          int step, int last, int nq, int cw) {
#pragma unroll 2
  for (int q = 0; q < nq; q++) {
    float4 xa[4], xc = Xs[cb + q];
#pragma unroll
    for (int i = 0; i < 4; i++) xa[i] = Xs[ra + i * kJPitch + q];
#pragma unroll
    for (int j = 0; j < kJCols; j++) {
      const float4 next = Xs[min(cb + (j + 1) * step, last) + q];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float2 d01 = neg_diff2(make_float2(xc.x, xc.y), make_float2(xa[i].x, xa[i].y));
        const float2 d23 = neg_diff2(make_float2(xc.z, xc.w), make_float2(xa[i].z, xa[i].w));
        float s_ = __fmaf_rn(d01.x, d01.x, acc[i][j]);
        s_ = __fmaf_rn(d01.y, d01.y, s_);
        s_ = __fmaf_rn(d23.x, d23.x, s_);
        acc[i][j] = __fmaf_rn(d23.y, d23.y, s_);
      }
      if (j + 1 >= cw) break;
      xc = next;
    }
  }
}

// Local join, one warp per row (UpdateGraph, nndescent.cu:1487-1580).  With the
// new rows first and the old ones behind them (T in all), the pairs are (a, c)
// with a new row a < c.  Four rows at a time (group i: rows 4i .. 4i + 3, columns
// from 4i) they are cut into tiles of cw columns, a group's tile l taking every
// n_i-th column from the l-th on; cw is the least that gives every tile of the
// row-join a lane of its own, up to kJCols (row-joins that need more take further
// passes over the rows).  A lane keeps its tile's sums in registers while the rows
// pass through shared memory a chunk of kJc dimensions at a time, so every pair is
// the reference's sequential FP32 difference sum over j = 0..d-1.  The tiles' row
// and column minima meet in shared memory: first the least distance of every slot
// (its bits, a 32-bit atomicMin), then, among the pairs at that distance, the
// least id.  Every new neighbour gets its closest other new one and its closest
// old one, every old neighbour its closest new one.  cross_only (the merge join,
// TiledNewOldNeighborsCompareKernelForMerge :1328-1383 launched without the new x
// new kernel, UpdateGraphForMerge :1582-1640) leaves out the new x new pairs: new
// neighbours get their closest old one only.
//
// Bound by instruction issue with the FMA and shared-memory pipes close behind (68,
// 55 and 60 % at 200k x 128, k = 32): a row-join's pairs give a lane some 30 sums, so
// 11 operand loads feed 28 pairs and no more.  Against tiles of 4 x 4, one or two per lane
// (the last slot of them mostly empty), six iterations: 200k x 128, k = 16 8.4 ->
// 6.0 ms, k = 32 12.9 -> 12.3; 1M x 64, k = 32 37.9 -> 37.3; 100k x 784 35.2 ->
// 33.2.  Chunks of 16 dimensions with the next on its way are 4 % slower than
// chunks of 32 without, five columns at three blocks per SM 10-20 %, twenty warps
// per SM at 96 registers (sixteen at 128) 10-14 %.
__global__ void __launch_bounds__(32 * kJoinWarps, 2)
    k_join(const float *__restrict__ X, int64_t n, int d, int S, const int32_t *__restrict__ newS,
           const int32_t *__restrict__ oldS, const int8_t *__restrict__ nf,
           const int8_t *__restrict__ of, int32_t *__restrict__ nrev, int32_t *__restrict__ orev,
           const float *__restrict__ worst, CandList cl, int cross_only) {
  extern __shared__ __align__(16) unsigned char smem_join[];
  using Smem = JoinSmem;
  const int lane = lane_id();
  unsigned char *base = smem_join + (threadIdx.x >> 5) * Smem::kBytes;
  uint32_t *bdist = reinterpret_cast<uint32_t *>(base);
  uint32_t *bid = bdist + Smem::kBest;
  int32_t *ids = reinterpret_cast<int32_t *>(base + Smem::kBest * 8);
  float4 *Xs = reinterpret_cast<float4 *>(base + Smem::kBest * 8 + Smem::kIds * 4);
  const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  unsigned long long w_rows = 0, w_cands = 0, w_pairs = 0;
  ListCursor cur;  // this warp's space in the candidate list
  const int64_t stride = (int64_t)gridDim.x * kJoinWarps;
  const int chunks = (d + kJc - 1) / kJc;
  SlotLists lists;
  int64_t row = (int64_t)blockIdx.x * kJoinWarps + (threadIdx.x >> 5);
  lists.load(row, n, S, newS, oldS, nf, of, nrev, orev);
  for (; row < n; row += stride) {
    int nn, no;
    {
      const SlotLists mine = lists;
      lists.load(row + stride, n, S, newS, oldS, nf, of, nrev, orev);
      __syncwarp();
      if (lane == 0) { nrev[row] = 0; orev[row] = 0; }
      mine.compact(S, ids, nn, no);
    }
    if (nn == 0 || nn + no < 2 || (cross_only && no == 0)) continue;
    const int T = nn + no;
    w_rows += T;
    w_pairs += (cross_only ? 0 : nn * (nn - 1) / 2) + nn * no;  // the reference's pairs
#pragma unroll
    for (int g = 0; g < Smem::kBest; g += 32) bdist[g + lane] = bid[g + lane] = 0xffffffffu;
    // lane i < rg: the columns of row group i
    const int rg = (nn + 3) >> 2;
    const int first_col = cross_only ? nn : 4 * lane;
    const int len = lane < rg ? T - first_col : 0;
    int cw = kJCols;
    int tiles_i = div_small(len + cw - 1, cw);  // of group `lane`
    int tiles = __reduce_add_sync(0xffffffffu, tiles_i);
    while (cw > 1 && tiles <= 32) {  // narrower, as long as a slot holds them
      const int t_i = div_small(len + cw - 2, cw - 1);
      const int t = __reduce_add_sync(0xffffffffu, t_i);
      if (t > 32) break;
      cw--;
      tiles_i = t_i;
      tiles = t;
    }
    int upto = tiles_i;  // tiles of the groups up to and with `lane`'s
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    uint32_t before[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu};
    for (int t0 = 0; t0 < tiles; t0 += 32) {
      // tile t0 + lane: its row group, columns c0, c0 + step, ...
      const int t = t0 + lane;
      int grp = 0;
#pragma unroll
      for (int r = 0; r < 7; r++) grp += t >= __shfl_sync(0xffffffffu, upto, r) ? 1 : 0;
      grp = min(grp, rg - 1);
      const int step = __shfl_sync(0xffffffffu, tiles_i, grp);
      const int start = __shfl_sync(0xffffffffu, upto, grp) - step;
      const int r0 = 4 * grp, c0 = (cross_only ? nn : r0) + t - start;
      const bool mine = t < tiles;
      float acc[4][kJCols];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < kJCols; j++) acc[i][j] = 0.0f;
      const int last = (T - 1) * kJPitch;
      const int ra = r0 * kJPitch, cb = min(mine ? c0 : 0, T - 1) * kJPitch;
      __syncwarp();  // the staged rows of the pass before are no longer read; ids are written
      stage_chunk(X, d, 0, min(kJc / 4, (d + 3) >> 2), ids, nn, T, Xs, vec);
      for (int ch = 0; ch < chunks; ch++) {
        const int nq = min(kJc / 4, (d - ch * kJc + 3) >> 2);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
        tile_sums(acc, Xs, ra, cb, step * kJPitch, last, nq, cw);
        __syncwarp();  // this chunk is no longer read
        if (ch + 1 < chunks)
          stage_chunk(X, d, (ch + 1) * kJc, min(kJc / 4, (d - (ch + 1) * kJc + 3) >> 2), ids, nn, T, Xs,
                      vec);
      }
      // the least distances; what is no pair of the join gets all ones
      {
        uint32_t rnew[4], rold[4];
#pragma unroll
        for (int i = 0; i < 4; i++) rnew[i] = rold[i] = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < kJCols; j++) {
          if (j >= cw) break;  // for the whole warp
          const int c = c0 + j * step;
          const bool there = mine && c < T, old = c >= nn;
          uint32_t cmin = 0xffffffffu;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            uint32_t v = __float_as_uint(acc[i][j]);
            if (!there || r0 + i >= nn || r0 + i >= c) v = 0xffffffffu;
            acc[i][j] = __uint_as_float(v);
            cmin = min(cmin, v);
            rnew[i] = min(rnew[i], old ? 0xffffffffu : v);
            rold[i] = min(rold[i], old ? v : 0xffffffffu);
          }
          if (cmin != 0xffffffffu) atomicMin(&bdist[old ? 64 + c - nn : c], cmin);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
          if (rnew[i] != 0xffffffffu) atomicMin(&bdist[r0 + i], rnew[i]);
          if (rold[i] != 0xffffffffu) atomicMin(&bdist[32 + r0 + i], rold[i]);
        }
      }
      __syncwarp();
      if (t0 > 0) {  // a slot whose least distance this pass has lowered starts over
#pragma unroll
        for (int g = 0; g < 3; g++) {
          const uint32_t now = bdist[32 * g + lane];
          if (now != before[g]) bid[32 * g + lane] = 0xffffffffu;
        }
        __syncwarp();
      }
#pragma unroll
      for (int g = 0; g < 3; g++) before[g] = bdist[32 * g + lane];
      // the least ids at those distances: first which pairs are at a minimum (bit
      // 4 j + i; unrolled, as the sums are in registers), then a loop over those few
      uint32_t at_row = 0, at_col = 0;
      {
        // no pair of the join: a value that no sum takes
        auto held = [](uint32_t v) { return v == 0xffffffffu ? 0xfffffffeu : v; };
        const uint4 mn = *reinterpret_cast<const uint4 *>(bdist + r0);
        const uint4 mo = *reinterpret_cast<const uint4 *>(bdist + 32 + r0);
        const uint32_t mns[4] = {held(mn.x), held(mn.y), held(mn.z), held(mn.w)};
        const uint32_t mos[4] = {held(mo.x), held(mo.y), held(mo.z), held(mo.w)};
#pragma unroll
        for (int j = 0; j < kJCols; j++) {
          if (j >= cw) break;  // for the whole warp
          const int c = min(c0 + j * step, T - 1);
          const bool old = c >= nn;
          const uint32_t cm = held(bdist[old ? 64 + c - nn : c]);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const uint32_t v = __float_as_uint(acc[i][j]);
            at_row |= v == (old ? mos[i] : mns[i]) ? 1u << (4 * j + i) : 0u;
            at_col |= v == cm ? 1u << (4 * j + i) : 0u;
          }
        }
      }
      for (uint32_t m = at_row | at_col; m; m &= m - 1) {
        const int b = __ffs(m) - 1, i = b & 3, c = c0 + (b >> 2) * step;
        const bool old = c >= nn;
        if ((at_row >> b) & 1) atomicMin(&bid[(old ? 32 : 0) + r0 + i], (uint32_t)ids[old ? 32 + c - nn : c]);
        if ((at_col >> b) & 1) atomicMin(&bid[old ? 64 + c - nn : c], (uint32_t)ids[r0 + i]);
      }
    }  // passes
    __syncwarp();
    // the candidates that can enter their target's list go to the candidate
    // list (space reserved a chunk at a time; no returning atomic per candidate)
    const int32_t x = lane < nn ? ids[lane] : 0, x3 = lane < no ? ids[32 + lane] : 0;
    const uint32_t d1 = bdist[lane], d2 = bdist[32 + lane], d3 = bdist[64 + lane];
    const float wx = lane < nn ? worst[x] : 0.0f, wx3 = lane < no ? worst[x3] : 0.0f;
    auto key = [&](uint32_t dist, int at) { return ((uint64_t)dist << 32) | bid[at]; };
    const bool v1 = lane < nn && d1 != 0xffffffffu && __uint_as_float(d1) < wx;
    const bool v2 = lane < nn && d2 != 0xffffffffu && __uint_as_float(d2) < wx;
    const bool v3 = lane < no && d3 != 0xffffffffu && __uint_as_float(d3) < wx3;
    const bool av[3] = {v1, v2, v3};
    const int32_t at[3] = {x, x, x3};
    const uint64_t ak[3] = {key(d1, lane), key(d2, 32 + lane), key(d3, 64 + lane)};
    w_cands += append_candidates(cl, cur, av, at, ak);
    __syncwarp();
  }
  list_fill(cl, cur.pos, cur.end);  // the rest of the last chunk
  // per-warp totals, one atomic each (no block-wide barrier)
#pragma unroll
  for (int o = 16; o; o >>= 1) w_cands += __shfl_xor_sync(0xffffffffu, w_cands, o);
  if (lane == 0) {
    if (w_rows) atomicAdd(&cl.counters[1], w_rows);
    if (w_cands) atomicAdd(&cl.counters[2], w_cands);
    if (w_pairs) atomicAdd(&cl.counters[4], w_pairs);
  }
}

// ---- FP32 local join of short rows ------------------------------------------
// The same join for d <= 28 (kQ = ceil(d / 4) 16-byte pieces a row): with so
// few dimensions the sums are a small part of the work, and what the tiles need
// around them (the tiles' places, their minima meeting in shared memory) is
// more than they save.  Here a lane holds one new row in registers and takes the
// other staged rows one after the other, each read by all lanes at once; the
// row's closest new and old rows are running minima of the lane, an old row's
// closest new row is a minimum over the warp.  With at most 16 (8) new rows the
// warp's halves (quarters) take every second (fourth) staged row.  Bound by
// instruction issue (76 % of the slots at 1M x 12, 1,715 warp instructions a
// row-join).
//
// Where the line lies, by the join time of six iterations, rows against tiles: 1M
// points, k = 32: d = 8 9.7 / 14.7 ms, 12 12.2 / 18.2, 16 15.5 / 20.0, 24 19.2 /
// 22.6, 28 21.4 / 25.1, 32 27.4 / 24.9; 300k, k = 16: d = 31 4.74 / 4.65 ms; 50k x 8,
// k = 16: 0.40 / 0.58; 1,500 x 8: 0.076 / 0.080.
constexpr int kRowJoinMaxDim = 28;

template <int kQ>
__device__ __forceinline__ float row_dist(const float4 *__restrict__ b, const float4 (&own)[kQ]) {
  float s = 0.0f;
#pragma unroll
  for (int q = 0; q < kQ; q++) {
    const float4 x = b[q];
    const float2 d01 = neg_diff2(make_float2(x.x, x.y), make_float2(own[q].x, own[q].y));
    const float2 d23 = neg_diff2(make_float2(x.z, x.w), make_float2(own[q].z, own[q].w));
    s = __fmaf_rn(d01.x, d01.x, s);
    s = __fmaf_rn(d01.y, d01.y, s);
    s = __fmaf_rn(d23.x, d23.x, s);
    s = __fmaf_rn(d23.y, d23.y, s);
  }
  return s;
}

template <int kQ>
__global__ void __launch_bounds__(32 * kJoinWarps, kQ <= 4 ? 4 : 3)
    k_join_rows(const float *__restrict__ X, int64_t n, int d, int S, const int32_t *__restrict__ newS,
                const int32_t *__restrict__ oldS, const int8_t *__restrict__ nf,
                const int8_t *__restrict__ of, int32_t *__restrict__ nrev, int32_t *__restrict__ orev,
                const float *__restrict__ worst, CandList cl, int cross_only) {
  extern __shared__ __align__(16) unsigned char smem_join[];
  const int lane = lane_id(), w = threadIdx.x >> 5;
  constexpr size_t kWarpBytes = (size_t)64 * kQ * 16 + 64 * 4;
  float4 *Xs = reinterpret_cast<float4 *>(smem_join + w * kWarpBytes);  // new rows, then old ones
  int32_t *ids = reinterpret_cast<int32_t *>(smem_join + w * kWarpBytes + (size_t)64 * kQ * 16);
  const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  unsigned long long w_rows = 0, w_cands = 0, w_pairs = 0;
  ListCursor cur;
  const int64_t stride = (int64_t)gridDim.x * kJoinWarps;
  SlotLists lists;
  int64_t row = (int64_t)blockIdx.x * kJoinWarps + w;
  lists.load(row, n, S, newS, oldS, nf, of, nrev, orev);
  for (; row < n; row += stride) {
    int nn, no;
    {
      const SlotLists mine = lists;
      lists.load(row + stride, n, S, newS, oldS, nf, of, nrev, orev);
      __syncwarp();
      if (lane == 0) { nrev[row] = 0; orev[row] = 0; }
      mine.compact(S, ids, nn, no);
    }
    if (nn == 0 || nn + no < 2 || (cross_only && no == 0)) continue;
    w_rows += nn + no;
    w_pairs += (cross_only ? 0 : nn * (nn - 1) / 2) + nn * no;  // the reference's pairs
    const int T = nn + no;
    if (vec) {
      for (int it = lane; it < T * kQ; it += 32) {
        const int r = it / kQ, q = it - r * kQ;
        const float *src = X + (int64_t)ids[r < nn ? r : 32 + r - nn] * d + 4 * q;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Xs + it);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    } else {
      for (int it = lane; it < T * kQ; it += 32) {
        const int r = it / kQ, c = 4 * (it - r * kQ);
        const float *src = X + (int64_t)ids[r < nn ? r : 32 + r - nn] * d;
        float4 v;  // zero padded: fmaf(0, 0, s) = s
        v.x = c < d ? __ldg(src + c) : 0.0f;
        v.y = c + 1 < d ? __ldg(src + c + 1) : 0.0f;
        v.z = c + 2 < d ? __ldg(src + c + 2) : 0.0f;
        v.w = c + 3 < d ? __ldg(src + c + 3) : 0.0f;
        Xs[it] = v;
      }
    }
    __syncwarp();
    // lane -> new row a, and the part g of the staged rows that it takes
    const int lgp = nn <= 8 ? 3 : nn <= 16 ? 4 : 5;
    const int P = 1 << lgp, h = 32 >> lgp, a = lane & (P - 1), g = lane >> lgp;
    float4 own[kQ];
#pragma unroll
    for (int q = 0; q < kQ; q++) own[q] = Xs[(a < nn ? a : 0) * kQ + q];
    // running minima: distance bits and the slot; equal distances are settled
    // below by the ids, in a second walk that compares both
    uint32_t m1 = 0xffffffffu, m2 = 0xffffffffu, m3 = 0xffffffffu;
    int i1 = 0, i2 = 0;
    bool tie = false;
    const bool isrow = a < nn;
    if (!cross_only) {
#pragma unroll 4
      for (int c = g; c < nn; c += h) {
        uint32_t v = __float_as_uint(row_dist<kQ>(Xs + c * kQ, own));
        if (c == a) v = 0xffffffffu;
        tie = tie || (v == m1 && c != a);  // the own column is not one
        if (v < m1) { m1 = v; i1 = c; }
      }
    }
    uint32_t at3 = 0;  // the new rows at the held old row's least distance
    if (h == 1) {
#pragma unroll 4
      for (int c = 0; c < no; c++) {
        uint32_t v = __float_as_uint(row_dist<kQ>(Xs + (nn + c) * kQ, own));
        if (!isrow) v = 0xffffffffu;
        tie = tie || v == m2;
        if (v < m2) { m2 = v; i2 = c; }
        const uint32_t least = __reduce_min_sync(0xffffffffu, v);
        const uint32_t at = __ballot_sync(0xffffffffu, v == least);
        if (lane == c) { m3 = least; at3 = at; }
      }
    } else {
      const uint32_t part = ((1u << P) - 1u) << (g << lgp);
      for (int c0 = 0; c0 < no; c0 += h) {  // every part the same number of steps
        const int c = c0 + g;
        uint32_t v = 0xffffffffu;
        if (c < no && isrow) v = __float_as_uint(row_dist<kQ>(Xs + (nn + c) * kQ, own));
        tie = tie || v == m2;
        if (v < m2) { m2 = v; i2 = c; }
        uint32_t least = v;
        for (int o = P >> 1; o; o >>= 1) least = min(least, __shfl_xor_sync(0xffffffffu, least, o));
        const uint32_t at = __ballot_sync(0xffffffffu, v == least) & part;
        if (a == c0 >> (5 - lgp)) { m3 = least; at3 = at; }  // lane c / h of the part keeps it
      }
    }
    tie = tie && isrow;
    const int i3 = (__ffs(at3) - 1) & (P - 1);
    tie = tie || ((at3 & (at3 - 1)) != 0 && m3 != 0xffffffffu);
    for (int o = P; o < 32; o <<= 1) {  // the parts of one new row
      const uint32_t o1 = __shfl_xor_sync(0xffffffffu, m1, o), o2 = __shfl_xor_sync(0xffffffffu, m2, o);
      const int p1 = __shfl_xor_sync(0xffffffffu, i1, o), p2 = __shfl_xor_sync(0xffffffffu, i2, o);
      tie = tie || (isrow && ((o1 == m1 && m1 != 0xffffffffu) || (o2 == m2 && m2 != 0xffffffffu)));
      if (o1 < m1) { m1 = o1; i1 = p1; }
      if (o2 < m2) { m2 = o2; i2 = p2; }
    }
    int32_t id1 = ids[i1], id2 = ids[32 + (i2 & 31)], id3 = ids[i3];
    const int c3 = (a << (5 - lgp)) + g;  // the held old row
    if (__any_sync(0xffffffffu, tie)) {
      // the least id at each least distance
      uint32_t b1 = 0xffffffffu, b2 = 0xffffffffu, b3 = 0xffffffffu;
      if (!cross_only)
        for (int c = 0; c < nn; c++) {
          const uint32_t v = __float_as_uint(row_dist<kQ>(Xs + c * kQ, own));
          if (c != a && v == m1) b1 = min(b1, (uint32_t)ids[c]);
        }
      for (int c = 0; c < no; c++) {
        const uint32_t v = __float_as_uint(row_dist<kQ>(Xs + (nn + c) * kQ, own));
        if (v == m2) b2 = min(b2, (uint32_t)ids[32 + c]);
        // lane l of the first part speaks for new row l
        const int holder = ((c & (h - 1)) << lgp) + (c >> (5 - lgp));
        const uint32_t least = __shfl_sync(0xffffffffu, m3, holder);
        const uint32_t id = __reduce_min_sync(0xffffffffu, isrow && v == least ? (uint32_t)ids[a] : 0xffffffffu);
        if (lane == holder) b3 = id;
      }
      id1 = (int32_t)b1;
      id2 = (int32_t)b2;
      id3 = (int32_t)b3;
    }
    const bool first = g == 0 && isrow, holds = c3 < no;
    const int32_t x = first ? ids[a] : 0, x3 = holds ? ids[32 + c3] : 0;
    const float wx = first ? worst[x] : 0.0f, wx3 = holds ? worst[x3] : 0.0f;
    const bool av[3] = {first && m1 != 0xffffffffu && __uint_as_float(m1) < wx,
                        first && m2 != 0xffffffffu && __uint_as_float(m2) < wx,
                        holds && m3 != 0xffffffffu && __uint_as_float(m3) < wx3};
    const int32_t at[3] = {x, x, x3};
    const uint64_t ak[3] = {pack(__uint_as_float(m1), id1), pack(__uint_as_float(m2), id2),
                            pack(__uint_as_float(m3), id3)};
    w_cands += append_candidates(cl, cur, av, at, ak);
    __syncwarp();
  }
  list_fill(cl, cur.pos, cur.end);
#pragma unroll
  for (int o = 16; o; o >>= 1) w_cands += __shfl_xor_sync(0xffffffffu, w_cands, o);
  if (lane == 0) {
    if (w_rows) atomicAdd(&cl.counters[1], w_rows);
    if (w_cands) atomicAdd(&cl.counters[2], w_cands);
    if (w_pairs) atomicAdd(&cl.counters[4], w_pairs);
  }
}

// ---------------------------------------------------------------------------
// BF16 tensor-core form of the local join.
//
// Candidate distances come from ||x||^2 + ||y||^2 - 2 x.y with x, y rounded to
// BF16 (norms of the rounded rows, FP32), the dot products on the tensor cores
// with FP32 accumulation (mma.sync m16n8k16, operands staged with cp.async
// and ldmatrix).  One pair always gets one value, whichever row joins it.
// After the last iteration every kept neighbour is re-ranked with the exact
// FP32 difference sum (k_rerank), so the graph handed on carries the
// reference's distances.
// ---------------------------------------------------------------------------
struct JoinSmemBf16 {
  // per warp: best[96] u64 | ids[64] | norms[64] | rows [64][dpad + 8] bf16
  __host__ __device__ static size_t bytes(int dpad) {
    return 96 * 8 + 64 * 4 + 64 * 4 + (size_t)64 * (dpad + 8) * 2;
  }
};

// Column sums of X (FP64, one thread per column, rows split over blocks):
// the BF16 copy is taken of the centred rows.
__global__ void k_col_sums(const float *__restrict__ X, int64_t n, int d, double *__restrict__ sums) {
  for (int j = threadIdx.x; j < d; j += blockDim.x) {
    double s = 0.0;
#pragma unroll 8
    for (int64_t row = blockIdx.x; row < n; row += gridDim.x) s += (double)X[row * d + j];
    atomicAdd(&sums[j], s);
  }
}

__global__ void k_col_mean(const double *__restrict__ sums, int d, int64_t n, float *__restrict__ mean) {
  for (int j = threadIdx.x; j < d; j += blockDim.x) mean[j] = (float)(sums[j] / (double)n);
}

// Largest |x - mean| over X (float bits: non-negative floats order as
// unsigned integers), for the FP16 form's power-of-two scale.
__global__ void k_abs_max(const float *__restrict__ X, int64_t n, int d,
                          const float *__restrict__ mean, uint32_t *__restrict__ out) {
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * d;
       i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, __float_as_uint(fabsf(__fsub_rn(X[i], mean[i % d]))));
#pragma unroll
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane_id() == 0 && m) atomicMax(out, m);
}

// 16-bit operand formats of the tensor-core forms.
struct Bf16Op {
  using T = __nv_bfloat16;
  static __device__ __forceinline__ T from(float x) { return __float2bfloat16_rn(x); }
  static __device__ __forceinline__ float to(T x) { return __bfloat162float(x); }
};
struct Fp16Op {
  using T = __half;
  static __device__ __forceinline__ T from(float x) { return __float2half_rn(x); }
  static __device__ __forceinline__ float to(T x) { return __half2float(x); }
};

// 16-bit copy of (X - mean) / scale (mean may be null: no centring; scale a
// power of two, 1 for BF16), zero padded to dpad columns, and the FP32
// squared norm of every rounded row taken back to the original scale.
// Distances do not change under a common shift, and centring keeps the
// coordinates small, which is where the rounding is finest.
template <typename Op>
__global__ void k_half_prepare(const float *__restrict__ X, int64_t n, int d, int dpad,
                               const float *__restrict__ mean, float inv_scale, float scale,
                               typename Op::T *__restrict__ Xh, float *__restrict__ nrm) {
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    float part = 0.0f;
    for (int j = lane; j < dpad; j += 32) {
      const float x = j < d ? __fsub_rn(X[row * d + j], mean ? mean[j] : 0.0f) : 0.0f;
      const typename Op::T h = Op::from(__fmul_rn(x, inv_scale));
      Xh[row * dpad + j] = h;
      const float v = __fmul_rn(Op::to(h), scale);
      part = __fmaf_rn(v, v, part);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, o));
    if (lane == 0) nrm[row] = part;
  }
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::);
}
__device__ __forceinline__ void ldsm_x4(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3,
                                        const void *smem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(s));
}
template <bool kFp16>
__device__ __forceinline__ void mma_16(float *c, const uint32_t *a, uint32_t b0, uint32_t b1) {
  if (kFp16)
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// kFp16: FP16 operands (scaled rows; dscale = -2 scale^2), else BF16
// (dscale = -2).  Xb holds the 16-bit rows.
template <bool kFp16>
__global__ void __launch_bounds__(128) k_join_bf16(const uint16_t *__restrict__ Xb,
                                                   const float *__restrict__ nrm, int64_t n,
                                                   int dpad, int S, float dscale,
                                                   const int32_t *__restrict__ newS,
                                                   const int32_t *__restrict__ oldS,
                                                   const int8_t *__restrict__ nf,
                                                   const int8_t *__restrict__ of,
                                                   int32_t *__restrict__ nrev,
                                                   int32_t *__restrict__ orev,
                                                   const float *__restrict__ worst, CandList cl) {
  extern __shared__ __align__(16) unsigned char smem_bf[];
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  unsigned char *base = smem_bf + (threadIdx.x >> 5) * JoinSmemBf16::bytes(dpad);
  unsigned long long *best = reinterpret_cast<unsigned long long *>(base);
  unsigned long long *best1 = best, *best2 = best + 32, *best3 = best + 64;
  int32_t *ids = reinterpret_cast<int32_t *>(base + 96 * 8);
  float *nr = reinterpret_cast<float *>(base + 96 * 8 + 256);
  uint16_t *Bs = reinterpret_cast<uint16_t *>(base + 96 * 8 + 512);
  const int ld = dpad + 8;  // row stride in elements (16-byte aligned, ldmatrix conflict free)
  const int chunks = dpad >> 3;  // 16-byte chunks per row
  unsigned long long w_rows = 0, w_cands = 0;
  ListCursor cur;
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    SampleLists lists;
    lists.load(row, n, S, newS, oldS, nf, of, nrev, orev);
    __syncwarp();
    if (lane == 0) { nrev[row] = 0; orev[row] = 0; }
    int nn, no;
    lists.compact(S, ids, nn, no);
    best1[lane] = ~0ull;
    best2[lane] = ~0ull;
    best3[lane] = ~0ull;
    __syncwarp();
    if (nn == 0 || nn + no < 2) continue;
    w_rows += nn + no;
    // stage rows: new at slots 0..nn-1, old at 32..32+no-1 (cp.async, 16 B)
    const int T = nn + no;
    for (int idx = lane; idx < T * chunks; idx += 32) {
      int r = idx / chunks, c = idx - r * chunks;
      int slot = r < nn ? r : 32 + (r - nn);
      cp_async16(Bs + slot * ld + c * 8, Xb + (int64_t)ids[slot] * dpad + c * 8);
    }
    if (lane < nn) nr[lane] = nrm[ids[lane]];
    if (lane < no) nr[32 + lane] = nrm[ids[32 + lane]];
    cp_async_wait_all();
    __syncwarp();
    // G = B_new (32 x dpad) * B_all (64 x dpad)^T
    float acc[2][8][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][j][e] = 0.0f;
    const int mts = nn > 16 ? 2 : 1;
    const bool any_old = no > 0;
    for (int kt = 0; kt < dpad; kt += 16) {
      uint32_t a[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; mt++)
        if (mt < mts)
          ldsm_x4(a[mt][0], a[mt][1], a[mt][2], a[mt][3],
                  Bs + (16 * mt + (lane & 15)) * ld + kt + ((lane >> 4) << 3));
#pragma unroll
      for (int pr = 0; pr < 4; pr++) {
        if (pr >= 2 && !any_old) continue;
        uint32_t b0, b1, b2, b3;
        const int prow = 16 * pr + ((lane >> 4) << 3) + (lane & 7);
        ldsm_x4(b0, b1, b2, b3, Bs + prow * ld + kt + (((lane >> 3) & 1) << 3));
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
          if (mt >= mts) continue;
          mma_16<kFp16>(acc[mt][2 * pr], a[mt], b0, b1);
          mma_16<kFp16>(acc[mt][2 * pr + 1], a[mt], b2, b3);
        }
      }
    }
    // epilogue: distances, row minima (best1 / best2) and old-column minima (best3)
    uint64_t cmin[4][2];  // old n-tiles 4..7, two columns each
#pragma unroll
    for (int q = 0; q < 4; q++) cmin[q][0] = cmin[q][1] = ~0ull;
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int a = 16 * mt + (lane >> 2) + 8 * h;
        const bool arow = mt < mts && a < nn;
        const float na = arow ? nr[a] : 0.0f;
        uint64_t rn = ~0ull, ro = ~0ull;
#pragma unroll
        for (int nt = 0; nt < 8; nt++) {
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int c = 8 * nt + 2 * (lane & 3) + e;
            const bool oldc = c >= 32;
            const bool ok = arow && (oldc ? (c - 32 < no) : (c < nn && c != a));
            if (!ok) continue;
            float dd = __fmaf_rn(dscale, acc[mt][nt][2 * h + e], __fadd_rn(na, nr[c]));
            dd = dd > 0.0f ? dd : 0.0f;
            const uint64_t kr = pack(dd, ids[c]);
            if (oldc) {
              ro = kr < ro ? kr : ro;
              const uint64_t kc = pack(dd, ids[a]);
              uint64_t &m = cmin[nt - 4][e];
              m = kc < m ? kc : m;
            } else {
              rn = kr < rn ? kr : rn;
            }
          }
        }
        // the four lanes of a row
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
          uint64_t x = __shfl_xor_sync(0xffffffffu, rn, o);
          rn = x < rn ? x : rn;
          x = __shfl_xor_sync(0xffffffffu, ro, o);
          ro = x < ro ? x : ro;
        }
        if (arow && (lane & 3) == 0) {
          best1[a] = rn;
          best2[a] = ro;
        }
      }
    }
    // the eight row-lanes of a column
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        uint64_t m = cmin[q][e];
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) {
          uint64_t x = __shfl_xor_sync(0xffffffffu, m, o);
          m = x < m ? x : m;
        }
        const int c = 8 * q + 2 * (lane & 3) + e;  // old column index
        if (lane < 4 && c < no) best3[c] = m;
      }
    __syncwarp();
    const int32_t x = lane < nn ? ids[lane] : 0, x3 = lane < no ? ids[32 + lane] : 0;
    const uint64_t b1 = lane < nn ? best1[lane] : ~0ull, b2 = lane < nn ? best2[lane] : ~0ull;
    const uint64_t b3 = lane < no ? best3[lane] : ~0ull;
    const float wx = lane < nn ? worst[x] : 0.0f, wx3 = lane < no ? worst[x3] : 0.0f;
    const bool v1 = b1 != ~0ull && pk_dist(b1) < wx, v2 = b2 != ~0ull && pk_dist(b2) < wx;
    const bool v3 = b3 != ~0ull && pk_dist(b3) < wx3;
    const bool av[3] = {v1, v2, v3};
    const int32_t at[3] = {x, x, x3};
    const uint64_t ak[3] = {b1, b2, b3};
    w_cands += append_candidates(cl, cur, av, at, ak);
    __syncwarp();
  }
  list_fill(cl, cur.pos, cur.end);
#pragma unroll
  for (int o = 16; o; o >>= 1) w_cands += __shfl_xor_sync(0xffffffffu, w_cands, o);
  if (lane == 0) {
    if (w_rows) atomicAdd(&cl.counters[1], w_rows);
    if (w_cands) atomicAdd(&cl.counters[2], w_cands);
  }
}

// FP32 re-rank of every kept neighbour (one warp per row): the reference's
// difference sum for each (row, neighbour) pair, rows re-sorted by (distance,
// id); old/new flags travel with their ids.
template <int kV>
__global__ void __launch_bounds__(32 * kStageWarps, 8) k_rerank(const float *__restrict__ X, int64_t n, int d, int k,
                         hdb_nnd_element *__restrict__ G) {
  extern __shared__ float smem_stage[];
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  float *sm = smem_stage + (threadIdx.x >> 5) * 33 * stage_pitch(d, kV) * kV;
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    int32_t lab = 0;
    if (lane < k) lab = G[row * k + lane].label_;
    const int32_t id = decode(lab);
    const float ds = diffsum_staged<kV>(X, d, row, id, k, sm);
    uint64_t key = lane < k ? pack(ds, id) : ~0ull;
    int32_t slab = lab;  // the entry (with its old/new flag) moves with its key
    warp_sort32_with(key, slab);
    if (lane < k) {
      hdb_nnd_element e;
      e.distance_ = pk_dist(key);
      e.label_ = slab;
      G[row * k + lane] = e;
    }
  }
}

__global__ void k_split(const hdb_nnd_element *__restrict__ G, int64_t total, int32_t *__restrict__ ids,
                        float *__restrict__ dist) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    hdb_nnd_element e = G[i];
    if (ids) ids[i] = decode(e.label_);
    if (dist) dist[i] = e.distance_;
  }
}

__device__ __forceinline__ float euclid_ref(const float *__restrict__ a, const float *__restrict__ b,
                                           int d) {
  float soma = 0.0f;
  for (int i = 0; i < d; i++) {
    float diff = __fsub_rn(a[i], b[i]);
    double sq = __dmul_rn((double)diff, (double)diff);
    soma = __double2float_rn(__dadd_rn((double)soma, sq));
  }
  return __fsqrt_rn(soma);
}

__global__ void k_fix_distances(const float *__restrict__ X, int64_t n, int d,
                                const int32_t *__restrict__ ids, int k, float *__restrict__ dist,
                                volatile uint32_t *outside) {
  const int64_t total = n * k;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t row = i / k;
    const int32_t v = ids[i];
    if (v < 0 || v >= n) {
      *outside = 1;
      continue;
    }
    dist[i] = euclid_ref(X + row * d, X + (int64_t)v * d, d);
  }
}

// ---- locality order ---------------------------------------------------------
// The local join gathers the rows of every row's samples, i.e. of its current
// neighbours.  With ids in arbitrary order those rows lie anywhere in X, and
// the ~2,000 consecutive rows the join works on at any moment fetch them all
// from HBM.  After the initial graph the points are renumbered so that near
// points get near ids: by instance, then by the Morton code of three
// projections on fixed +-1 vectors (10 bits each over the projection's range).
// The rows in flight then gather from a few MB of X, which L2 holds.  The final
// graph is mapped back to the original ids and every row re-sorted by
// (distance, id), so the order is the caller's.
constexpr int kLocProj = 3;

__device__ __forceinline__ float loc_sign(int p, int j) {
  return (xorshift64star(((uint64_t)(p + 1) << 32) | (uint32_t)j) >> 63) ? -1.0f : 1.0f;
}

// One warp per row: the three projections; per block the range of each.
__global__ void k_loc_project(const float *__restrict__ X, int64_t n, int d,
                              float *__restrict__ proj, uint32_t *__restrict__ range) {
  __shared__ uint32_t blk[2 * kLocProj];
  if (threadIdx.x < 2 * kLocProj) blk[threadIdx.x] = (threadIdx.x & 1) ? 0u : 0xffffffffu;
  __syncthreads();
  const int lane = lane_id(), wpb = blockDim.x >> 5;
  uint32_t lo[kLocProj], hi[kLocProj];
#pragma unroll
  for (int p = 0; p < kLocProj; p++) { lo[p] = 0xffffffffu; hi[p] = 0u; }
  for (int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); row < n;
       row += (int64_t)gridDim.x * wpb) {
    float acc[kLocProj] = {0.0f, 0.0f, 0.0f};
    for (int j = lane; j < d; j += 32) {
      const float x = X[row * d + j];
#pragma unroll
      for (int p = 0; p < kLocProj; p++) acc[p] += loc_sign(p, j) * x;
    }
#pragma unroll
    for (int p = 0; p < kLocProj; p++) {
#pragma unroll
      for (int o = 16; o; o >>= 1) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], o);
      const uint32_t key = float_key(acc[p]);
      lo[p] = min(lo[p], key);
      hi[p] = max(hi[p], key);
      if (lane == p) proj[row * kLocProj + p] = acc[p];
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int p = 0; p < kLocProj; p++) {
      atomicMin(&blk[2 * p], lo[p]);
      atomicMax(&blk[2 * p + 1], hi[p]);
    }
  }
  __syncthreads();
  if (threadIdx.x < kLocProj) {
    atomicMin(&range[2 * threadIdx.x], blk[2 * threadIdx.x]);
    atomicMax(&range[2 * threadIdx.x + 1], blk[2 * threadIdx.x + 1]);
  }
}

__device__ __forceinline__ uint32_t spread3(uint32_t x) {  // 10 bits -> every third bit
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__global__ void k_loc_keys(const float *__restrict__ proj, int64_t n, Segments seg,
                           const uint32_t *__restrict__ range, uint64_t *__restrict__ keys,
                           uint32_t *__restrict__ vals) {
  float lo[kLocProj], scale[kLocProj];
#pragma unroll
  for (int p = 0; p < kLocProj; p++) {
    lo[p] = key_float(range[2 * p]);
    const float w = key_float(range[2 * p + 1]) - lo[p];
    scale[p] = w > 0.0f ? 1024.0f / w : 0.0f;
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t m = 0;
#pragma unroll
    for (int p = 0; p < kLocProj; p++) {
      const float q = (proj[i * kLocProj + p] - lo[p]) * scale[p];
      const uint32_t c = q <= 0.0f ? 0u : (q >= 1023.0f ? 1023u : (uint32_t)q);
      m |= spread3(c) << p;
    }
    const uint64_t inst = seg.count > 0 ? (uint64_t)seg.of_point(i) : 0;
    keys[i] = (inst << 32) | m;
    vals[i] = (uint32_t)i;
  }
}

__global__ void k_loc_inverse(const uint32_t *__restrict__ order, int64_t n, int32_t *__restrict__ inv) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    inv[order[i]] = (int32_t)i;
}

__global__ void k_loc_rows(const float *__restrict__ X, const uint32_t *__restrict__ order, int64_t n,
                           int d, float *__restrict__ Xp) {
  const int lane = lane_id(), wpb = blockDim.x >> 5;
  for (int64_t r = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); r < n;
       r += (int64_t)gridDim.x * wpb) {
    const int64_t o = order[r];
    for (int j = lane; j < d; j += 32) Xp[r * d + j] = X[o * d + j];
  }
}

// A row with every id mapped through idmap, re-sorted by (distance, mapped
// id); each entry keeps its old/new flag.  One warp per row.
__device__ __forceinline__ void remap_row(int k, int32_t in_lab, float in_dist,
                                          const int32_t *__restrict__ idmap, int32_t &out_lab,
                                          float &out_dist) {
  const int lane = lane_id();
  const bool have = lane < k;
  const int32_t id = have ? idmap[decode(in_lab)] : 0;
  uint64_t key = have ? pack(in_dist, id) : ~0ull;
  int32_t flag = have && in_lab < 0;  // moves with its key (ids are distinct within a row)
  warp_sort32_with(key, flag);
  const int32_t mine = pk_id(key);
  out_dist = pk_dist(key);
  out_lab = flag ? -mine - 1 : mine;
}

__global__ void k_loc_restore(const hdb_nnd_element *__restrict__ Gp, const uint32_t *__restrict__ order,
                              int64_t n, int k, hdb_nnd_element *__restrict__ G) {
  const int lane = lane_id(), wpb = blockDim.x >> 5;
  for (int64_t r = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); r < n;
       r += (int64_t)gridDim.x * wpb) {
    hdb_nnd_element e = lane < k ? Gp[r * k + lane] : hdb_nnd_element{0.0f, 0};
    int32_t ol;
    float od;
    remap_row(k, e.label_, e.distance_, reinterpret_cast<const int32_t *>(order), ol, od);
    if (lane < k) G[(int64_t)order[r] * k + lane] = hdb_nnd_element{od, ol};
  }
}

int bits_for_rows(int64_t n) {
  int b = 1;
  while (b < 40 && (int64_t(1) << b) < n) b++;
  return b;
}

}  // namespace

namespace {

// Launches one of the kernels that stage rows for difference sums over the rows
// of X: shared memory for the rows' width, four turns of resident blocks.
template <class Kernel, class... Args>
void launch_staged(Context *ctx, Kernel by4, Kernel by2, Kernel by1, const float *X, int64_t n, int d,
                   Args... args) {
  const int kV = stage_floats(X, d);
  const Kernel fn = kV == 4 ? by4 : kV == 2 ? by2 : by1;
  const size_t smem = kStageWarps * stage_bytes(d, kV);
  const int resident = (int)std::min<size_t>(8, (size_t(220) << 10) / (smem + 1024));
  fn<<<grid_for(ctx, n, kStageWarps, 4 * resident), 32 * kStageWarps, smem, ctx->stream>>>(X, n, d, args...);
  ctx->launches++;
}

// The candidate list of joins whose targets are n rows, with the second buffer of its
// grouping.  chunk: what a warp takes of its slots at a time.
struct Candidates {
  int64_t n;
  int shift;
  int64_t buckets;
  Buf<uint64_t> list_key, list_key2;
  Buf<unsigned long long> best, counters;
  Buf<uint32_t> list_tgt, list_tgt2, bstart, rstart;
  CandList cl;
  RowList rl;

  Candidates(Context *ctx, int64_t n, int64_t slots, uint32_t chunk)
      : n(n), shift(bucket_shift(n)), buckets(ceil_div(n, int64_t(1) << shift)) {
    best = Buf<unsigned long long>(ctx, n);
    counters = Buf<unsigned long long>(ctx, 5);
    list_tgt = Buf<uint32_t>(ctx, slots);
    list_key = Buf<uint64_t>(ctx, slots);
    list_tgt2 = Buf<uint32_t>(ctx, slots);
    list_key2 = Buf<uint64_t>(ctx, slots);
    bstart = Buf<uint32_t>(ctx, std::max<int64_t>(513, buckets + 1));
    rstart = Buf<uint32_t>(ctx, n + 1);
    cl = CandList{best, list_tgt, list_key, counters, slots, chunk, (uint32_t)(buckets << shift)};
    HDB_CUDA(cudaMemsetAsync(best, 0xff, n * 8, ctx->stream));
    HDB_CUDA(cudaMemsetAsync(counters, 0, 5 * sizeof(unsigned long long), ctx->stream));
  }
  // groups a join's candidates by row
  void group(Context *ctx) {
    const int bits = bits_for_rows((int64_t)cl.none + 1);
    const bool second = radix_group_u32_u64(ctx, list_tgt, list_key, list_tgt2, list_key2, cl.cap,
                                            counters.get() + 3, shift, bits, bstart);
    uint32_t *tgt = second ? list_tgt2 : list_tgt;
    uint64_t *key = second ? list_key2 : list_key, *out = second ? list_key : list_key2;
    if (bits - shift > 9) {  // several passes: the digit starts of the last one are not the buckets'
      k_bucket_bounds<<<grid_for(ctx, buckets + 1, 8), 256, 0, ctx->stream>>>(
          tgt, counters.get() + 3, cl.cap, shift, buckets, bstart);
      ctx->launches++;
      HDB_CHECK_LAUNCH();
    }
    k_group_rows<<<(unsigned)buckets, kGroupThreads, 0, ctx->stream>>>(n, shift, tgt, key, bstart, rstart,
                                                                    out);
    ctx->launches++;
    HDB_CHECK_LAUNCH();
    rl = RowList{rstart, out, best};
  }
};

// Device state of one NN-Descent run over n rows: the graph lists, the
// samples of an iteration and the join's candidates.  warps: the most warps that
// append to their list.
struct NndState {
  int64_t n;
  int k, S;
  Buf<int32_t> gid, newS, oldS, nrev, orev;
  Buf<float> gdist, worst;
  Buf<int8_t> nf, of;
  Candidates c;

  NndState(Context *ctx, int64_t n, int k, int S, int64_t warps)
      : n(n), k(k), S(S), c(ctx, n, list_slots(n, warps), list_chunk(n, warps)) {
    cudaStream_t st = ctx->stream;
    gid = Buf<int32_t>(ctx, n * k);
    gdist = Buf<float>(ctx, n * k);
    worst = Buf<float>(ctx, n);
    newS = Buf<int32_t>(ctx, n * 2 * S);
    oldS = Buf<int32_t>(ctx, n * 2 * S);
    nrev = Buf<int32_t>(ctx, n);
    orev = Buf<int32_t>(ctx, n);
    nf = Buf<int8_t>(ctx, n);
    of = Buf<int8_t>(ctx, n);
    HDB_CUDA(cudaMemsetAsync(nrev, 0, n * 4, st));
    HDB_CUDA(cudaMemsetAsync(orev, 0, n * 4, st));
  }
  SampleOut samples() const { return SampleOut{newS, oldS, nf, of, nrev, orev}; }

  // the samples of an iteration; after the first, of the rows merged with the
  // candidates of the join before
  void sample(Context *ctx, bool merge, int64_t split) {
    HDB_CUDA(cudaFuncSetAttribute(k_sample, cudaFuncAttributePreferredSharedMemoryCarveout, kSampleShare));
    k_sample<<<grid_for(ctx, n, 8, 16), 256, 0, ctx->stream>>>(
        n, k, S, merge, gid, gdist, worst, c.rl, c.counters, samples(), split);
    ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
  void finalize(Context *ctx, hdb_nnd_element *out) {
    k_finalize<<<grid_for(ctx, n, 8, 16), 256, 0, ctx->stream>>>(n, k, gid, gdist, c.rl, out);
    ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
};

template <int kQ>
void join_rows(Context *ctx, const float *X, int64_t n, int d, int S, const SampleOut &s, const float *worst,
               const CandList &cl, int cross_only) {
  const size_t smem = (size_t)kJoinWarps * (64 * kQ * 16 + 64 * 4);
  HDB_CUDA(cudaFuncSetAttribute(k_join_rows<kQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = grid_for(ctx, n, kJoinWarps, kQ <= 4 ? 4 : 3);
  k_join_rows<kQ><<<grid, 32 * kJoinWarps, smem, ctx->stream>>>(
      X, n, d, S, s.newS, s.oldS, s.nf, s.of, s.nrev, s.orev, worst, cl, cross_only);
  ctx->launches++;
}

// The FP32 join's form: 1 by rows, up to kRowJoinMaxDim dimensions and unless the
// context forces tiles, else 2, in tiles.
int fp32_join_form(const Context *ctx, int d) { return d <= kRowJoinMaxDim && ctx->join_tiles != 2 ? 1 : 2; }

// One FP32 local join over n rows' samples s.
void fp32_join(Context *ctx, const float *X, int64_t n, int d, int S, const SampleOut &s, const float *worst,
               const CandList &cl, int cross_only) {
  if (fp32_join_form(ctx, d) == 1) {
    using Join = void (*)(Context *, const float *, int64_t, int, int, const SampleOut &, const float *,
                          const CandList &, int);
    static const Join by_pieces[7] = {join_rows<1>, join_rows<2>, join_rows<3>, join_rows<4>,
                                      join_rows<5>, join_rows<6>, join_rows<7>};
    by_pieces[(d + 3) / 4 - 1](ctx, X, n, d, S, s, worst, cl, cross_only);
    return;
  }
  // the blocks that fit on the GPU at once (a grid-stride loop over the rows):
  // each warp holds one chunk of list space, so their number bounds what the
  // list loses to unused chunk tails
  const int grid = grid_for(ctx, n, kJoinWarps, 2);
  const size_t smem = kJoinWarps * JoinSmem::kBytes;
  HDB_CUDA(cudaFuncSetAttribute(k_join, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_join<<<grid, 32 * kJoinWarps, smem, ctx->stream>>>(X, n, d, S, s.newS, s.oldS, s.nf, s.of, s.nrev,
                                                       s.orev, worst, cl, cross_only);
  ctx->launches++;
}

// Warps of the joins that append to the list.
int64_t fp32_join_warps(const Context *ctx, int64_t n) {
  return (int64_t)kJoinWarps * grid_for(ctx, n, kJoinWarps, 4);
}
int64_t tc_join_warps(const Context *ctx, int64_t n) {
  return 4 * std::min<int64_t>((n + 1) / 2, 2 * (int64_t)ctx->num_sms);
}

}  // namespace

int64_t nndescent_bytes(const Context *ctx, int64_t n, int32_t d, const hdb_knn_params &p) {
  const int64_t k = p.k, S = p.sample_num;
  const bool half = p.precision == HDB_PREC_BF16 || p.precision == HDB_PREC_FP16;
  const bool tc = half && tc_dpad(d) <= kTcMaxDpad;
  const int64_t dpad = tc ? tc_dpad(d) : (d + 15) & ~15;
  int64_t b = 4 * (int64_t)d;                    // X in locality order
  if (half) b += 2 * dpad + 4;                   // 16-bit rows + norms
  b += 8 * k + 4 + 16 * S + 30;                  // lists, worst, samples, counters
  b += 8 * k;                                    // graph in locality order
  // the wide 16-bit join's grid depends on what fits on an SM; at most 64 warps do
  const int64_t warps = tc     ? tc_join_warps(ctx, n)
                        : half ? std::min<int64_t>((n + 3) & ~int64_t(3), 64 * (int64_t)ctx->num_sms)
                               : fp32_join_warps(ctx, n);
  return b * n + list_bytes(list_slots(n, warps));
}

void nndescent(Context *ctx, const float *X, int64_t n, int32_t d, const hdb_knn_params &p,
               hdb_nnd_element *G, int64_t *dropped_out, JoinStats *js, const Segments &seg) {
  const int k = p.k, S = p.sample_num;
  HDB_REQUIRE(k >= 1 && k <= kMaxK, HDB_ERR_ARG, "NN-Descent: k must be in [1, 32]");
  HDB_REQUIRE(S >= 1 && 2 * S <= k, HDB_ERR_ARG,
              "NN-Descent: SAMPLE_NUM must satisfy 1 <= SAMPLE_NUM and 2*SAMPLE_NUM <= k");
  HDB_REQUIRE(n > k && n < (int64_t(1) << 31) - 1, HDB_ERR_ARG, "NN-Descent: need k < n < 2^31");
  HDB_REQUIRE(d >= 1 && d <= 4096, HDB_ERR_ARG, "NN-Descent: d must be in [1, 4096]");
  HDB_REQUIRE(p.iterations >= 0, HDB_ERR_ARG, "NN-Descent: negative iteration count");
  HDB_REQUIRE(p.precision == HDB_PREC_FP32 || p.precision == HDB_PREC_BF16 ||
                  p.precision == HDB_PREC_FP16,
              HDB_ERR_ARG, "NN-Descent: unknown precision");
  cudaStream_t st = ctx->stream;
  // 16-bit forms: BF16, or FP16 of the rows scaled by one power of two; the
  // tensor-core tile pipeline (tcgen05) up to 256 padded dimensions, the
  // mma.sync join beyond
  const bool fp16 = p.precision == HDB_PREC_FP16;
  const bool bf16 = p.precision == HDB_PREC_BF16 || fp16;
  const bool use_tc = bf16 && tc_dpad(d) <= kTcMaxDpad;
  const int dpad = use_tc ? tc_dpad(d) : (d + 15) & ~15;
  const int jw16 = 4;  // warps per block of the mma.sync join
  size_t smem_bf = 0;
  int grid_bf = 0;
  if (bf16 && !use_tc) {
    smem_bf = JoinSmemBf16::bytes(dpad) * jw16;
    HDB_REQUIRE(smem_bf <= 227 * 1024, HDB_ERR_ARG, "NN-Descent 16-bit form: d too large for the join tile");
    const auto fn = fp16 ? k_join_bf16<true> : k_join_bf16<false>;
    // the most that any call asks for: another thread's call may come between this and the launch
    HDB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    int resident = 0;  // a persistent grid, as of the other joins
    HDB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, fn, 32 * jw16, smem_bf));
    grid_bf = grid_for(ctx, n, jw16, std::max(1, resident));
  }
  NndState s(ctx, n, k, S,
             use_tc ? tc_join_warps(ctx, n) : bf16 ? (int64_t)grid_bf * jw16 : fp32_join_warps(ctx, n));
  int32_t *gid = s.gid, *newS = s.newS, *oldS = s.oldS, *nrev = s.nrev, *orev = s.orev;
  float *gdist = s.gdist, *worst = s.worst;
  int8_t *nf = s.nf, *of = s.of;
  const CandList &cl = s.c.cl;
  std::vector<cudaEvent_t> jev;
  if (js) {
    jev.resize(2 * (size_t)p.iterations);
    for (auto &e : jev) HDB_CUDA(cudaEventCreate(&e));
  }

  const int wpb = 8;
  const int grid_rows = grid_for(ctx, n, wpb, 16);
  // renumber the points in locality order (k_loc_project); X stays the
  // caller's, the iterations work on Xw and the renumbered lists, and the
  // initial graph is drawn straight into the new numbering
  Buf<uint32_t> order(ctx, n);
  Buf<float> Xp(ctx, (size_t)n * d);
  {
    Buf<float> proj(ctx, (size_t)n * kLocProj);
    Buf<uint32_t> range(ctx, 2 * kLocProj);
    const uint32_t range0[2 * kLocProj] = {0xffffffffu, 0u, 0xffffffffu, 0u, 0xffffffffu, 0u};
    HDB_CUDA(cudaMemcpyAsync(range, range0, sizeof(range0), cudaMemcpyHostToDevice, st));
    k_loc_project<<<grid_rows, 32 * wpb, 0, st>>>(X, n, d, proj, range); ctx->launches++;
    Buf<uint64_t> keys(ctx, n);
    k_loc_keys<<<grid_for(ctx, n, 256), 256, 0, st>>>(proj, n, seg, range, keys, order); ctx->launches++;
    HDB_CHECK_LAUNCH();
    int ibits = 0;
    while (seg.count > 0 && (int64_t(1) << ibits) < seg.count) ibits++;
    radix_sort_u64(ctx, keys, order, n, 0, 30 + (seg.count > 0 ? 2 + ibits : 0));
    Buf<int32_t> inv(ctx, n);
    k_loc_inverse<<<grid_for(ctx, n, 256), 256, 0, st>>>(order, n, inv); ctx->launches++;
    k_loc_rows<<<grid_rows, 32 * wpb, 0, st>>>(X, order, n, d, Xp); ctx->launches++;
    HDB_CHECK_LAUNCH();
    launch_staged(ctx, k_init<4>, k_init<2>, k_init<1>, Xp, n, d, k, seg, order.get(), inv.get(), gid, gdist,
                  worst);
    HDB_CHECK_LAUNCH();
  }
  const float *Xw = Xp;
  Buf<hdb_nnd_element> Gp(ctx, (size_t)n * k);
  Buf<uint16_t> Xb;
  Buf<float> nrm;
  float dscale = -2.0f;
  TcJoin tj;
  if (bf16) {
    Xb = Buf<uint16_t>(ctx, (size_t)n * dpad);
    nrm = Buf<float>(ctx, n);
    Buf<double> csum(ctx, d);
    Buf<float> cmean(ctx, d);
    HDB_CUDA(cudaMemsetAsync(csum, 0, d * sizeof(double), st));
    k_col_sums<<<16 * ctx->num_sms, 256, 0, st>>>(Xw, n, d, csum); ctx->launches++;
    k_col_mean<<<1, 256, 0, st>>>(csum, d, n, cmean); ctx->launches++;
    HDB_CHECK_LAUNCH();
    if (fp16) {
      // one power-of-two scale s with max |x - mean| / s in [2^14, 2^15): far
      // from the FP16 overflow and subnormal ranges, exact to apply
      Buf<uint32_t> amax(ctx, 1);
      HDB_CUDA(cudaMemsetAsync(amax, 0, sizeof(uint32_t), st));
      k_abs_max<<<grid_for(ctx, n * d, 256), 256, 0, st>>>(Xw, n, d, cmean, amax); ctx->launches++;
      HDB_CHECK_LAUNCH();
      HDB_CUDA(cudaMemcpyAsync(ctx->pinned, amax, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
      ctx->sync();
      float gmax;
      memcpy(&gmax, ctx->pinned, sizeof(float));
      int e = 0;
      if (gmax > 0.0f && std::isfinite(gmax)) std::frexp(gmax, &e);
      const float sc = std::ldexp(1.0f, e - 15);
      dscale = -2.0f * sc * sc;
      k_half_prepare<Fp16Op><<<grid_rows, 32 * wpb, 0, st>>>(
          Xw, n, d, dpad, cmean, 1.0f / sc, sc, reinterpret_cast<__half *>(Xb.get()), nrm);
    } else {
      k_half_prepare<Bf16Op><<<grid_rows, 32 * wpb, 0, st>>>(
          Xw, n, d, dpad, cmean, 1.0f, 1.0f, reinterpret_cast<__nv_bfloat16 *>(Xb.get()), nrm);
    }
    ctx->launches++;
    HDB_CHECK_LAUNCH();
    if (use_tc) tc_join_prepare(ctx, Xb, n, dpad, fp16, dscale, &tj);
  }
  if (js) js->config = bf16 ? 0 : fp32_join_form(ctx, d);
  for (int it = 0; it < p.iterations; it++) {
    s.sample(ctx, it > 0, 0);
    if (js) HDB_CUDA(cudaEventRecord(jev[2 * it], st));
    if (use_tc) {
      tc_join_launch(ctx, tj, S, nrm, newS, oldS, nf, of, nrev, orev, worst, cl);
    } else {
      if (fp16)
        k_join_bf16<true><<<grid_bf, 32 * jw16, smem_bf, st>>>(Xb, nrm, n, dpad, S, dscale, newS,
                                                               oldS, nf, of, nrev, orev, worst, cl);
      else if (bf16)
        k_join_bf16<false><<<grid_bf, 32 * jw16, smem_bf, st>>>(Xb, nrm, n, dpad, S, dscale, newS,
                                                                oldS, nf, of, nrev, orev, worst, cl);
      else
        fp32_join(ctx, Xw, n, d, S, s.samples(), worst, cl, 0);
      if (bf16) ctx->launches++;
    }
    if (js) HDB_CUDA(cudaEventRecord(jev[2 * it + 1], st));
    HDB_CHECK_LAUNCH();
    s.c.group(ctx);
  }
  if (p.iterations == 0) s.c.group(ctx);  // an empty list
  s.finalize(ctx, Gp);
  if (bf16) {
    launch_staged(ctx, k_rerank<4>, k_rerank<2>, k_rerank<1>, Xw, n, d, k, Gp.get());
    HDB_CHECK_LAUNCH();
  }
  k_loc_restore<<<grid_rows, 32 * wpb, 0, st>>>(Gp, order, n, k, G); ctx->launches++;
  HDB_CHECK_LAUNCH();
  HDB_CUDA(cudaMemcpyAsync(ctx->pinned, s.c.counters, 5 * sizeof(unsigned long long),
                           cudaMemcpyDeviceToHost, st));
  ctx->sync();
  if (use_tc)
    HDB_REQUIRE(!(ctx->take_dev_err() & DEVERR_TIMEOUT), HDB_ERR_TIMEOUT,
                "NN-Descent: a wait of the tensor-core join pipeline gave up");
  const int64_t *hs = static_cast<const int64_t *>(ctx->pinned);
  if (dropped_out) *dropped_out = hs[0];
  if (js) {
    js->rows_gathered = hs[1];
    js->candidates = hs[2];
    js->pairs = hs[4];
    js->launches = p.iterations;
    js->ms = 0.0;
    for (int it = 0; it < p.iterations; it++) {
      float ms = 0.0f;
      HDB_CUDA(cudaEventElapsedTime(&ms, jev[2 * it], jev[2 * it + 1]));
      js->ms += ms;
    }
    for (auto &e : jev) cudaEventDestroy(e);
  }
}

void knn_merge(Context *ctx, const float *X1, int64_t n1, const hdb_nnd_element *G1,
               const float *X2, int64_t n2, const hdb_nnd_element *G2, int32_t d,
               const hdb_knn_params &p, hdb_nnd_element *G, int64_t *dropped_out) {
  const int k = p.k, S = p.sample_num;
  HDB_REQUIRE(k >= 1 && k <= kMaxK, HDB_ERR_ARG, "KNNMerge: k must be in [1, 32]");
  HDB_REQUIRE(S >= 1 && 2 * S <= k, HDB_ERR_ARG,
              "KNNMerge: MERGE_SAMPLE_NUM must satisfy 1 <= SAMPLE_NUM and 2*SAMPLE_NUM <= k");
  HDB_REQUIRE(n1 > k && n2 > k, HDB_ERR_ARG, "KNNMerge: each point set needs more than k points");
  const int64_t n = n1 + n2;
  HDB_REQUIRE(n < (int64_t(1) << 31) - 1, HDB_ERR_ARG, "KNNMerge: need n1 + n2 < 2^31");
  HDB_REQUIRE(d >= 1 && d <= 4096, HDB_ERR_ARG, "KNNMerge: d must be in [1, 4096]");
  HDB_REQUIRE(p.iterations >= 0, HDB_ERR_ARG, "KNNMerge: negative iteration count");
  HDB_REQUIRE(p.precision == HDB_PREC_FP32, HDB_ERR_ARG,
              "KNNMerge: the merge join is the FP32 difference sum (precision must be FP32)");
  cudaStream_t st = ctx->stream;
  (void)ctx->take_dev_err();
  // MergeVectors (knnmerge.cu:358-399): the two sets back to back
  Buf<float> X(ctx, (size_t)n * d);
  HDB_CUDA(cudaMemcpyAsync(X.get(), X1, (size_t)n1 * d * sizeof(float), cudaMemcpyDeviceToDevice, st));
  HDB_CUDA(cudaMemcpyAsync(X.get() + (size_t)n1 * d, X2, (size_t)n2 * d * sizeof(float),
                           cudaMemcpyDeviceToDevice, st));
  NndState s(ctx, n, k, S, fp32_join_warps(ctx, n));

  launch_staged(ctx, k_merge_init<4>, k_merge_init<2>, k_merge_init<1>, X, n, d, k, n1, G1, G2, s.gid.get(), s.gdist.get(),
                s.worst.get(), ctx->dev_err);
  HDB_CHECK_LAUNCH();
  ctx->sync();
  const uint32_t e = ctx->take_dev_err();
  HDB_REQUIRE(!(e & DEVERR_ID_RANGE), HDB_ERR_ARG, "KNNMerge: a subgraph id lies outside its set");
  HDB_REQUIRE(!(e & DEVERR_SELF_ID), HDB_ERR_ARG, "KNNMerge: a subgraph row lists itself");
  HDB_REQUIRE(!(e & DEVERR_DUP_ID), HDB_ERR_ARG, "KNNMerge: a subgraph row repeats an id");

  // NNDescentForMerge (nndescent.cu:1999-2087): PrepareForUpdateForMerge +
  // UpdateGraphForMerge per iteration
  for (int it = 0; it < p.iterations; it++) {
    s.sample(ctx, it > 0, n1);
    fp32_join(ctx, X, n, d, S, s.samples(), s.worst, s.c.cl, 1);
    HDB_CHECK_LAUNCH();
    s.c.group(ctx);
  }
  if (p.iterations == 0) s.c.group(ctx);  // an empty list
  s.finalize(ctx, G);
  HDB_CUDA(cudaMemcpyAsync(ctx->pinned, s.c.counters, sizeof(unsigned long long),
                           cudaMemcpyDeviceToHost, st));
  ctx->sync();
  if (dropped_out) *dropped_out = *static_cast<const int64_t *>(ctx->pinned);
}

void fp32_join_candidates(Context *ctx, const float *X, int64_t n, int32_t d, int32_t S, int64_t m,
                          const int32_t *newS, const int32_t *oldS, const int32_t *counts,
                          const float *worst, bool cross_only, uint32_t *start, uint64_t *key,
                          int64_t cap) {
  cudaStream_t st = ctx->stream;
  std::vector<int8_t> hf(2 * (size_t)m);
  std::vector<int32_t> hr(2 * (size_t)m);
  for (int64_t j = 0; j < m; j++)
    for (int old = 0; old < 2; old++) {
      hf[old * m + j] = (int8_t)counts[4 * j + old];
      hr[old * m + j] = counts[4 * j + 2 + old];
    }
  Buf<int8_t> fwd(ctx, 2 * m);
  Buf<int32_t> rev(ctx, 2 * m);
  HDB_CUDA(cudaMemcpyAsync(fwd, hf.data(), hf.size(), cudaMemcpyHostToDevice, st));
  HDB_CUDA(cudaMemcpyAsync(rev, hr.data(), hr.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  // two chunks that follow one another in a warp hold more than one chunk's candidates
  const int64_t slots = 2 * cap + fp32_join_warps(ctx, m) * kListChunkMin;
  Candidates c(ctx, n, slots, kListChunkMin);
  const SampleOut lists{const_cast<int32_t *>(newS), const_cast<int32_t *>(oldS), fwd.get(), fwd.get() + m,
                        rev.get(), rev.get() + m};
  fp32_join(ctx, X, m, d, S, lists, worst, c.cl, cross_only);
  HDB_CHECK_LAUNCH();
  c.group(ctx);
  unsigned long long *h = static_cast<unsigned long long *>(ctx->pinned);
  HDB_CUDA(cudaMemcpyAsync(h, c.counters, 5 * sizeof(*h), cudaMemcpyDeviceToHost, st));
  ctx->sync();
  HDB_REQUIRE(h[0] == 0 && (int64_t)h[2] <= cap, HDB_ERR_ARG, "more candidates than key holds");
  HDB_CUDA(cudaMemcpyAsync(start, c.rstart, (n + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  HDB_CUDA(cudaMemcpyAsync(key, c.rl.key, h[2] * sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
  ctx->sync();
}

void bf16_distance_tiles(Context *ctx, const float *X, int64_t n, int32_t d, const int32_t *ids,
                         const int32_t *counts, int64_t tiles, float *out) {
  HDB_REQUIRE(n >= 1 && n < (int64_t(1) << 31) && d >= 1 && tc_dpad(d) <= kTcMaxDpad, HDB_ERR_ARG,
              "BF16 distance tiles: need 1 <= n < 2^31 and 1 <= d <= 256");
  HDB_REQUIRE(tiles >= 0, HDB_ERR_ARG, "BF16 distance tiles: negative tile count");
  if (tiles == 0) return;
  const int dpad = tc_dpad(d);
  Buf<uint16_t> Xb(ctx, (size_t)n * dpad);
  Buf<float> nrm(ctx, n);
  k_half_prepare<Bf16Op><<<grid_for(ctx, n, 8, 16), 256, 0, ctx->stream>>>(
      X, n, d, dpad, nullptr, 1.0f, 1.0f, reinterpret_cast<__nv_bfloat16 *>(Xb.get()), nrm);
  ctx->launches++;
  HDB_CHECK_LAUNCH();
  tc_gram_probe(ctx, Xb, nrm, n, dpad, ids, counts, tiles, out);
  ctx->sync();
  HDB_REQUIRE(!(ctx->take_dev_err() & DEVERR_TIMEOUT), HDB_ERR_TIMEOUT,
              "BF16 distance tiles: a pipeline wait gave up");
}

void knn_split(Context *ctx, const hdb_nnd_element *G, int64_t n, int32_t k, int32_t *ids,
               float *dist) {
  k_split<<<grid_for(ctx, n * k, 256), 256, 0, ctx->stream>>>(G, n * k, ids, dist); ctx->launches++;
  HDB_CHECK_LAUNCH();
}

void fix_distances(Context *ctx, const float *X, int64_t n, int32_t d, const int32_t *ids,
                   int32_t k, float *dist) {
  // the flag is in host memory: reading the device's error word back and clearing it takes
  // 13 us, as long as the kernel of a small set
  volatile uint32_t *outside =
      reinterpret_cast<volatile uint32_t *>(static_cast<char *>(ctx->pinned) + kPinnedFlagOffset);
  *outside = 0;
  k_fix_distances<<<grid_for(ctx, n * k, 256), 256, 0, ctx->stream>>>(X, n, d, ids, k, dist, outside); ctx->launches++;
  HDB_CHECK_LAUNCH();
  ctx->sync();
  HDB_REQUIRE(!*outside, HDB_ERR_ARG, "fix_distances: a neighbour id lies outside [0, n)");
}

}  // namespace hdb
