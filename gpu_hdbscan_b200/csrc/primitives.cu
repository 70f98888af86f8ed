// Device-wide primitives used by every stage: exclusive scans and a stable
// LSD radix sort.  Both are plain HBM-streaming kernels (tiles of 2048
// elements per 256-thread block); no library code.
#include <cooperative_groups.h>

#include <algorithm>
#include <utility>

#include "hdb_internal.cuh"

namespace hdb {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total.
template <typename T>
__device__ T block_exclusive_scan(T v, T *total, T *warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < (int)(blockDim.x >> 5)) warp_sums[lane] = w;
  }
  __syncthreads();
  T warp_prefix = warp > 0 ? warp_sums[warp - 1] : T(0);
  *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

template <typename In, typename Out>
__global__ void __launch_bounds__(kScanThreads) scan_tile_sums(const In *__restrict__ in,
                                                                Out *__restrict__ sums,
                                                                int64_t n) {
  __shared__ Out warp_sums[32];
  int64_t base = (int64_t)blockIdx.x * kScanTile;
  Out s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    int64_t idx = base + (int64_t)i * kScanThreads + threadIdx.x;
    if (idx < n) s += (Out)in[idx];
  }
  Out total;
  block_exclusive_scan<Out>(s, &total, warp_sums);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <typename In, typename Out>
__global__ void __launch_bounds__(kScanThreads) scan_tile_apply(const In *__restrict__ in,
                                                                 Out *__restrict__ out,
                                                                 const Out *__restrict__ offsets,
                                                                 int64_t n, Out *total_out) {
  __shared__ Out tile[kScanTile];
  __shared__ Out warp_sums[32];
  int64_t base = (int64_t)blockIdx.x * kScanTile;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    int idx = i * kScanThreads + threadIdx.x;
    int64_t g = base + idx;
    tile[idx] = g < n ? (Out)in[g] : Out(0);
  }
  __syncthreads();
  Out local[kScanItems];
  Out s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    local[i] = tile[threadIdx.x * kScanItems + i];
    s += local[i];
  }
  Out total;
  Out pre = block_exclusive_scan<Out>(s, &total, warp_sums);
  Out off = offsets ? offsets[blockIdx.x] : Out(0);
  Out run = off + pre;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    tile[threadIdx.x * kScanItems + i] = run;
    run += local[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    int idx = i * kScanThreads + threadIdx.x;
    int64_t g = base + idx;
    if (g < n) out[g] = tile[idx];
  }
  if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = off + total;
}

template <typename In, typename Out>
void scan_impl(Context *ctx, const In *in, Out *out, int64_t n, Out *total) {
  if (n <= 0) {
    if (total) HDB_CUDA(cudaMemsetAsync(total, 0, sizeof(Out), ctx->stream));
    return;
  }
  int64_t nb = ceil_div(n, kScanTile);
  if (nb == 1) {
    scan_tile_apply<In, Out><<<1, kScanThreads, 0, ctx->stream>>>(in, out, nullptr, n, total); ctx->launches++;
    HDB_CHECK_LAUNCH();
    return;
  }
  Buf<Out> sums(ctx, nb), offs(ctx, nb);
  scan_tile_sums<In, Out><<<(unsigned)nb, kScanThreads, 0, ctx->stream>>>(in, sums, n); ctx->launches++;
  HDB_CHECK_LAUNCH();
  scan_impl<Out, Out>(ctx, sums, offs, nb, (Out *)nullptr);
  scan_tile_apply<In, Out><<<(unsigned)nb, kScanThreads, 0, ctx->stream>>>(in, out, offs, n,
                                                                            total); ctx->launches++;
  HDB_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort.  One tile of kSortThreads * kItems keys per block;
// each pass sorts by (key >> shift) & mask, digits of up to 8 bits (256 bins)
// or 9 bits (512 bins).  The per-tile digit counts are laid out either
// digit-major ([digit][tile]: one flat exclusive scan gives every tile its
// output positions) or tile-major ([tile][digit]: every block reads and
// writes its own counts contiguously, and a column scan over chunks of
// tiles gives the positions).  The sorts of this file use tile-major counts
// and tiles of 4096 keys; the caller-buffer variant keeps the digit-major
// layout and 2048-key tiles its buffer sizes are stated in.
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;          // tile-major sorts: 4096-key tiles
constexpr int kSortItemsFlat = 8;       // digit-major (caller-buffer) sort: 2048-key tiles
constexpr uint32_t kColOneTiles = 2048; // up to here one cluster does the whole column scan

// How many keys there are: n, or what the device holds where the host only
// knows a bound (a list that kernels append to).
__device__ __forceinline__ int64_t key_count(int64_t n, const unsigned long long *__restrict__ dev) {
  if (!dev) return n;
  const int64_t c = (int64_t)*dev;
  return c < n ? c : n;
}

// Dynamic shared memory of one scatter block: the tile's keys and values in
// digit order, the per-warp digit counts, each digit's first tile position
// and first output position, and the warp totals of the digit scan.
template <typename K, typename V, bool kVals, int kBins, int kItems, bool kStable>
struct SortSmem {
  static constexpr int kHists = kStable ? kSortWarps : 1;  // ranks per warp, or over the block
  static constexpr int kTile = kSortThreads * kItems;
  static constexpr size_t kValsAt = sizeof(K) * kTile;
  static constexpr size_t kHistAt = kValsAt + (kVals ? sizeof(V) * kTile : 0);
  static constexpr size_t kStartAt = kHistAt + sizeof(uint32_t) * kHists * kBins;
  static constexpr size_t kGofsAt = kStartAt + sizeof(uint32_t) * kBins;
  static constexpr size_t kWsumAt = kGofsAt + sizeof(uint32_t) * kBins;
  static constexpr size_t kBytes = kWsumAt + sizeof(uint32_t) * kSortWarps;
};

template <bool kTileMajor>
__device__ __forceinline__ int64_t count_at(int d, uint32_t tile, uint32_t nblocks, int bins) {
  return kTileMajor ? (int64_t)tile * bins + d : (int64_t)d * nblocks + tile;
}

template <typename K, int kBins, int kItems, bool kTileMajor>
__global__ void __launch_bounds__(kSortThreads) radix_hist(const K *__restrict__ keys,
                                                            uint32_t *__restrict__ counts,
                                                            int64_t n, int shift, uint32_t mask,
                                                            uint32_t nblocks,
                                                            const unsigned long long *dev_n) {
  constexpr int kTile = kSortThreads * kItems;
  __shared__ uint32_t hist[kBins];
  n = key_count(n, dev_n);
  if ((int64_t)blockIdx.x * kTile >= n) return;
  for (int i = threadIdx.x; i < kBins; i += kSortThreads) hist[i] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kTile;
  K k[kItems];
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    const int64_t idx = base + (int64_t)i * kSortThreads + threadIdx.x;
    k[i] = idx < n ? keys[idx] : K(0);
  }
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    const int64_t idx = base + (int64_t)i * kSortThreads + threadIdx.x;
    if (idx < n) atomicAdd(&hist[(uint32_t)(k[i] >> shift) & mask], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kBins; i += kSortThreads)
    counts[count_at<kTileMajor>(i, blockIdx.x, nblocks, kBins)] = hist[i];
}

// The lanes of the caller's digit d (<= mask, below kBins) among the lanes that are
// ok: a ballot per bit.  A match_any takes a turn per distinct digit instead, some
// 58 cycles of a unit that the SM's four partitions share, and bounded the stable
// scatter (63 % of that unit's rate over the whole kernel): 2M x 32's reverse
// entries, five passes, 862 -> 627 us; 10M x 12's lists, second passes, 25.7 -> 23.0
// ms; one block's sort of 5,000 64-bit keys 66 -> 52 us.
template <int kBins>
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool ok, uint32_t mask) {
  uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int b = 0; (1 << b) < kBins; b++) {
    if (!((mask >> b) & 1u)) break;  // for the whole warp: a narrower digit
    const bool one = (d >> b) & 1u;
    const uint32_t with = __ballot_sync(0xffffffffu, one);
    peers &= one ? with : ~with;
  }
  return peers;
}

// Scatter of one tile for one digit.  Keys are ranked, the tile is laid out in
// digit order in shared memory, and each digit's run is then written by
// consecutive threads to consecutive addresses.  Values of type V (u32 or u64)
// move with their keys when kVals.  kStable keeps the input order within a digit:
// the lanes of a digit find one another by ballots (digit_peers).  Without it the
// ranks are the arrivals at the digit's count, and one count per digit does for the
// block, which leaves room for four blocks on an SM: six lists of 100k x 12 in one
// pass of 9 bits 348 -> 245 us, the first pass of six lists of 1M x 12 2.70 -> 2.36
// ms.  (Masks in shared memory in place of a match are slower: 2.9 ms at 6 bits.)
template <typename K, typename V, bool kVals, int kBins, int kItems, bool kTileMajor, bool kStable>
__global__ void __launch_bounds__(kSortThreads, kStable ? 3 : 4) radix_scatter(
    const K *__restrict__ keys_in, const V *__restrict__ vals_in, K *__restrict__ keys_out,
    V *__restrict__ vals_out, const uint32_t *__restrict__ offsets, int64_t n, int shift,
    uint32_t mask, uint32_t nblocks, const unsigned long long *dev_n) {
  using L = SortSmem<K, V, kVals, kBins, kItems, kStable>;
  constexpr int kTile = L::kTile;
  n = key_count(n, dev_n);
  if ((int64_t)blockIdx.x * kTile >= n) return;
  constexpr int kPer = kBins / kSortThreads;  // digits owned by each thread in the scan
  extern __shared__ __align__(16) unsigned char sort_smem[];
  K *tk = reinterpret_cast<K *>(sort_smem);
  V *tv = reinterpret_cast<V *>(sort_smem + L::kValsAt);
  uint32_t(*whist)[kBins] = reinterpret_cast<uint32_t(*)[kBins]>(sort_smem + L::kHistAt);
  uint32_t *dstart = reinterpret_cast<uint32_t *>(sort_smem + L::kStartAt);
  uint32_t *gofs = reinterpret_cast<uint32_t *>(sort_smem + L::kGofsAt);
  uint32_t *wsum = reinterpret_cast<uint32_t *>(sort_smem + L::kWsumAt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < L::kHists * kBins; i += kSortThreads) (&whist[0][0])[i] = 0;
  __syncthreads();
  const int64_t tile0 = (int64_t)blockIdx.x * kTile;
  const int64_t base = tile0 + (int64_t)warp * (32 * kItems);
  K k[kItems];
  V v[kItems];
  uint32_t dl[kItems];  // digit (low 16 bits) | rank among the warp's keys of that digit << 16
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int64_t idx = base + j * 32 + lane;
    k[j] = idx < n ? keys_in[idx] : K(0);
    if (kVals) v[j] = idx < n ? vals_in[idx] : V(0);
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const bool ok = base + j * 32 + lane < n;
    const uint32_t d = ok ? ((uint32_t)(k[j] >> shift) & mask) : (uint32_t)kBins;  // past the end: no digit
    uint32_t rank = 0;
    if (!kStable) {
      if (ok) rank = atomicAdd(&whist[0][d], 1u);
    } else {
      const uint32_t peers = digit_peers<kBins>(d, ok, mask);
      const int leader = __ffs(peers) - 1;
      if (ok) rank = whist[warp][d];
      __syncwarp();
      if (ok && lane == leader) whist[warp][d] = rank + __popc(peers);
      __syncwarp();
      rank += __popc(peers & lanemask_lt());
    }
    dl[j] = d | (rank << 16);
  }
  __syncthreads();
  {
    // kPer consecutive digits per thread: warp prefixes, then the digits'
    // counts in the tile, then an exclusive scan of the thread totals
    uint32_t run[kPer];
    uint32_t tsum = 0;
#pragma unroll
    for (int r = 0; r < kPer; r++) {
      const int d = threadIdx.x * kPer + r;
      uint32_t acc = 0;
#pragma unroll
      for (int w = 0; w < L::kHists; w++) {
        const uint32_t c = whist[w][d];
        whist[w][d] = acc;
        acc += c;
      }
      run[r] = acc;
      tsum += acc;
    }
    uint32_t x = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t excl = x - tsum;
    for (int w = 0; w < warp; w++) excl += wsum[w];
#pragma unroll
    for (int r = 0; r < kPer; r++) {
      const int d = threadIdx.x * kPer + r;
      dstart[d] = excl;
      excl += run[r];
      gofs[d] = offsets[count_at<kTileMajor>(d, blockIdx.x, nblocks, kBins)];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const uint32_t d = dl[j] & 0xffffu;
    if (d < (uint32_t)kBins) {
      const uint32_t pos = dstart[d] + (kStable ? whist[warp][d] : 0u) + (dl[j] >> 16);
      tk[pos] = k[j];
      if (kVals) tv[pos] = v[j];
    }
  }
  __syncthreads();
  const int64_t valid = n - tile0 < kTile ? n - tile0 : kTile;
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = j * kSortThreads + threadIdx.x;
    if (i < valid) {
      const K key = tk[i];
      const uint32_t d = (uint32_t)(key >> shift) & mask;
      const uint32_t pos = gofs[d] + (uint32_t)i - dstart[d];
      keys_out[pos] = key;
      if (kVals) vals_out[pos] = tv[i];
    }
  }
}

// Column scan of tile-major counts [tiles][kBins]: every tile's output position
// of its first key of each digit, and each digit's first position (base, with
// the total behind it).
//
// Up to kColOneTiles tiles, one cluster does it in one launch: CTA c owns 64
// digits, 16 threads each, a thread a run of consecutive tiles; the digits'
// totals are scanned over the cluster through distributed shared memory.  At
// 60 tiles of 512 bins it takes 4.7 us, where three launches with 512 tiles to a
// block took 33 us; at 1,300 tiles 16.4 us, as the three launches below with
// their gaps.
constexpr int kColDigits = 64, kColLanes = 16;
template <int kBins>
__global__ void __cluster_dims__(kBins / kColDigits, 1, 1) __launch_bounds__(kColDigits *kColLanes)
    radix_col_one(const uint32_t *__restrict__ counts, uint32_t *__restrict__ base,
                  uint32_t *__restrict__ offs, int64_t n, const unsigned long long *dev_n) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int kTile = kSortThreads * kSortItems;
  __shared__ uint32_t part[kColLanes][kColDigits];
  __shared__ uint32_t first[kColDigits];
  __shared__ uint32_t cta_total, half_total;
  n = key_count(n, dev_n);
  const uint32_t tiles = (uint32_t)((n + kTile - 1) / kTile);
  const int dl = threadIdx.x % kColDigits, l = threadIdx.x / kColDigits;
  const int rank = (int)cluster.block_rank(), lane = threadIdx.x & 31;
  const int d = rank * kColDigits + dl;
  const uint32_t per = (tiles + kColLanes - 1) / kColLanes;
  const uint32_t r0 = min((uint32_t)l * per, tiles), r1 = min(r0 + per, tiles);
  uint32_t s = 0;
#pragma unroll 8
  for (uint32_t r = r0; r < r1; r++) s += counts[(int64_t)r * kBins + d];
  part[l][dl] = s;
  __syncthreads();
  uint32_t total = 0, incl = 0;
  if (l == 0) {  // two warps: the digit's total, then an inclusive scan over the CTA's digits
#pragma unroll
    for (int j = 0; j < kColLanes; j++) {
      const uint32_t c = part[j][dl];
      part[j][dl] = total;
      total += c;
    }
    incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (threadIdx.x == 31) half_total = incl;
  }
  __syncthreads();
  if (l == 0) {
    if (threadIdx.x >= 32) incl += half_total;
    if (threadIdx.x == kColDigits - 1) cta_total = incl;
  }
  cluster.sync();
  if (l == 0) {
    uint32_t before = 0;
    for (int c = 0; c < rank; c++) before += *cluster.map_shared_rank(&cta_total, c);
    first[dl] = before + incl - total;
    base[d] = before + incl - total;
    if (d == kBins - 1) base[kBins] = before + incl;
  }
  cluster.sync();  // the other CTAs have read cta_total; `first` is written
  uint32_t run = first[dl] + part[l][dl];
#pragma unroll 8
  for (uint32_t r = r0; r < r1; r++) {
    const int64_t at = (int64_t)r * kBins + d;
    const uint32_t c = counts[at];
    offs[at] = run;
    run += c;
  }
}

// More tiles: one thread per digit and chunk of `rows` tiles, in three
// launches.  (1) per chunk, each digit's count in it;
template <int kBins>
__global__ void __launch_bounds__(kBins) radix_col_sums(const uint32_t *__restrict__ counts,
                                                        uint32_t *__restrict__ csum, uint32_t rows,
                                                        int64_t n, const unsigned long long *dev_n) {
  constexpr int kTile = kSortThreads * kSortItems;
  const int64_t nblocks = (key_count(n, dev_n) + kTile - 1) / kTile;
  const int d = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * rows;
  const int64_t r1 = r0 + rows < nblocks ? r0 + rows : nblocks;
  uint32_t s = 0;
#pragma unroll 8
  for (int64_t r = r0; r < r1; r++) s += counts[r * kBins + d];
  csum[(int64_t)blockIdx.x * kBins + d] = s;
}

// (2) radix_col_one over the chunks' sums: each chunk's output position of its
// first key of each digit (one block that scanned them was bound by its SM's
// share of L2: 489 chunks 27 us, 9.8 this way), and the digits' first positions.

// (3) every tile's output position of its first key of each digit.
template <int kBins>
__global__ void __launch_bounds__(kBins) radix_col_apply(const uint32_t *__restrict__ counts,
                                                         const uint32_t *__restrict__ cofs,
                                                         uint32_t *__restrict__ offs, uint32_t rows,
                                                         int64_t n, const unsigned long long *dev_n) {
  constexpr int kTile = kSortThreads * kSortItems;
  const int64_t nblocks = (key_count(n, dev_n) + kTile - 1) / kTile;
  const int d = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * rows;
  const int64_t r1 = r0 + rows < nblocks ? r0 + rows : nblocks;
  uint32_t run = cofs[(int64_t)blockIdx.x * kBins + d];
#pragma unroll 8
  for (int64_t r = r0; r < r1; r++) {
    const uint32_t c = counts[r * kBins + d];
    offs[r * kBins + d] = run;
    run += c;
  }
}

template <typename K, typename V, bool kVals, int kBins, int kItems, bool kTileMajor, bool kStable = true>
void launch_scatter(cudaStream_t st, const K *kin, const V *vin, K *kout, V *vout,
                    const uint32_t *offs, int64_t n, int shift, uint32_t mask, uint32_t nb,
                    const unsigned long long *dev_n = nullptr) {
  using L = SortSmem<K, V, kVals, kBins, kItems, kStable>;
  auto *fn = radix_scatter<K, V, kVals, kBins, kItems, kTileMajor, kStable>;
  if (L::kBytes > 48 * 1024)
    HDB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kBytes));
  fn<<<nb, kSortThreads, L::kBytes, st>>>(kin, vin, kout, vout, offs, n, shift, mask, nb, dev_n);
  HDB_CHECK_LAUNCH();
}

// LSD sort of the pairs in (keys, vals) with (ktmp, vtmp) as the second
// buffer; returns whether the result is in the second one.  Digit widths: the
// fewest passes of at most log2(kBins) bits over [begin_bit, end_bit), the bits
// spread evenly over them (25 bits with 512 bins: 9 + 8 + 8).  Stable with kStable.
// Without it the first pass leaves a digit's keys in any order and takes as many
// bits as it can, the later ones, which take a ballot a bit, the rest (1M x 12, 12
// bits: 9 + 3 2.2 ms for the second passes, 6 + 6 2.7 with a match).  dev_n: the count
// on the device, n then being a bound.  base_out (optional): the last pass's
// base, kBins + 1 values.
template <typename K, typename V, int kBins, bool kStable = true>
bool radix_sort_pingpong(Context *ctx, K *keys, V *vals, K *ktmp, V *vtmp, int64_t n, int begin_bit,
                         int end_bit, const unsigned long long *dev_n, uint32_t *base_out) {
  HDB_REQUIRE(n < (int64_t(1) << 32), HDB_ERR_ARG, "radix sort: more than 2^32 elements");
  constexpr int kMaxBits = kBins == 512 ? 9 : 8;
  static_assert(kBins == 256 || kBins == 512, "radix sort: 256 or 512 bins");
  constexpr int kTile = kSortThreads * kSortItems;
  const cudaStream_t st = ctx->stream;
  const uint32_t nb = (uint32_t)ceil_div(n, kTile);
  // chunks of the column scan: a few per SM, at most 512 tiles each
  const uint32_t rows = (uint32_t)std::min<int64_t>(
      512, std::max<int64_t>(32, ceil_div(nb, 4 * (int64_t)ctx->num_sms)));
  const bool one = nb <= kColOneTiles;
  const uint32_t nchunks = one ? 1 : (uint32_t)ceil_div(nb, rows);
  Buf<uint32_t> counts(ctx, (size_t)nb * kBins), offs(ctx, (size_t)nb * kBins),
      csum(ctx, (size_t)nchunks * kBins), cofs(ctx, (size_t)nchunks * kBins), base_buf;
  uint32_t *base = base_out;
  if (!base) {
    base_buf = Buf<uint32_t>(ctx, kBins + 1);
    base = base_buf;
  }
  K *kin = keys, *kout = ktmp;
  V *vin = vals, *vout = vtmp;
  int passes = 0;
  int left = end_bit - begin_bit;
  int npass = (left + kMaxBits - 1) / kMaxBits;
  for (int shift = begin_bit; left > 0; passes++, npass--) {
    const int bits = kStable ? (left + npass - 1) / npass : std::min(left, kMaxBits);
    const uint32_t mask = (1u << bits) - 1u;
    radix_hist<K, kBins, kSortItems, true><<<nb, kSortThreads, 0, st>>>(kin, counts, n, shift, mask,
                                                                       nb, dev_n);
    HDB_CHECK_LAUNCH();
    if (one) {
      radix_col_one<kBins><<<kBins / kColDigits, kColDigits * kColLanes, 0, st>>>(counts, base, offs,
                                                                                 n, dev_n);
      ctx->launches++;
    } else {
      radix_col_sums<kBins><<<nchunks, kBins, 0, st>>>(counts, csum, rows, n, dev_n);
      radix_col_one<kBins><<<kBins / kColDigits, kColDigits * kColLanes, 0, st>>>(
          csum, base, cofs, (int64_t)nchunks * kTile, nullptr);
      radix_col_apply<kBins><<<nchunks, kBins, 0, st>>>(counts, cofs, offs, rows, n, dev_n);
      ctx->launches += 3;
    }
    HDB_CHECK_LAUNCH();
    if (!kStable && passes == 0)
      launch_scatter<K, V, true, kBins, kSortItems, true, kStable>(st, kin, vin, kout, vout, offs, n,
                                                                   shift, mask, nb, dev_n);
    else if (vals)
      launch_scatter<K, V, true, kBins, kSortItems, true>(st, kin, vin, kout, vout, offs, n, shift,
                                                          mask, nb, dev_n);
    else
      launch_scatter<K, V, false, kBins, kSortItems, true>(st, kin, nullptr, kout, nullptr, offs,
                                                           n, shift, mask, nb, dev_n);
    ctx->launches += 2;
    std::swap(kin, kout);
    std::swap(vin, vout);
    shift += bits;
    left -= bits;
  }
  return (passes & 1) != 0;
}

// Up to kBlockSort pairs: every pass in one block and one launch, the pairs in
// shared memory between passes; a digit that all keys share is skipped.  5,000
// 64-bit keys: 52 us, where eight passes of three launches took 95 us and their
// gaps.  Up to 1,024 pairs one item a thread.
constexpr int kBlockSortThreads = 1024;
constexpr int kBlockSort = 8 * kBlockSortThreads;
template <typename K, typename V, bool kVals, int kItems>
struct BlockSortSmem {
  static constexpr int kMost = kItems * kBlockSortThreads;
  K key[kMost];
  uint32_t whist[kBlockSortThreads / 32][256];
  uint32_t dstart[256];
  uint32_t wsum[8];
  unsigned long long differ;
  V val[kVals ? kMost : 1];
};

template <typename K, typename V, bool kVals, int kItems>
__global__ void __launch_bounds__(kBlockSortThreads)
    radix_sort_block(K *__restrict__ keys, V *__restrict__ vals, int n, int begin_bit, int end_bit) {
  extern __shared__ __align__(16) unsigned char smem_block_sort[];
  using Smem = BlockSortSmem<K, V, kVals, kItems>;
  Smem &sh = *reinterpret_cast<Smem *>(smem_block_sort);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int base = w * (32 * kItems) + lane;  // a warp's keys are consecutive
  K k[kItems];
  V v[kItems];
  const K k0 = keys[0];
  if (tid == 0) sh.differ = 0;
  __syncthreads();
  K mine = 0;
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = base + 32 * j;
    k[j] = i < n ? keys[i] : k0;
    if (kVals && i < n) v[j] = vals[i];
    mine |= k[j] ^ k0;
  }
  if (mine) atomicOr(&sh.differ, (unsigned long long)mine);
  __syncthreads();
  const unsigned long long differ = sh.differ;
  for (int shift = begin_bit; shift < end_bit; shift += 8) {
    const uint32_t mask = (1u << min(8, end_bit - shift)) - 1u;
    if (((uint32_t)(differ >> shift) & mask) == 0) continue;  // for the whole block
    for (int i = tid; i < 256 * (kBlockSortThreads / 32); i += kBlockSortThreads) (&sh.whist[0][0])[i] = 0;
    __syncthreads();
    uint32_t dl[kItems];
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const bool ok = base + 32 * j < n;
      const uint32_t d = (uint32_t)(k[j] >> shift) & mask;
      const uint32_t peers = digit_peers<256>(d, ok, mask);
      const uint32_t below = __popc(peers & ((1u << lane) - 1u));
      uint32_t b = 0;
      if (ok) b = sh.whist[w][d];
      __syncwarp();
      if (ok && below == 0) sh.whist[w][d] = b + __popc(peers);
      __syncwarp();
      dl[j] = (ok ? d : 256u) | ((b + below) << 16);  // past the end: no digit
    }
    __syncthreads();
    if (tid < 256) {  // the digit's count per warp -> prefix; the digits' starts
      uint32_t acc = 0;
#pragma unroll 8
      for (int q = 0; q < kBlockSortThreads / 32; q++) {
        const uint32_t c = sh.whist[q][tid];
        sh.whist[q][tid] = acc;
        acc += c;
      }
      uint32_t x = acc;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) sh.wsum[w] = x;
      sh.dstart[tid] = x - acc;
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t before = 0;
      for (int q = 0; q < w; q++) before += sh.wsum[q];
      sh.dstart[tid] += before;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const uint32_t d = dl[j] & 0xffffu;
      if (d < 256) {
        const uint32_t at = sh.dstart[d] + sh.whist[w][d] + (dl[j] >> 16);
        sh.key[at] = k[j];
        if (kVals) sh.val[at] = v[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const int i = base + 32 * j;
      if (i < n) {
        k[j] = sh.key[i];
        if (kVals) v[j] = sh.val[i];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = base + 32 * j;
    if (i < n) {
      keys[i] = k[j];
      if (kVals) vals[i] = v[j];
    }
  }
}

template <typename K, typename V, bool kVals, int kItems>
void launch_block_sort(Context *ctx, K *keys, V *vals, int64_t n, int begin_bit, int end_bit) {
  const int smem = (int)sizeof(BlockSortSmem<K, V, kVals, kItems>);
  auto *fn = radix_sort_block<K, V, kVals, kItems>;
  HDB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  fn<<<1, kBlockSortThreads, smem, ctx->stream>>>(keys, vals, (int)n, begin_bit, end_bit);
  ctx->launches++;
  HDB_CHECK_LAUNCH();
}

template <typename K, typename V, int kBins>
void radix_sort_impl(Context *ctx, K *keys, V *vals, int64_t n, int begin_bit, int end_bit) {
  if (n <= 1 || end_bit <= begin_bit) return;
  if (n <= kBlockSort) {
    const bool few = n <= kBlockSortThreads;
    const auto fn = vals ? (few ? launch_block_sort<K, V, true, 1> : launch_block_sort<K, V, true, 8>)
                         : (few ? launch_block_sort<K, V, false, 1> : launch_block_sort<K, V, false, 8>);
    fn(ctx, keys, vals, n, begin_bit, end_bit);
    return;
  }
  Buf<K> ktmp(ctx, n);
  Buf<V> vtmp;
  if (vals) vtmp = Buf<V>(ctx, n);
  if (radix_sort_pingpong<K, V, kBins>(ctx, keys, vals, ktmp, vals ? vtmp.get() : nullptr, n,
                                       begin_bit, end_bit, nullptr, nullptr)) {
    HDB_CUDA(cudaMemcpyAsync(keys, ktmp, n * sizeof(K), cudaMemcpyDeviceToDevice, ctx->stream));
    if (vals)
      HDB_CUDA(cudaMemcpyAsync(vals, vtmp, n * sizeof(V), cudaMemcpyDeviceToDevice, ctx->stream));
  }
}

}  // namespace

void scan_exclusive_i32_i64(Context *ctx, const int32_t *in, int64_t *out, int64_t n,
                            int64_t *total) {
  scan_impl<int32_t, int64_t>(ctx, in, out, n, total);
}
void scan_exclusive_i32_i32(Context *ctx, const int32_t *in, int32_t *out, int64_t n,
                            int32_t *total) {
  scan_impl<int32_t, int32_t>(ctx, in, out, n, total);
}
void scan_exclusive_u32_u32(Context *ctx, const uint32_t *in, uint32_t *out, int64_t n,
                            uint32_t *total) {
  scan_impl<uint32_t, uint32_t>(ctx, in, out, n, total);
}
// 9-bit digits when they save a pass over 8-bit ones (e.g. 25-bit row ids).
static bool nine_bit_digits_help(int bits) { return (bits + 8) / 9 < (bits + 7) / 8; }

void radix_sort_u32(Context *ctx, uint32_t *keys, uint32_t *values, int64_t n, int begin_bit,
                    int end_bit) {
  if (nine_bit_digits_help(end_bit - begin_bit))
    radix_sort_impl<uint32_t, uint32_t, 512>(ctx, keys, values, n, begin_bit, end_bit);
  else
    radix_sort_impl<uint32_t, uint32_t, 256>(ctx, keys, values, n, begin_bit, end_bit);
}
void radix_sort_u64(Context *ctx, uint64_t *keys, uint32_t *values, int64_t n, int begin_bit,
                    int end_bit) {
  if (nine_bit_digits_help(end_bit - begin_bit))
    radix_sort_impl<uint64_t, uint32_t, 512>(ctx, keys, values, n, begin_bit, end_bit);
  else
    radix_sort_impl<uint64_t, uint32_t, 256>(ctx, keys, values, n, begin_bit, end_bit);
}
bool radix_group_u32_u64(Context *ctx, uint32_t *keys, uint64_t *values, uint32_t *keys2,
                         uint64_t *values2, int64_t cap, const unsigned long long *count,
                         int begin_bit, int end_bit, uint32_t *base) {
  return radix_sort_pingpong<uint32_t, uint64_t, 512, false>(ctx, keys, values, keys2, values2, cap,
                                                             begin_bit, end_bit, count, base);
}

// Stable LSD radix sort of u32 keys with u32 values in caller-provided
// buffers (nothing is allocated): ktmp/vtmp hold n elements each, counts and
// offs hold ceil(n / 2048) * 256 entries, scan_sums and scan_offs hold
// ceil(counts / 2048) entries, and that count must itself fit one scan tile.
// The result ends in keys/vals.  Used by the allocation-free entry point.
void radix_sort_u32_buffers(cudaStream_t st, uint32_t *keys, uint32_t *vals, uint32_t *ktmp,
                            uint32_t *vtmp, uint32_t *counts, uint32_t *offs, uint32_t *scan_sums,
                            uint32_t *scan_offs, int64_t n, int begin_bit, int end_bit) {
  if (n <= 1 || end_bit <= begin_bit) return;
  const uint32_t nb = (uint32_t)ceil_div(n, kSortThreads * kSortItemsFlat);
  const int64_t nc = (int64_t)nb * 256;
  const int64_t ns = ceil_div(nc, kScanTile);
  HDB_REQUIRE(ns <= kScanTile, HDB_ERR_ARG, "radix sort buffers: too many elements");
  uint32_t *kin = keys, *kout = ktmp, *vin = vals, *vout = vtmp;
  int passes = 0;
  for (int shift = begin_bit; shift < end_bit; shift += 8, passes++) {
    radix_hist<uint32_t, 256, kSortItemsFlat, false><<<nb, kSortThreads, 0, st>>>(
        kin, counts, n, shift, 0xffu, nb, nullptr);
    HDB_CHECK_LAUNCH();
    if (ns == 1) {
      scan_tile_apply<uint32_t, uint32_t><<<1, kScanThreads, 0, st>>>(counts, offs, nullptr, nc,
                                                                      nullptr);
    } else {
      scan_tile_sums<uint32_t, uint32_t><<<(unsigned)ns, kScanThreads, 0, st>>>(counts, scan_sums,
                                                                                nc);
      scan_tile_apply<uint32_t, uint32_t><<<1, kScanThreads, 0, st>>>(scan_sums, scan_offs, nullptr,
                                                                      ns, nullptr);
      scan_tile_apply<uint32_t, uint32_t><<<(unsigned)ns, kScanThreads, 0, st>>>(counts, offs,
                                                                                 scan_offs, nc,
                                                                                 nullptr);
    }
    HDB_CHECK_LAUNCH();
    launch_scatter<uint32_t, uint32_t, true, 256, kSortItemsFlat, false>(st, kin, vin, kout, vout,
                                                                         offs, n, shift, 0xffu, nb);
    uint32_t *t = kin; kin = kout; kout = t;
    t = vin; vin = vout; vout = t;
  }
  if (passes & 1) {
    HDB_CUDA(cudaMemcpyAsync(keys, kin, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    HDB_CUDA(cudaMemcpyAsync(vals, vin, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  }
}

}  // namespace hdb
