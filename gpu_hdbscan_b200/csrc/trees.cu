// Single-linkage tree, condensed tree, stability, excess-of-mass selection
// and labels -- all on the device.
//
// Reference: build_Linkage_tree, build_Condensed_tree, compute_stability,
// get_clusters and do_labelling (HDBSCAN/trees/tree.cu:171-746), which run as
// serial host loops (union-find replay, BFS, per-cluster scans).
//
// Linkage tree.  Node N+r merges the two components joined by sorted MST edge
// r; its children are the components' current roots, i.e. the largest edge
// rank inside each endpoint's component among edges < r (or the vertex itself).
// Edge ranks are processed as a binary divide and conquer: at every level each
// block of ranks [s, s+S) unions its lower half with a lock-free union-find,
// tags each component with its largest rank, and relabels the endpoints of its
// upper half by those tags.  Endpoint labels seen by different blocks of one
// level are disjoint, so all blocks share one union-find array.  Once the blocks
// are small enough for a thread block (k_link_blocks), the remaining levels run
// in its shared memory.  After log2(N) levels every edge's endpoint labels are
// exactly its two children.
//
// Condensed tree.  A node is visited by the reference's BFS iff it is the root
// or holds >= mpts points.  Chains of "one big child" nodes share a cluster; a
// node whose children are both big (a split) starts two clusters, numbered in
// BFS order (depth, then left to right).  Chain heads come from pointer jumping
// over the nodes.  Everything else about the order follows from two facts: down a
// chain the ranks descend, so the nodes in descending rank, grouped by cluster,
// are the chains top-down; and two nodes of one depth part at a split, so a
// split's depth and the number of points to its left, which place it in BFS
// order, are sums over the few splits above it of their chains' lengths and their
// left children's sizes.  Each point falls out at the lowest visited ancestor.
// Stability is summed per cluster in the reference's row order (chain nodes
// top-down, identical terms for the points of each small side), in FP32 with
// separate multiply/add roundings, or in FP64 when asked.
#include <algorithm>

#include "hdb_internal.cuh"
#include "trees.cuh"

namespace hdb {

namespace {

// ---------------------------------------------------------------------------
// Linkage tree
// ---------------------------------------------------------------------------
// Union-find over labels [0, 2n-1); hooks always point to a larger label, so
// every path ends at a root.  Hooking the smaller root keeps the hot labels
// -- a big component's internal label n + rank, which many edges of a level
// name -- as parents: the vertices joining it each hook their own record
// instead of contending for the hot one.  The step bounds only guard against corrupted
// state and report through the device error word.  A label's state at one
// level -- parent, the largest rank tagged to it (as a root), whether it was
// counted, the points its root accumulated -- is one 16-byte record, so the
// reset of a label is one store and a root's fields share a sector.
constexpr int64_t kUfBound = int64_t(1) << 31;

struct __align__(16) UfNode {
  int32_t p, maxr, seen, acc;
};

__device__ __forceinline__ int32_t uf_find(UfNode *u, int32_t x) {
  for (int64_t s = 0; s < kUfBound; s++) {
    const int32_t px = *reinterpret_cast<volatile int32_t *>(&u[x].p);
    if (px == x) return x;
    const int32_t ppx = *reinterpret_cast<volatile int32_t *>(&u[px].p);
    if (ppx != px) *reinterpret_cast<volatile int32_t *>(&u[x].p) = ppx;
    x = px;
  }
  return x;
}

__device__ __forceinline__ void uf_union(UfNode *u, int32_t a, int32_t b, uint32_t *err) {
  for (int64_t s = 0; s < kUfBound; s++) {
    a = uf_find(u, a);
    b = uf_find(u, b);
    if (a == b) return;
    if (a < b) { int32_t t = a; a = b; b = t; }
    if (atomicCAS(&u[b].p, b, a) == b) return;
  }
  atomicOr(err, DEVERR_TIMEOUT);
}

// Lower-half edge of a block that has an upper half at block size S.
__device__ __forceinline__ bool active_lower(int64_t r, int64_t S, int64_t m) {
  int64_t pos = r & (S - 1);
  int64_t half = S >> 1;
  return pos < half && (r - pos) + half < m;
}

__global__ void k_link_init(const hdb_mst_edge *__restrict__ mst, int64_t m,
                            int32_t *__restrict__ la, int32_t *__restrict__ lb) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    la[r] = mst[r].from_node;
    lb[r] = mst[r].to_node;
  }
}

__global__ void k_uf_init(int64_t total, int64_t n, UfNode *__restrict__ u,
                          int32_t *__restrict__ size) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    u[i] = UfNode{(int32_t)i, -1, 0, 0};
    size[i] = i < n ? 1 : 0;
  }
}

__global__ void k_level_union(const int32_t *__restrict__ la, const int32_t *__restrict__ lb,
                              int64_t m, int64_t S, UfNode *u, uint32_t *err) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x)
    if (active_lower(r, S, m)) uf_union(u, la[r], lb[r], err);
}

// MST input check: endpoints in [0, n).
__global__ void k_validate_mst(const hdb_mst_edge *__restrict__ mst, int64_t m, int64_t n,
                               uint32_t *err) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    hdb_mst_edge e = mst[r];
    if (e.from_node < 0 || e.from_node >= n || e.to_node < 0 || e.to_node >= n)
      atomicOr(err, DEVERR_ID_RANGE);
  }
}

// Tags every component with its largest rank and counts its points.  At the
// upper levels most active edges of a block share one root, so the lanes that
// share the first active lane's root combine their rank maximum and point
// count with redux.sync and one of them updates the root; the other lanes
// update their own roots.  The same components' labels stand on most of those
// edges, so a label's mark is read before it is taken: as an exchange each, the
// marks of one label queued up (20M points: 51 ms over 16 levels, 33 with the read).
__device__ __forceinline__ bool first_seen(UfNode *u, int32_t x) {
  if (*reinterpret_cast<volatile int32_t *>(&u[x].seen) != 0) return false;
  return atomicExch(&u[x].seen, 1) == 0;
}
__global__ void k_level_tag(const int32_t *__restrict__ la, const int32_t *__restrict__ lb,
                            int64_t m, int64_t S, int64_t n, UfNode *u,
                            const int32_t *__restrict__ size) {
  const int lane = lane_id();
  for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x; r0 < m; r0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = r0 + threadIdx.x;
    const bool act = r < m && active_lower(r, S, m);
    int32_t root = -1, add = 0;
    if (act) {
      const int32_t a = la[r], b = lb[r];
      root = uf_find(u, a);
      if (first_seen(u, a)) add += a < n ? 1 : size[a];
      if (first_seen(u, b)) add += b < n ? 1 : size[b];
    }
    const uint32_t am = __ballot_sync(0xffffffffu, act);
    if (!act) continue;
    const int32_t lead = __shfl_sync(am, root, __ffs(am) - 1);
    const uint32_t same = __ballot_sync(am, root == lead);
    if (root == lead) {
      const int32_t mr = __reduce_max_sync(same, (int32_t)r);
      const int32_t sum = __reduce_add_sync(same, add);
      if (lane == __ffs(same) - 1) {
        atomicMax(&u[root].maxr, mr);
        if (sum != 0) atomicAdd(&u[root].acc, sum);
      }
    } else {
      atomicMax(&u[root].maxr, (int32_t)r);
      if (add != 0) atomicAdd(&u[root].acc, add);
    }
  }
}

// The size of every component's new node (lower halves), and the new labels of
// the upper halves.
__global__ void k_level_relabel(int32_t *__restrict__ la, int32_t *__restrict__ lb, int64_t m,
                                int64_t S, int64_t n, UfNode *u, int32_t *__restrict__ size) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    if ((r & (S - 1)) < (S >> 1)) {
      if (!active_lower(r, S, m)) continue;
      const int32_t root = uf_find(u, la[r]);
      if (u[root].maxr == (int32_t)r) size[n + r] = u[root].acc;
      continue;
    }
    int32_t a = la[r], b = lb[r];
    int32_t ra = uf_find(u, a), rb = uf_find(u, b);
    int32_t ma = u[ra].maxr, mb = u[rb].maxr;
    if (ma >= 0) la[r] = (int32_t)(n + ma);
    if (mb >= 0) lb[r] = (int32_t)(n + mb);
  }
}

__global__ void k_level_reset(const int32_t *__restrict__ la, const int32_t *__restrict__ lb,
                              int64_t m, int64_t S, UfNode *__restrict__ u) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    if (!active_lower(r, S, m)) continue;
    const int32_t a = la[r], b = lb[r];
    u[a] = UfNode{a, -1, 0, 0};
    u[b] = UfNode{b, -1, 0, 0};
  }
}

// The levels of S ranks and fewer, one thread block per S consecutive ranks, in
// shared memory, and the tree's nodes.  The labels that the block's edges come
// with take the slots of a hash table (their local names); the node of the
// block's rank i is local name kSlots + i.  Every level runs the same steps as
// the kernels above, its labels' state in shared memory and the edges' labels in
// registers, with four block barriers; a level of the kernels above is a pass
// over all edges per step, so a block takes as many ranks as an SM's shared memory
// holds.  Against blocks of 512 ranks, four to an SM and two levels more outside
// (the whole tree, random spanning trees and the MSTs of blobs in 12 dimensions):
// 250 k edges 0.52 -> 0.47 ms, 500 k 0.82 -> 0.76, 2M 2.8 -> 2.7 and 3.1 -> 3.0, 10M
// 18.5 -> 18.1, 20M 66.3 -> 60.5.
struct LinkSmem {
  static constexpr int S = 2048, kThreads = 1024;
  static constexpr int kSlotBits = 13, kSlots = 1 << kSlotBits, kNames = kSlots + S;
  static_assert(kSlots == 4 * S, "a block's 2 S labels fill half of the table");
  int32_t label[kSlots];  // -1: empty
  int32_t p[kNames], maxr[kNames], acc[kNames], size[kNames];
  uint32_t seen[(kNames + 31) / 32];
};

__device__ __forceinline__ int32_t sm_find(int32_t *p, int32_t x, int bound) {
  volatile int32_t *vp = p;
  for (int s = 0; s < bound; s++) {
    const int32_t px = vp[x];
    if (px == x) return x;
    const int32_t ppx = vp[px];
    if (ppx != px) vp[x] = ppx;
    x = px;
  }
  return x;
}

__global__ void __launch_bounds__(LinkSmem::kThreads)
    k_link_blocks(const hdb_mst_edge *__restrict__ mst, const int32_t *__restrict__ la,
                  const int32_t *__restrict__ lb, const int32_t *__restrict__ size, int64_t m,
                  int64_t n, hdb_linkage_node *__restrict__ out, uint32_t *err) {
  using L = LinkSmem;
  constexpr int S = L::S, kThreads = L::kThreads, kPer = S / kThreads;
  extern __shared__ __align__(16) unsigned char smem_link[];
  L &sh = *reinterpret_cast<L *>(smem_link);
  const int64_t first = (int64_t)blockIdx.x * S;
  const int cnt = (int)min((int64_t)S, m - first);
  for (int i = threadIdx.x; i < L::kNames; i += kThreads) {
    if (i < L::kSlots) sh.label[i] = -1;
    sh.p[i] = i;
    sh.maxr[i] = -1;
    sh.acc[i] = 0;
  }
  for (int i = threadIdx.x; i < (int)(sizeof(sh.seen) / 4); i += kThreads) sh.seen[i] = 0;
  __syncthreads();
  int32_t a[kPer], b[kPer];  // local names of the edge's endpoint labels
  auto name = [&](int32_t label) -> int32_t {
    uint32_t h = ((uint32_t)label * 0x9E3779B1u) >> (32 - L::kSlotBits);
    for (int probe = 0; probe < L::kSlots; probe++) {  // at most 2 S labels in 4 S slots
      const int32_t prev = atomicCAS(&sh.label[h], -1, label);
      if (prev == -1) sh.size[h] = label < n ? 1 : size[label];
      if (prev == -1 || prev == label) break;
      h = h + 1 == (uint32_t)L::kSlots ? 0 : h + 1;
    }
    return (int32_t)h;
  };
#pragma unroll
  for (int j = 0; j < kPer; j++) {
    const int i = j * kThreads + threadIdx.x;
    a[j] = b[j] = 0;
    if (i < cnt) {
      a[j] = name(la[first + i]);
      b[j] = name(lb[first + i]);
    }
  }
  __syncthreads();
  for (int s = S; s >= 2; s >>= 1) {
    const int half = s >> 1;
    if (half >= cnt) continue;  // no upper half: for the whole block
    auto lower = [&](int i) { return i < cnt && (i & (s - 1)) < half && (i & ~(s - 1)) + half < cnt; };
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      if (!lower(j * kThreads + threadIdx.x)) continue;
      int32_t x = a[j], y = b[j];
      int step = 0;
      for (; step < L::kNames; step++) {
        x = sm_find(sh.p, x, L::kNames);
        y = sm_find(sh.p, y, L::kNames);
        if (x == y) break;
        if (x < y) { const int32_t t = x; x = y; y = t; }
        if (atomicCAS(&sh.p[y], y, x) == y) break;
      }
      if (step == L::kNames) atomicOr(err, DEVERR_TIMEOUT);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const int i = j * kThreads + threadIdx.x;
      if (!lower(i)) continue;
      const int32_t root = sm_find(sh.p, a[j], L::kNames);
      int32_t add = 0;
      for (int32_t x : {a[j], b[j]}) {
        const uint32_t bit = 1u << (x & 31);
        volatile uint32_t *mark = &sh.seen[x >> 5];
        if (!(*mark & bit) && !(atomicOr(&sh.seen[x >> 5], bit) & bit)) add += sh.size[x];
      }
      if (*reinterpret_cast<volatile int32_t *>(&sh.maxr[root]) < i) atomicMax(&sh.maxr[root], i);
      if (add) atomicAdd(&sh.acc[root], add);
    }
    __syncthreads();
    int32_t na[kPer], nb[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const int i = j * kThreads + threadIdx.x;
      na[j] = a[j];
      nb[j] = b[j];
      if (lower(i)) {
        const int32_t root = sm_find(sh.p, a[j], L::kNames);
        if (sh.maxr[root] == i) sh.size[L::kSlots + i] = sh.acc[root];
      } else if (i < cnt && (i & (s - 1)) >= half) {
        const int32_t ma = sh.maxr[sm_find(sh.p, a[j], L::kNames)];
        const int32_t mb = sh.maxr[sm_find(sh.p, b[j], L::kNames)];
        if (ma >= 0) na[j] = L::kSlots + ma;
        if (mb >= 0) nb[j] = L::kSlots + mb;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      if (lower(j * kThreads + threadIdx.x)) {
        for (int32_t x : {a[j], b[j]}) {
          sh.p[x] = x;
          sh.maxr[x] = -1;
          sh.acc[x] = 0;
          atomicAnd(&sh.seen[x >> 5], ~(1u << (x & 31)));
        }
      }
      a[j] = na[j];
      b[j] = nb[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < kPer; j++) {
    const int i = j * kThreads + threadIdx.x;
    if (i >= cnt) continue;
    auto global = [&](int32_t x) {
      return x < L::kSlots ? sh.label[x] : (int32_t)(n + first) + (x - L::kSlots);
    };
    hdb_linkage_node o;
    o.left_node = global(a[j]);
    o.right_node = global(b[j]);
    o.weight = mst[first + i].weight;
    o.node_size = sh.size[a[j]] + sh.size[b[j]];
    out[first + i] = o;
  }
}

// ---------------------------------------------------------------------------
// Condensed tree, stability, EOM, labels
// ---------------------------------------------------------------------------
// Clusters or splits that one block works on in a single launch.
constexpr int64_t kOneBlockItems = 8192;

enum : int8_t { KIND_SPLIT = 0, KIND_BOTHSMALL = 1, KIND_LEFTBIG = 2, KIND_RIGHTBIG = 3 };

// A single-linkage tree, or a forest with one tree per instance (seg):
// internal node n + r for rank r < m, where m = n - (number of trees).
struct TreeView {
  const hdb_linkage_node *h;
  int64_t n;  // points
  int64_t m;  // internal nodes
  int32_t mpts;
  Segments seg;
  __device__ __forceinline__ int32_t sz(int64_t x) const {
    return x < n ? 1 : h[x - n].node_size;
  }
  // Root of its tree: the last rank of the tree's instance.
  __device__ __forceinline__ bool is_root(int64_t r) const {
    if (seg.count == 0) return r == m - 1;
    const int32_t t = seg.of_rank(r);
    return r == seg.off[t + 1] - t - 2;
  }
};

__device__ __forceinline__ float lambda_of(float w) {
  // tree.cu:308-313: INFINITE = INT_MAX, else 1.0 / weight in double
  return w > 0.0f ? __double2float_rn(__drcp_rn((double)w)) : 2147483648.0f;
}

// Per internal node: parent pointers, side, kind, visited flag, lambda; and the
// first half of the hierarchy's check: children are earlier nodes and sizes add up,
// so parent pointers always go to larger ids (every upward walk ends at the root).
// A node that fails writes nothing.
__global__ void k_nodes(TreeView t, int32_t *__restrict__ par, int8_t *__restrict__ side,
                        int8_t *__restrict__ kind, int8_t *__restrict__ visited,
                        float *__restrict__ lam, uint32_t *err) {
  const int64_t m = t.m;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    const hdb_linkage_node h = t.h[r];
    const int64_t x = t.n + r;
    bool ok = h.left_node >= 0 && h.left_node < x && h.right_node >= 0 && h.right_node < x &&
              h.left_node != h.right_node;
    int64_t ls = 0, rs = 0;
    if (ok) {
      ls = t.sz(h.left_node);
      rs = t.sz(h.right_node);
      ok = ls + rs == h.node_size;
    }
    if (!ok) {
      atomicOr(err, DEVERR_ID_RANGE);
      continue;
    }
    par[h.left_node] = (int32_t)x;
    par[h.right_node] = (int32_t)x;
    side[h.left_node] = 0;
    side[h.right_node] = 1;
    const bool lb = ls >= t.mpts, rb = rs >= t.mpts;
    kind[r] = (lb && rb) ? KIND_SPLIT : (!lb && !rb) ? KIND_BOTHSMALL : lb ? KIND_LEFTBIG : KIND_RIGHTBIG;
    visited[r] = t.is_root(r) || h.node_size >= t.mpts;
    lam[r] = lambda_of(h.weight);
  }
}

// The other half: no node has two parents (its pointer is one parent's, so it does
// not point back to the other).  With that, the 2 m children are all the nodes but
// the roots, which the kernels below rely on: every visited node has its parent's
// chain or starts one, and every cluster has a node.
__global__ void k_one_parent(TreeView t, const int32_t *__restrict__ par, uint32_t *err) {
  const int64_t m = t.m;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    const hdb_linkage_node h = t.h[r];
    const int64_t x = t.n + r;
    if (h.left_node < 0 || h.left_node >= x || h.right_node < 0 || h.right_node >= x) continue;
    if (par[h.left_node] != (int32_t)x || par[h.right_node] != (int32_t)x)
      atomicOr(err, DEVERR_ID_RANGE);
  }
}

// Chain-head pointers: a node that continues its parent's chain points to the
// parent, a head to itself.
__global__ void k_head_init(TreeView t, const int32_t *__restrict__ par, const int8_t *__restrict__ side,
                            const int8_t *__restrict__ kind, const int8_t *__restrict__ visited,
                            int32_t *__restrict__ head, int32_t *__restrict__ split,
                            int32_t *__restrict__ vis) {
  const int64_t m = t.m;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    const bool v = visited[r];
    vis[r] = v;
    split[r] = v && kind[r] == KIND_SPLIT;
    if (!v) { head[r] = -1; continue; }
    int32_t h = (int32_t)r;
    if (!t.is_root(r)) {
      const int64_t x = t.n + r;
      const int32_t pr = par[x] - (int32_t)t.n;
      const int8_t pk = kind[pr];
      if ((pk == KIND_LEFTBIG && side[x] == 0) || (pk == KIND_RIGHTBIG && side[x] == 1)) h = pr;
    }
    head[r] = h;
  }
}

// Round `it` of the jumping, in place (a pointer read late has jumped further
// already); once a round changed nothing the later ones return at once, so the
// host queues as many as the longest chain could take and waits for none.
__global__ void k_head_jump(int64_t m, int32_t *head, int32_t *changed, int it) {
  if (it > 0 && changed[it - 1] == 0) return;
  volatile int32_t *vh = head;
  bool any = false;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t h = vh[r];
    if (h < 0) continue;
    const int32_t hh = vh[h];
    if (hh != h) {
      vh[r] = hh;
      any = true;
    }
  }
  if (__any_sync(0xffffffffu, any) && lane_id() == 0) changed[it] = 1;
}

// Provisional clusters: 0 .. trees - 1 the roots', trees + 2 q + side those of
// the q-th split's children (splits in ascending rank).  cid is indexed by the
// clusters' head nodes.
__global__ void k_split_nodes(TreeView t, const int32_t *__restrict__ split,
                              const int64_t *__restrict__ pos, int64_t trees,
                              int32_t *__restrict__ node, int32_t *__restrict__ cid) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < t.m;
       r += (int64_t)gridDim.x * blockDim.x) {
    if (t.is_root(r)) cid[r] = t.seg.count > 0 ? t.seg.of_rank(r) : 0;
    if (!split[r]) continue;
    const int64_t q = pos[r];
    node[q] = (int32_t)r;
    const hdb_linkage_node h = t.h[r];
    cid[h.left_node - t.n] = (int32_t)(trees + 2 * q);
    cid[h.right_node - t.n] = (int32_t)(trees + 2 * q + 1);
  }
}

// Cluster of every visited node, and the visited nodes in descending rank with
// their cluster as the sort key.
__global__ void k_node_cluster(int64_t m, const int32_t *__restrict__ vis,
                               const int64_t *__restrict__ vpos, int64_t nv,
                               const int32_t *__restrict__ head, const int32_t *__restrict__ cid,
                               int32_t *__restrict__ ncl, uint32_t *__restrict__ keys,
                               uint32_t *__restrict__ vals) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = vis[r] ? cid[head[r]] : -1;
    ncl[r] = c;
    if (c < 0) continue;
    const int64_t at = nv - 1 - vpos[r];
    keys[at] = (uint32_t)c;
    vals[at] = (uint32_t)r;
  }
}

__global__ void k_seg_bounds(const uint32_t *__restrict__ keys, int64_t cnt, int64_t *__restrict__ s0,
                             int64_t *__restrict__ s1) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t c = keys[i];
    if (i == 0 || keys[i - 1] != c) s0[c] = i;
    if (i == cnt - 1 || keys[i + 1] != c) s1[c] = i + 1;
  }
}

// A split's place, relative to the split above it: its chain's length, and the
// points to the left of the child that starts the chain.
struct SplitUp {
  int32_t up, depth, left, pad;
};
__global__ void k_split_up(TreeView t, int64_t ns, int64_t trees, const int32_t *__restrict__ node,
                           const int32_t *__restrict__ ncl, const int64_t *__restrict__ s0,
                           const int64_t *__restrict__ s1, SplitUp *__restrict__ out) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < ns;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = ncl[node[q]];
    SplitUp u{-1, (int32_t)(s1[c] - s0[c]), 0, 0};
    if (c >= trees) {
      u.up = (int32_t)((c - trees) >> 1);
      if ((c - trees) & 1) u.left = (int32_t)t.sz(t.h[node[u.up]].left_node);
    }
    out[q] = u;
  }
}

__device__ __forceinline__ SplitUp split_jump(const SplitUp *in, int64_t q) {
  SplitUp u = in[q];
  if (u.up >= 0) {
    const SplitUp v = in[u.up];
    u = SplitUp{v.up, u.depth + v.depth, u.left + v.left, 0};
  }
  return u;
}

__global__ void k_split_jump(int64_t ns, const SplitUp *__restrict__ in, SplitUp *__restrict__ out) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < ns;
       q += (int64_t)gridDim.x * blockDim.x)
    out[q] = split_jump(in, q);
}

// BFS order as a sort key: depth, then points to the left (bits wide).
__global__ void k_split_keys(int64_t ns, const SplitUp *__restrict__ up, int bits,
                             uint64_t *__restrict__ keys, uint32_t *__restrict__ vals) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < ns;
       q += (int64_t)gridDim.x * blockDim.x) {
    keys[q] = ((uint64_t)up[q].depth << bits) | (uint64_t)up[q].left;
    vals[q] = (uint32_t)q;
  }
}

__global__ void k_split_inst(const uint32_t *__restrict__ order, const int32_t *__restrict__ node,
                             int64_t ns, Segments seg, uint32_t *__restrict__ inst) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < ns;
       q += (int64_t)gridDim.x * blockDim.x)
    inst[q] = (uint32_t)seg.of_rank(node[order[q]]);
}

// Final cluster indices: the root 0, the t-th split in BFS order gives 1 + 2 t
// (left) and 2 + 2 t (right).  A forest numbers its clusters tree after tree:
// the splits are sorted by (instance, BFS order), split t of instance s gives
// s + 1 + 2 t and s + 2 + 2 t, and instance s's root the index just before its
// first split's.  fin maps the provisional clusters; split_nodes the order.
__global__ void k_final_ids(int64_t ns, int64_t trees, const uint32_t *__restrict__ order,
                            const int32_t *__restrict__ node, const uint32_t *__restrict__ split_inst,
                            int32_t *__restrict__ fin, uint32_t *__restrict__ split_nodes) {
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t0 == 0 && !split_inst) fin[0] = 0;
  for (int64_t t = t0; t < ns; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = order[t], base = split_inst ? split_inst[t] : 0;
    split_nodes[t] = (uint32_t)node[q];
    fin[trees + 2 * q] = (int32_t)(base + 1 + 2 * t);
    fin[trees + 2 * q + 1] = (int32_t)(base + 2 + 2 * t);
  }
}

// One thread per instance s: its root's cluster index croot[s] = s + 2 *
// (splits of earlier instances), and cseg of the root.
__global__ void k_forest_roots(TreeView t, const uint32_t *__restrict__ split_inst, int64_t ns,
                               int32_t *__restrict__ fin, int32_t *__restrict__ croot,
                               int32_t *__restrict__ cseg, int64_t C) {
  const int32_t T = t.seg.count;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s <= T;
       s += (int64_t)gridDim.x * blockDim.x) {
    if (s == T) { croot[T] = (int32_t)C; continue; }
    int64_t lo = 0, hi = ns;  // first split of an instance >= s
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if ((int64_t)split_inst[mid] < s) lo = mid + 1; else hi = mid;
    }
    const int64_t c = s + 2 * lo;
    croot[s] = (int32_t)c;
    cseg[c] = (int32_t)s;
    fin[s] = (int32_t)c;
  }
}

// The nodes' clusters as ids n + index, and the chains' segments, in the final
// numbering.
__global__ void k_final_clusters(int64_t m, int64_t n, int64_t C, const int32_t *__restrict__ fin,
                                 int32_t *__restrict__ ncl, const int64_t *__restrict__ t0,
                                 const int64_t *__restrict__ t1, int64_t *__restrict__ s0,
                                 int64_t *__restrict__ s1) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < m || r < C;
       r += (int64_t)gridDim.x * blockDim.x) {
    if (r < m && ncl[r] >= 0) ncl[r] = (int32_t)n + fin[ncl[r]];
    if (r < C) {
      s0[fin[r]] = t0[r];
      s1[fin[r]] = t1[r];
    }
  }
}

__global__ void k_cluster_info(TreeView t, const uint32_t *__restrict__ split_nodes, int64_t ns,
                               const uint32_t *__restrict__ split_inst,
                               const int32_t *__restrict__ ncl, const float *__restrict__ lam,
                               float *__restrict__ birth, int32_t *__restrict__ cparent,
                               int32_t *__restrict__ ckid0, int32_t *__restrict__ cseg) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < ns;
       q += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = split_nodes[q];
    int32_t pc = ncl[r];  // cluster whose chain ends at this split
    const int32_t base = split_inst ? (int32_t)split_inst[q] : 0;
    int32_t c0 = (int32_t)(base + 1 + 2 * q), c1 = c0 + 1;
    if (cseg) cseg[c0] = cseg[c1] = base;
    birth[c0] = lam[r];
    birth[c1] = lam[r];
    cparent[c0] = pc - (int32_t)t.n;
    cparent[c1] = pc - (int32_t)t.n;
    ckid0[pc - t.n] = c0;
  }
}

// Chain node data laid out in chain order, so the per-cluster sums stream
// contiguous memory: lambda, and either (count of points falling out, 0) or,
// for the split that ends the chain, (-size(left), size(right)).
struct ChainItem {
  float lam;
  int32_t a, b;
  int32_t pad;
};

__global__ void k_chain_items(TreeView t, const uint32_t *__restrict__ chain, int64_t cnt,
                              const int8_t *__restrict__ kind, const float *__restrict__ lam,
                              ChainItem *__restrict__ items) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t r = chain[i];
    const hdb_linkage_node h = t.h[r];
    const int8_t kd = kind[r];
    ChainItem it;
    it.lam = lam[r];
    it.pad = 0;
    if (kd == KIND_SPLIT) {
      it.a = -t.sz(h.left_node);
      it.b = t.sz(h.right_node);
    } else {
      it.a = kd == KIND_LEFTBIG ? t.sz(h.right_node)
             : kd == KIND_RIGHTBIG ? t.sz(h.left_node)
                                   : t.sz(h.left_node) + t.sz(h.right_node);
      it.b = 0;
    }
    items[i] = it;
  }
}

template <typename T> struct FpBits;
template <> struct FpBits<float> {
  static constexpr int kMant = 23;
  __device__ static int exp_field(float x) { return (__float_as_uint(x) >> 23) & 0xff; }
  __device__ static float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }
  __device__ static float add(float a, float b) { return __fadd_rn(a, b); }
  __device__ static float sub(float a, float b) { return __fsub_rn(a, b); }
  __device__ static float mul(float a, float b) { return __fmul_rn(a, b); }
  static constexpr int kBias = 127;
};
template <> struct FpBits<double> {
  static constexpr int kMant = 52;
  __device__ static int exp_field(double x) {
    return (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  }
  __device__ static double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
  __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
  __device__ static double sub(double a, double b) { return __dsub_rn(a, b); }
  __device__ static double mul(double a, double b) { return __dmul_rn(a, b); }
  static constexpr int kBias = 1023;
};

// s after `cnt` sequential round-to-nearest-even additions of v >= 0 --
// exactly what one row per point gives (compute_stability, tree.cu:504-512).
// Inside one binade of s the additions advance s by a fixed multiple of its
// ulp; with v an odd multiple of half an ulp (a tie) the first step may differ
// and every later one is equal.  So: take single steps until two consecutive
// increments inside one binade agree (and v < s, which keeps s1 - s exact),
// then jump to the last step that stays in the binade.
template <typename T>
__device__ T add_repeated(T s, T v, int64_t cnt) {
  using B = FpBits<T>;
  if (!(v > T(0))) {
    for (; cnt > 0; cnt--) s = B::add(s, v);
    return s;
  }
  T last_inc = T(-1);
  int last_exp = -1;
  while (cnt > 0) {
    const T s1 = B::add(s, v);
    cnt--;
    const int e0 = B::exp_field(s), e1 = B::exp_field(s1);
    // large step, subnormal ulp (that of a sum below 2^-103, 2^-970 in FP64), or binade change
    if (!(v < s) || e0 <= B::kMant || e0 != e1) {
      s = s1;
      last_inc = T(-1);
      continue;
    }
    const T inc = B::sub(s1, s);  // exact: s <= s1 <= 2s
    s = s1;
    if (inc == T(0)) return s;  // v under half an ulp: s stays put from now on
    if (inc == last_inc && e1 == last_exp && cnt > 0) {
      // steady: s advances by inc = dq ulps per step while it stays in binade e1
      const T u = B::pow2(e1 - B::kBias - B::kMant);
      const int64_t q = (int64_t)B::mul(s, B::pow2(B::kMant - (e1 - B::kBias)));  // s / u
      const int64_t dq = (int64_t)B::mul(inc, B::pow2(B::kMant - (e1 - B::kBias)));
      const int64_t qmax = (int64_t(1) << (B::kMant + 1)) - 1;
      int64_t t = (qmax - q) / dq;
      if (t > cnt) t = cnt;
      if (t > 0) {
        s = B::mul((T)(q + t * dq), u);  // exact: integer significand times a power of two
        cnt -= t;
      }
      last_inc = T(-1);
      continue;
    }
    last_inc = inc;
    last_exp = e1;
  }
  return s;
}

// A chain item's addends in the reference's row order: a points with lambda
// each, or for the split that ends the chain (lambda - birth) * child_size of
// its left and then its right child.
template <typename T>
struct Addends {
  T y0, y1;
  int32_t m0;  // rows that add y0
  __device__ __forceinline__ Addends(const ChainItem &it, float birth) {
    using B = FpBits<T>;
    const T v = B::sub((T)it.lam, (T)birth);
    const bool split = it.a < 0;
    y0 = split ? B::mul(v, (T)(-it.a)) : v;
    y1 = split ? B::mul(v, (T)it.b) : T(0);
    m0 = split ? 1 : it.a;
  }
};

// The running sum s = q * u, u its ulp.  While s stays in one binade, adding
// y >= 0 with round-to-nearest moves q by y / u rounded to an integer, whatever
// q is, unless y / u lies halfway between two integers (the even one of the
// two neighbours of q + y / u is taken then).  So a run of additions that
// neither meets such a tie nor leaves the binade is a sum of integers, in any
// order: every thread rounds its own addends.  A long chain leaves a binade some
// twenty times and, once s is large, meets hardly any ties; those stretches
// are added one by one.  A sum in no such binade (0, infinite, not a number) is
// kept by addends that leave it as it is: lambdas that equal the birth, or any
// after an infinite one.
template <typename T>
struct Binade {
  double u, inv_u;  // powers of two
  int64_t q, top;   // s / u, and where the binade ends
  double item_top;  // an addend of this many steps leaves it for certain
  bool ok;
  __device__ __forceinline__ explicit Binade(T s) {
    using B = FpBits<T>;
    const int e = B::exp_field(s) - B::kBias;
    // normal, and far enough from the ends of the double range for u and 1 / u
    ok = s > T(0) && e > (B::kMant == 52 ? -900 : -126) && e < (B::kMant == 52 ? 900 : 128);
    u = ok ? FpBits<double>::pow2(e - B::kMant) : 1.0;
    inv_u = ok ? FpBits<double>::pow2(B::kMant - e) : 1.0;
    q = ok ? (int64_t)((double)s * inv_u) : 0;
    top = int64_t(1) << (B::kMant + 1);
    item_top = (double)(int64_t(1) << B::kMant);
  }
  // m additions of y: their steps into `steps`, and about as many into `about`
  // (which cannot overflow); false if they have to be taken one by one
  __device__ __forceinline__ bool take(T y, int32_t m, uint64_t &steps, double &about) const {
    const double x = (double)y * inv_u;  // exact
    const double r = rint(x);
    if (!(y >= T(0)) || !(x * (double)m < item_top) || fabs(x - r) == 0.5) return false;
    steps += (uint64_t)m * (uint64_t)r;
    about += (double)m * r;
    return true;
  }
  __device__ __forceinline__ bool stays(uint64_t steps, double about) const {
    return about < (double)top && q + (int64_t)steps < top;
  }
  __device__ __forceinline__ T after(uint64_t steps) const { return (T)((double)(q + (int64_t)steps) * u); }
};

// An item's additions leave s as it is.
template <typename T>
__device__ __forceinline__ bool keeps(T s, const Addends<T> &ad) {
  using B = FpBits<T>;
  return s != s || (B::add(s, ad.y0) == s && B::add(s, ad.y1) == s);
}

// s after the m items that the warp's first m lanes hold, one by one.
template <typename T>
__device__ __noinline__ T add_serially(T s, const ChainItem &mine, float birth, int m) {
  using B = FpBits<T>;
  const Addends<T> ad(mine, birth);
  const int lane = lane_id();
  const uint32_t split_mask = __ballot_sync(0xffffffffu, lane < m && mine.a < 0);
  const uint32_t rep_mask = __ballot_sync(0xffffffffu, lane < m && mine.a > 1);
  if (rep_mask == 0) {  // unrolled: bound by the chain of additions
#pragma unroll
    for (int t = 0; t < 32; t++) {
      const T y0 = __shfl_sync(0xffffffffu, ad.y0, t), y1 = __shfl_sync(0xffffffffu, ad.y1, t);
      if (t < m) {
        s = B::add(s, y0);
        if ((split_mask >> t) & 1u) s = B::add(s, y1);
      }
    }
    return s;
  }
  for (int t = 0; t < m; t++) {
    const T y0 = __shfl_sync(0xffffffffu, ad.y0, t), y1 = __shfl_sync(0xffffffffu, ad.y1, t);
    const int32_t m0 = __shfl_sync(0xffffffffu, ad.m0, t);
    if ((rep_mask >> t) & 1u) s = add_repeated<T>(s, y0, m0);
    else s = B::add(s, y0);
    if ((split_mask >> t) & 1u) s = B::add(s, y1);
  }
  return s;
}

// s after the m <= 32 items of a warp.
template <typename T>
__device__ __forceinline__ T add_warp(T s, const ChainItem &mine, float birth, int m) {
  const Binade<T> bin(s);
  const Addends<T> ad(mine, birth);
  uint64_t steps = 0;
  double about = 0.0;
  if (!bin.ok) {  // for the whole warp
    if (__all_sync(0xffffffffu, lane_id() >= m || keeps<T>(s, ad))) return s;
    return add_serially<T>(s, mine, birth, m);
  }
  const bool fine = lane_id() >= m || (bin.take(ad.y0, ad.m0, steps, about) &&
                                       bin.take(ad.y1, 1, steps, about));
  if (__all_sync(0xffffffffu, fine)) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      steps += __shfl_xor_sync(0xffffffffu, steps, o);
      about += __shfl_xor_sync(0xffffffffu, about, o);
    }
    if (bin.stays(steps, about)) return bin.after(steps);
  }
  return add_serially<T>(s, mine, birth, m);
}

// Stability of each cluster: its chain items summed in FP32 in the reference's
// row order (and in FP64 alongside when kBoth).  One warp per cluster, 32 items
// per load, the next ones in flight; chains of more than kLongChain items are
// left to k_stability_long (their clusters listed in long_list).
// Both kernels stream 16 bytes an item and are bound by the latency of a step
// (load, round, reduce); the sum one by one had a chain of 32 additions and 64
// shuffles per 32 items instead.  10M x 12, 200 blobs, one chain holding most
// of the points: 238 -> 6.1 ms; 20M x 128, 200 blobs: 52 ms before.  Sums
// that stay as they are (get_clusters, all of it): two chains of 1M whose lambdas
// equal the birth 22.4 -> 0.8 ms, one of 2M with infinite ones 41.6 -> 1.0; 12M items, half of them ties, 337 -> 93.
constexpr int kLongChain = 4096;
template <bool kBoth>
__global__ void k_stability(int64_t C, const int64_t *__restrict__ seg_start,
                            const int64_t *__restrict__ seg_end, const ChainItem *__restrict__ items,
                            const float *__restrict__ birth, float *__restrict__ stab,
                            double *__restrict__ stab64, int32_t *__restrict__ long_list,
                            int32_t *__restrict__ long_count) {
  const int lane = lane_id();
  const int wpb = blockDim.x >> 5;
  for (int64_t c = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); c < C;
       c += (int64_t)gridDim.x * wpb) {
    const int64_t s0 = seg_start[c], e = seg_end[c];
    if (e - s0 > kLongChain) {
      if (lane == 0) long_list[atomicAdd(long_count, 1)] = (int32_t)c;
      continue;
    }
    const float b = birth[c];
    float s = 0.0f;
    double s64 = 0.0;
    ChainItem next = {0.0f, 0, 0, 0};
    if (s0 + lane < e) next = items[s0 + lane];
    for (int64_t base = s0; base < e; base += 32) {
      const ChainItem mine = next;
      if (base + 32 + lane < e) next = items[base + 32 + lane];
      const int m = (int)min((int64_t)32, e - base);
      s = add_warp<float>(s, mine, b, m);
      if (kBoth) s64 = add_warp<double>(s64, mine, b, m);
    }
    if (lane == 0) {
      stab[c] = s;
      stab64[c] = kBoth ? s64 : (double)s;
    }
  }
}

// One block per long chain, 4,096 items a step; a step with a tie or the end
// of a binade in it is taken again by one warp, 32 items at a time.
constexpr int kLongThreads = 1024, kLongItems = 4;
template <typename T>
struct LongStep {
  uint64_t steps;
  double about;
};
template <typename T>
__device__ T add_block(T s, const ChainItem (&mine)[kLongItems], float birth, int64_t base, int64_t e,
                       const ChainItem *__restrict__ items, LongStep<T> *sh, T *sh_s) {
  const int lane = lane_id(), w = threadIdx.x >> 5;
  const Binade<T> bin(s);
  if (bin.ok) {  // for the whole block
    uint64_t steps = 0;
    double about = 0.0;
    bool fine = true;
#pragma unroll
    for (int j = 0; j < kLongItems; j++) {
      if (base + j * kLongThreads + threadIdx.x >= e) continue;
      const Addends<T> ad(mine[j], birth);
      fine = fine && bin.take(ad.y0, ad.m0, steps, about) && bin.take(ad.y1, 1, steps, about);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      steps += __shfl_xor_sync(0xffffffffu, steps, o);
      about += __shfl_xor_sync(0xffffffffu, about, o);
    }
    if (lane == 0) sh[w] = LongStep<T>{steps, about};
    const bool all = __syncthreads_and(fine);
    if (all) {
      steps = sh[lane].steps;
      about = sh[lane].about;
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        steps += __shfl_xor_sync(0xffffffffu, steps, o);
        about += __shfl_xor_sync(0xffffffffu, about, o);
      }
      if (bin.stays(steps, about)) {  // the same in every thread
        __syncthreads();  // sh is free again
        return bin.after(steps);
      }
    }
  } else {
    bool keep = true;
#pragma unroll
    for (int j = 0; j < kLongItems; j++)
      if (base + j * kLongThreads + threadIdx.x < e) keep = keep && keeps<T>(s, Addends<T>(mine[j], birth));
    if (__syncthreads_and(keep)) return s;
  }
  if (w == 0) {
    const int64_t end = min(e, base + kLongThreads * kLongItems);
    ChainItem next = base + lane < end ? items[base + lane] : ChainItem{0.0f, 0, 0, 0};
    for (int64_t i = base; i < end; i += 32) {
      const ChainItem it = next;
      if (i + 32 + lane < end) next = items[i + 32 + lane];
      s = add_warp<T>(s, it, birth, (int)min((int64_t)32, end - i));
    }
    if (lane == 0) *sh_s = s;
  }
  __syncthreads();
  s = *sh_s;
  __syncthreads();
  return s;
}

template <bool kBoth>
__global__ void __launch_bounds__(kLongThreads)
    k_stability_long(const int32_t *__restrict__ long_list, const int32_t *__restrict__ long_count,
                     const int64_t *__restrict__ seg_start, const int64_t *__restrict__ seg_end,
                     const ChainItem *__restrict__ items, const float *__restrict__ birth,
                     float *__restrict__ stab, double *__restrict__ stab64) {
  static_assert(kLongThreads == 32 * 32, "one partial sum per lane");
  __shared__ LongStep<double> sh[32];
  __shared__ double sh_s;
  const int32_t count = *long_count;
  for (int32_t l = blockIdx.x; l < count; l += gridDim.x) {
    const int32_t c = long_list[l];
    const int64_t s0 = seg_start[c], e = seg_end[c];
    const float b = birth[c];
    float s = 0.0f;
    double s64 = 0.0;
    ChainItem next[kLongItems];
    auto load = [&](int64_t base) {
#pragma unroll
      for (int j = 0; j < kLongItems; j++) {
        const int64_t i = base + j * kLongThreads + threadIdx.x;
        if (i < e) next[j] = items[i];
      }
    };
    load(s0);
    for (int64_t base = s0; base < e; base += kLongThreads * kLongItems) {
      ChainItem mine[kLongItems];
#pragma unroll
      for (int j = 0; j < kLongItems; j++) mine[j] = next[j];
      load(base + kLongThreads * kLongItems);
      s = add_block<float>(s, mine, b, base, e, items, reinterpret_cast<LongStep<float> *>(sh),
                           reinterpret_cast<float *>(&sh_s));
      if (kBoth) s64 = add_block<double>(s64, mine, b, base, e, items, sh, &sh_s);
    }
    if (threadIdx.x == 0) {
      stab[c] = s;
      stab64[c] = kBoth ? s64 : (double)s;
    }
  }
}

// Excess of mass, bottom-up: the last of two siblings to finish continues
// with their parent (get_clusters, tree.cu:692-725).  Roots (the clusters
// without a parent: index 0, or one per tree of a forest) are never
// evaluated, as in the reference.  T: float (HDB_STAB_FP32) or double.
//
// The climb up the deepest branch is a serial chain.  kShared: one block does
// it all, the values and arrivals in shared memory (up to kOneBlockItems
// clusters), where a step takes a tenth of what it takes through L2 (0.49 ms for
// the tree of 2M points otherwise).
template <typename T, bool kShared>
__global__ void __launch_bounds__(kShared ? 1024 : 128)
    k_eom(int64_t C, const int32_t *__restrict__ ckid0, const int32_t *__restrict__ cparent,
          const T *__restrict__ stab, T *sub, int8_t *self_sel, int32_t *arrive) {
  extern __shared__ __align__(16) unsigned char smem_eom[];
  if (kShared) {
    sub = reinterpret_cast<T *>(smem_eom);
    arrive = reinterpret_cast<int32_t *>(smem_eom + sizeof(T) * C);
    for (int64_t c = threadIdx.x; c < C; c += blockDim.x) arrive[c] = 0;
    __syncthreads();
  }
  volatile T *vsub = sub;
  for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c0 < C;
       c0 += (int64_t)gridDim.x * blockDim.x) {
    if (cparent[c0] < 0 || ckid0[c0] >= 0) continue;  // start from leaf clusters
    int64_t c = c0;
    // leaf: no children -> subtree stability 0, never above its own
    vsub[c] = stab[c];
    self_sel[c] = 1;
    for (int64_t guard = 0; guard < C; guard++) {
      const int64_t p = cparent[c];
      if (p < 0 || cparent[p] < 0) break;  // parent is a root
      if (kShared) __threadfence_block(); else __threadfence();
      if (atomicAdd(&arrive[p], 1) == 0) break;  // sibling not done yet
      if (kShared) __threadfence_block(); else __threadfence();
      const int32_t k0 = ckid0[p];
      using B = FpBits<T>;
      const T ssum = B::add(B::add(T(0), vsub[k0]), vsub[k0 + 1]), own = stab[p];
      const bool over = ssum > own;
      vsub[p] = over ? ssum : own;
      self_sel[p] = over ? 0 : 1;
      c = p;
    }
  }
}

template <typename T>
void eom(Context *ctx, int64_t C, const int32_t *ckid0, const int32_t *cparent, const T *stab,
         int8_t *self_sel) {
  cudaStream_t st = ctx->stream;
  if (C <= kOneBlockItems) {
    const size_t smem = (sizeof(T) + sizeof(int32_t)) * C;
    HDB_CUDA(cudaFuncSetAttribute(k_eom<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)((sizeof(T) + sizeof(int32_t)) * kOneBlockItems)));
    k_eom<T, true><<<1, 1024, smem, st>>>(C, ckid0, cparent, stab, nullptr, self_sel, nullptr);
  } else {
    Buf<T> sub(ctx, C);
    Buf<int32_t> arrive(ctx, C);
    HDB_CUDA(cudaMemsetAsync(arrive, 0, C * sizeof(int32_t), st));
    k_eom<T, false><<<grid_for(ctx, C, 128), 128, 0, st>>>(C, ckid0, cparent, stab, sub, self_sel, arrive);
  }
  ctx->launches++;
  HDB_CHECK_LAUNCH();
}

// The cluster that covers each one: the highest cluster that selects itself on
// its way up (itself included, roots not), by doubling.  A cluster that covers
// itself is selected (get_clusters drops what lies below a selected cluster).
struct Cover {
  int32_t up, top;
};
__global__ void k_cover_init(int64_t C, const int32_t *__restrict__ cparent,
                             const int8_t *__restrict__ self_sel, Cover *__restrict__ out) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    const int32_t p = cparent[c];
    out[c] = Cover{p >= 0 && cparent[p] >= 0 ? p : -1, p >= 0 && self_sel[c] ? (int32_t)c : -1};
  }
}

__device__ __forceinline__ Cover cover_jump(const Cover *in, int64_t c) {
  Cover x = in[c];
  if (x.up >= 0) {
    const Cover y = in[x.up];
    x = Cover{y.up, y.top >= 0 ? y.top : x.top};
  }
  return x;
}

__global__ void k_cover_jump(int64_t C, const Cover *__restrict__ in, Cover *__restrict__ out) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x)
    out[c] = cover_jump(in, c);
}

// All rounds of a doubling over few items in one block (one launch instead of
// one a round): a and b are the two buffers, read and written in turn, so
// neither is read through the read-only cache.
template <typename T, T (*kJump)(const T *, int64_t)>
__device__ __forceinline__ void jump_all(int64_t count, T *a, T *b, int rounds) {
  for (int i = 0; i < rounds; i++) {
    for (int64_t q = threadIdx.x; q < count; q += blockDim.x) b[q] = kJump(a, q);
    __syncthreads();
    T *t = a; a = b; b = t;
  }
}
__global__ void __launch_bounds__(1024) k_split_jump_all(int64_t ns, SplitUp *a, SplitUp *b, int rounds) {
  jump_all<SplitUp, split_jump>(ns, a, b, rounds);
}
__global__ void __launch_bounds__(1024) k_cover_jump_all(int64_t C, Cover *a, Cover *b, int rounds) {
  jump_all<Cover, cover_jump>(C, a, b, rounds);
}

__global__ void k_selected(int64_t C, const Cover *__restrict__ cov, int32_t *__restrict__ sel,
                           int32_t *__restrict__ cover) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    cover[c] = cov[c].top;
    sel[c] = cov[c].top == (int32_t)c ? 1 : 0;
  }
}

// Points: fall-out node = parent of the highest ancestor holding < mpts points.
__global__ void k_points(TreeView t, const int32_t *__restrict__ par, const int32_t *__restrict__ ncl,
                         const float *__restrict__ lam, const int32_t *__restrict__ cover,
                         const float *__restrict__ birth, const int32_t *__restrict__ label_of,
                         int32_t *__restrict__ labels, int32_t *__restrict__ pcl,
                         float *__restrict__ plam) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < t.n;
       p += (int64_t)gridDim.x * blockDim.x) {
    int64_t a = p;
    while (true) {
      int32_t up = par[a];
      if (up < 0 || t.sz(up) >= t.mpts) break;
      a = up;
    }
    int64_t f = par[a] < 0 ? a : par[a];  // a is the root only if n < mpts
    int64_t fr = f - t.n;
    int32_t c = ncl[fr];
    float lp = lam[fr];
    int32_t s = cover[c - t.n];
    int32_t lab = -1;
    if (s >= 0 && lp > birth[s]) lab = label_of[s];
    labels[p] = lab;
    if (pcl) { pcl[p] = c; plam[p] = lp; }
  }
}

// Label of a selected cluster: its rank among the selected clusters of its
// tree (a forest restarts the count at each instance's root).
__global__ void k_label_map(int64_t C, const int32_t *__restrict__ sel, const int32_t *__restrict__ pos,
                            const int32_t *__restrict__ cseg, const int32_t *__restrict__ croot,
                            int32_t *__restrict__ label_of) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x)
    label_of[c] = sel[c] ? pos[c] - (cseg ? pos[croot[cseg[c]]] : 0) : -1;
}

__global__ void k_inst_clusters(int32_t T, const int32_t *__restrict__ pos,
                                const int32_t *__restrict__ croot, int32_t *__restrict__ out) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < T;
       s += (int64_t)gridDim.x * blockDim.x)
    out[s] = pos[croot[s + 1]] - pos[croot[s]];
}

__global__ void k_condensed_rows(TreeView t, const uint32_t *__restrict__ split_nodes, int64_t ns,
                                 const int32_t *__restrict__ ncl, const float *__restrict__ lam,
                                 const int32_t *__restrict__ pcl, const float *__restrict__ plam,
                                 hdb_condensed_node *__restrict__ rows, uint64_t *__restrict__ keys,
                                 uint32_t *__restrict__ vals) {
  const int64_t total = t.n + 2 * ns;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    hdb_condensed_node row;
    if (i < t.n) {
      row.parent = pcl[i];
      row.child = (int32_t)i;
      row.lambda_val = plam[i];
      row.child_size = 1;
    } else {
      int64_t q = (i - t.n) >> 1;
      int side = (int)((i - t.n) & 1);
      int64_t r = split_nodes[q];
      hdb_linkage_node h = t.h[r];
      row.parent = ncl[r];
      row.child = (int32_t)(t.n + 1 + 2 * q + side);
      row.lambda_val = lam[r];
      row.child_size = t.sz(side ? h.right_node : h.left_node);
    }
    rows[i] = row;
    keys[i] = ((uint64_t)(uint32_t)row.parent << 32) | (uint32_t)row.child;
    vals[i] = (uint32_t)i;
  }
}

__global__ void k_permute_rows(const hdb_condensed_node *__restrict__ in, const uint32_t *__restrict__ idx,
                               int64_t cnt, hdb_condensed_node *__restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[idx[i]];
}

__global__ void k_stab_out(int64_t C, int64_t n, const float *__restrict__ stab,
                           hdb_stability *__restrict__ out) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    hdb_stability s;
    s.cluster_id = (int32_t)(n + c);
    s.lambda = stab[c];
    out[c] = s;
  }
}

int bits_for(int64_t v) {
  int b = 0;
  while (b < 63 && (int64_t(1) << b) <= v) b++;
  return b < 1 ? 1 : b;
}

}  // namespace

void linkage_tree(Context *ctx, const hdb_mst_edge *mst, int64_t n, hdb_linkage_node *out,
                  const Segments &seg) {
  HDB_REQUIRE(n >= 2 && n < (int64_t(1) << 30), HDB_ERR_ARG, "linkage tree: bad n");
  cudaStream_t st = ctx->stream;
  const int64_t m = n - (seg.count > 0 ? seg.count : 1), total = n + m;
  Buf<int32_t> la(ctx, m), lb(ctx, m), size(ctx, total);
  Buf<UfNode> u(ctx, total);
  const int gm = grid_for(ctx, m, 256), gt = grid_for(ctx, total, 256);
  k_validate_mst<<<gm, 256, 0, st>>>(mst, m, n, ctx->dev_err); ctx->launches++;
  HDB_CHECK_LAUNCH();
  HDB_REQUIRE(!(ctx->take_dev_err() & DEVERR_ID_RANGE), HDB_ERR_ARG,
              "linkage tree: MST edge endpoint outside [0, n)");
  k_link_init<<<gm, 256, 0, st>>>(mst, m, la, lb); ctx->launches++;
  k_uf_init<<<gt, 256, 0, st>>>(total, n, u, size); ctx->launches++;
  HDB_CHECK_LAUNCH();
  const int64_t inner = LinkSmem::S;
  int64_t S = 1;
  while (S < m) S <<= 1;
  for (; S > inner; S >>= 1) {
    k_level_union<<<gm, 256, 0, st>>>(la, lb, m, S, u, ctx->dev_err); ctx->launches++;
    k_level_tag<<<gm, 256, 0, st>>>(la, lb, m, S, n, u, size); ctx->launches++;
    k_level_relabel<<<gm, 256, 0, st>>>(la, lb, m, S, n, u, size); ctx->launches++;
    if (S > 2 * inner) {
      k_level_reset<<<gm, 256, 0, st>>>(la, lb, m, S, u); ctx->launches++;
    }
    HDB_CHECK_LAUNCH();
  }
  const int smem = (int)sizeof(LinkSmem);
  HDB_CUDA(cudaFuncSetAttribute(k_link_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_link_blocks<<<(unsigned)ceil_div(m, inner), LinkSmem::kThreads, smem, st>>>(mst, la, lb, size, m, n, out,
                                                                             ctx->dev_err);
  ctx->launches++;
  HDB_CHECK_LAUNCH();
  HDB_REQUIRE(!(ctx->take_dev_err() & DEVERR_TIMEOUT), HDB_ERR_INTERNAL,
              "linkage tree: union-find exceeded its step bound");
}

void condense_select(Context *ctx, const hdb_linkage_node *h, int64_t n, int32_t mpts,
                     int32_t stab_mode, int32_t *labels, int32_t *num_clusters,
                     hdb_condensed_node *condensed, int64_t *condensed_size,
                     hdb_stability *stability, int64_t *num_stability, const Segments &seg,
                     int32_t *inst_clusters) {
  HDB_REQUIRE(n >= 2 && n < (int64_t(1) << 30), HDB_ERR_ARG, "condensed tree: bad n");
  HDB_REQUIRE(mpts >= 2, HDB_ERR_ARG, "condensed tree: mpts (min cluster size) must be >= 2");
  const bool forest = seg.count > 0;
  HDB_REQUIRE(!forest || (!condensed && !stability), HDB_ERR_ARG,
              "condensed tree: condensed rows and stabilities are per single tree");
  cudaStream_t st = ctx->stream;
  const int64_t trees = forest ? seg.count : 1;
  const int64_t m = n - trees, total = n + m;
  TreeView t{h, n, m, mpts, seg};
  const int gm = grid_for(ctx, m, 256), gn = grid_for(ctx, n, 256);
  int64_t *hp = static_cast<int64_t *>(ctx->pinned);
  int32_t *hflag = reinterpret_cast<int32_t *>(hp + 8);

  Buf<int32_t> par(ctx, total);
  Buf<int8_t> side(ctx, total), kind(ctx, m), visited(ctx, m);
  Buf<float> lam(ctx, m);
  HDB_CUDA(cudaMemsetAsync(par, 0xff, total * sizeof(int32_t), st));
  k_nodes<<<gm, 256, 0, st>>>(t, par, side, kind, visited, lam, ctx->dev_err); ctx->launches++;
  k_one_parent<<<gm, 256, 0, st>>>(t, par, ctx->dev_err); ctx->launches++;
  HDB_CHECK_LAUNCH();
  HDB_REQUIRE(!(ctx->take_dev_err() & DEVERR_ID_RANGE), HDB_ERR_ARG,
              "condensed tree: hierarchy is not a valid single-linkage tree");

  // chain heads by pointer jumping; the splits and the visited nodes counted
  Buf<int32_t> head(ctx, m), split(ctx, m), vis(ctx, m), changed(ctx, 64);
  Buf<int64_t> spos(ctx, m + 1), vpos(ctx, m + 1);
  HDB_CUDA(cudaMemsetAsync(changed, 0, 64 * sizeof(int32_t), st));
  k_head_init<<<gm, 256, 0, st>>>(t, par, side, kind, visited, head, split, vis); ctx->launches++;
  HDB_CHECK_LAUNCH();
  scan_exclusive_i32_i64(ctx, split, spos, m, spos.get() + m);
  scan_exclusive_i32_i64(ctx, vis, vpos, m, vpos.get() + m);
  HDB_CUDA(cudaMemcpyAsync(hp, spos.get() + m, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  HDB_CUDA(cudaMemcpyAsync(hp + 1, vpos.get() + m, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  for (int it = 0; it < bits_for(m); it++) {  // 2^rounds > m: the longest chain
    k_head_jump<<<gm, 256, 0, st>>>(m, head, changed, it); ctx->launches++;
  }
  HDB_CHECK_LAUNCH();
  ctx->sync();
  const int64_t ns = hp[0], nv = hp[1];
  const int64_t C = trees + 2 * ns;

  // provisional clusters; the chains, top-down, grouped by cluster
  Buf<int32_t> node(ctx, ns > 0 ? ns : 1), cid(ctx, m), ncl(ctx, m);
  k_split_nodes<<<gm, 256, 0, st>>>(t, split, spos, trees, node, cid); ctx->launches++;
  Buf<uint32_t> ckeys(ctx, nv), chain(ctx, nv);
  k_node_cluster<<<gm, 256, 0, st>>>(m, vis, vpos, nv, head, cid, ncl, ckeys, chain); ctx->launches++;
  HDB_CHECK_LAUNCH();
  radix_sort_u32(ctx, ckeys, chain, nv, 0, bits_for(C));
  Buf<int64_t> t0(ctx, C), t1(ctx, C), s0(ctx, C), s1(ctx, C);
  k_seg_bounds<<<grid_for(ctx, nv, 256), 256, 0, st>>>(ckeys, nv, t0, t1); ctx->launches++;
  HDB_CHECK_LAUNCH();

  // splits in BFS order -> final cluster numbers
  Buf<uint32_t> snodes(ctx, ns > 0 ? ns : 1), sinst;
  Buf<int32_t> fin(ctx, C), cseg, croot;
  if (forest) {
    sinst = Buf<uint32_t>(ctx, ns > 0 ? ns : 1);
    cseg = Buf<int32_t>(ctx, C);
    croot = Buf<int32_t>(ctx, trees + 1);
  }
  {
    const int gs = grid_for(ctx, ns, 256);
    Buf<uint32_t> order(ctx, ns > 0 ? ns : 1);
    if (ns > 0) {
      Buf<SplitUp> up(ctx, ns), up2(ctx, ns);
      Buf<uint64_t> skeys(ctx, ns);
      k_split_up<<<gs, 256, 0, st>>>(t, ns, trees, node, ncl, t0, t1, up); ctx->launches++;
      SplitUp *ua = up, *ub = up2;
      const int rounds = bits_for(ns);
      if (ns <= kOneBlockItems) {
        k_split_jump_all<<<1, 1024, 0, st>>>(ns, ua, ub, rounds); ctx->launches++;
        if (rounds & 1) std::swap(ua, ub);
      } else {
        for (int it = 0; it < rounds; it++) {
          k_split_jump<<<gs, 256, 0, st>>>(ns, ua, ub); ctx->launches++;
          std::swap(ua, ub);
        }
      }
      const int bits = bits_for(n);  // depth and points to the left are below n
      k_split_keys<<<gs, 256, 0, st>>>(ns, ua, bits, skeys, order); ctx->launches++;
      HDB_CHECK_LAUNCH();
      radix_sort_u64(ctx, skeys, order, ns, 0, 2 * bits);
      if (forest) {  // (instance, BFS order)
        k_split_inst<<<gs, 256, 0, st>>>(order, node, ns, seg, sinst); ctx->launches++;
        HDB_CHECK_LAUNCH();
        radix_sort_u32(ctx, sinst, order, ns, 0, bits_for(seg.count));
      }
    }
    k_final_ids<<<gs, 256, 0, st>>>(ns, trees, order, node, sinst.get(), fin, snodes); ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
  if (forest) {
    k_forest_roots<<<grid_for(ctx, trees + 1, 256), 256, 0, st>>>(t, sinst, ns, fin, croot, cseg,
                                                                   C); ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
  k_final_clusters<<<gm, 256, 0, st>>>(m, n, C, fin, ncl, t0, t1, s0, s1); ctx->launches++;
  HDB_CHECK_LAUNCH();

  // per-cluster info
  Buf<float> birth(ctx, C), stab(ctx, C);
  Buf<double> stab64(ctx, C);
  Buf<int32_t> cparent(ctx, C), ckid0(ctx, C);
  Buf<int8_t> self_sel(ctx, C);
  HDB_CUDA(cudaMemsetAsync(birth, 0, C * sizeof(float), st));
  HDB_CUDA(cudaMemsetAsync(cparent, 0xff, C * sizeof(int32_t), st));
  HDB_CUDA(cudaMemsetAsync(ckid0, 0xff, C * sizeof(int32_t), st));
  HDB_CUDA(cudaMemsetAsync(self_sel, 0, C, st));
  if (ns > 0) {
    k_cluster_info<<<grid_for(ctx, ns, 256), 256, 0, st>>>(t, snodes, ns, sinst.get(), ncl, lam,
                                                            birth, cparent, ckid0, cseg.get()); ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
  const int gc = grid_for(ctx, C, 128);
  {
    Buf<ChainItem> items(ctx, nv);
    k_chain_items<<<grid_for(ctx, nv, 256), 256, 0, st>>>(t, chain, nv, kind, lam, items); ctx->launches++;
    // at most m / kLongChain clusters have a long chain
    Buf<int32_t> long_list(ctx, m / kLongChain + 1), long_count(ctx, 1);
    HDB_CUDA(cudaMemsetAsync(long_count, 0, sizeof(int32_t), st));
    const int gs = grid_for(ctx, C, 4), gl = (int)std::min<int64_t>(m / kLongChain, 2 * ctx->num_sms);
    auto warps = stab_mode == HDB_STAB_FP64 ? k_stability<true> : k_stability<false>;
    auto blocks = stab_mode == HDB_STAB_FP64 ? k_stability_long<true> : k_stability_long<false>;
    warps<<<gs, 128, 0, st>>>(C, s0, s1, items, birth, stab, stab64, long_list, long_count);
    if (gl > 0) {
      blocks<<<gl, kLongThreads, 0, st>>>(long_list, long_count, s0, s1, items, birth, stab, stab64);
      ctx->launches++;
    }
    ctx->launches++;
    HDB_CHECK_LAUNCH();
  }

  // excess of mass
  if (stab_mode == HDB_STAB_FP64) eom<double>(ctx, C, ckid0, cparent, stab64, self_sel);
  else eom<float>(ctx, C, ckid0, cparent, stab, self_sel);
  Buf<int32_t> sel(ctx, C), cover(ctx, C);
  {
    Buf<Cover> cov(ctx, C), cov2(ctx, C);
    Cover *ca = cov, *cb = cov2;
    k_cover_init<<<gc, 128, 0, st>>>(C, cparent, self_sel, ca); ctx->launches++;
    const int rounds = bits_for(C);
    if (C <= kOneBlockItems) {
      k_cover_jump_all<<<1, 1024, 0, st>>>(C, ca, cb, rounds); ctx->launches++;
      if (rounds & 1) std::swap(ca, cb);
    } else {
      for (int it = 0; it < rounds; it++) {
        k_cover_jump<<<gc, 128, 0, st>>>(C, ca, cb); ctx->launches++;
        std::swap(ca, cb);
      }
    }
    k_selected<<<gc, 128, 0, st>>>(C, ca, sel, cover); ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
  Buf<int32_t> selpos(ctx, C + 1), label_of(ctx, C);
  scan_exclusive_i32_i32(ctx, sel, selpos, C, selpos.get() + C);
  k_label_map<<<gc, 128, 0, st>>>(C, sel, selpos, cseg.get(), croot.get(), label_of); ctx->launches++;
  HDB_CHECK_LAUNCH();

  // labels (and the per-point condensed rows when asked)
  Buf<int32_t> pcl;
  Buf<float> plam;
  if (condensed) {
    pcl = Buf<int32_t>(ctx, n);
    plam = Buf<float>(ctx, n);
  }
  k_points<<<gn, 256, 0, st>>>(t, par, ncl, lam, cover, birth, label_of, labels,
                               condensed ? pcl.get() : nullptr, condensed ? plam.get() : nullptr); ctx->launches++;
  HDB_CHECK_LAUNCH();
  HDB_CUDA(cudaMemcpyAsync(hflag, selpos.get() + C, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  Buf<int32_t> icl;
  if (forest && inst_clusters) {
    icl = Buf<int32_t>(ctx, trees);
    k_inst_clusters<<<grid_for(ctx, trees, 256), 256, 0, st>>>(seg.count, selpos, croot, icl); ctx->launches++;
    HDB_CHECK_LAUNCH();
    HDB_CUDA(cudaMemcpyAsync(inst_clusters, icl, trees * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  }
  if (condensed) {
    const int64_t rows = n + 2 * ns;
    Buf<hdb_condensed_node> tmp(ctx, rows);
    Buf<uint64_t> rkeys(ctx, rows);
    Buf<uint32_t> ridx(ctx, rows);
    k_condensed_rows<<<grid_for(ctx, rows, 256), 256, 0, st>>>(t, snodes, ns, ncl, lam, pcl, plam,
                                                                tmp, rkeys, ridx); ctx->launches++;
    HDB_CHECK_LAUNCH();
    radix_sort_u64(ctx, rkeys, ridx, rows, 0, 64);
    k_permute_rows<<<grid_for(ctx, rows, 256), 256, 0, st>>>(tmp, ridx, rows, condensed); ctx->launches++;
    HDB_CHECK_LAUNCH();
    if (condensed_size) *condensed_size = rows;
  }
  if (stability) {
    k_stab_out<<<gc, 128, 0, st>>>(C, n, stab, stability); ctx->launches++;
    HDB_CHECK_LAUNCH();
  }
  if (num_stability) *num_stability = C;
  ctx->sync();
  if (num_clusters) *num_clusters = hflag[0];
}

}  // namespace hdb
