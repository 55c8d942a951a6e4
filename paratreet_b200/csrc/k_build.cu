// k_build.cu -- K5 octree build from the sorted keys, all levels at once.
//
// Restates Subtree::recursiveBuild (src/Subtree.h:314-349): every Internal
// node (more than `bucket` particles, src/Subtree.h:263-267) gets exactly 8
// children with keys key<<3 | c; child c's particle range ends at the first
// sorted key >= removeLeadingZeros(child_key + 1) (OctTree::
// findChildsLastParticle, src/Modularization.C:60-65 with src/Utility.h:33-50,
// :91-93, :127-130), the last child takes the rest.  Nodes are numbered breadth
// first (level after level, the children of a node contiguous, nodes of a level
// in key order); buckets are the leaves in DFS order (Subtree::leaves,
// src/Subtree.h:268-273).
//
// In the sorted keys a node of level L is a run of equal L-level prefixes, so
// the whole topology follows from two numbers per particle i (levels two keys
// share, 0..21):
//   d1(i) = levels shared with particle i - 1 (-1 for i = 0),
//   c(i)  = levels shared with particle i + bucket, at most 20 (-1 past the end):
// an Internal node of level L starts at i iff d1(i) < L <= c(i), and the
// deepest Internal level that contains i is A(i) = max c(j), j in [i - bucket,
// i], so a leaf (of level A(i) + 1) starts at i iff d1(i) <= A(i).  Four
// launches build the tree: count the Internal nodes of every level and the
// leaves per tile of particles; scan the tiles' counts; emit the Internal nodes
// and the bucket list (a node's rank in its level = the starts before it); and
// one thread per child finds its range and writes it.  The host reads the 22
// totals once.  (The level-by-level form this replaced -- flag, scan, a serial
// search for 8 children per thread, counts up and ranks down, a host read per
// level -- took 0.40 ms at N = 4096, 0.96 ms at 2^20 and 1.4 ms at 2^24, almost
// all of it launch gaps, host reads and chains of dependent loads.)
#include <cfloat>

#include "pt_internal.cuh"

namespace pt {

constexpr int kBuildThreads = 256;
constexpr int kBuildRounds = 4;
constexpr int kBuildTile = kBuildThreads * kBuildRounds;  // particles per CTA
constexpr int kBuildWarps = kBuildThreads / 32;
constexpr int kBuildSegs = kBuildRounds * kBuildWarps;  // 32: one segment = one warp in one round
static_assert(kBuildSegs == 32, "the segment scan maps one segment to one lane");
constexpr int kLeafCol = kMaxDepth;  // counter column of the leaves (0..20: Internal nodes of a level)

__device__ __forceinline__ int node_type_for(int64_t n, int bucket, int depth) {
  if (n == 0) return kTypeEmpty;
  if (n <= bucket || depth >= kMaxDepth) return kTypeLeaf;
  return kTypeInternal;
}

// Levels two sorted keys (placeholder bit 63 set in both) share, 0..21.
__device__ __forceinline__ int shared_levels(uint64_t a, uint64_t b) {
  const uint64_t x = a ^ b;
  return x == 0 ? kMaxDepth : (__clzll((long long)x) - 1) / 3;
}

// c(j) of the tile's particles and of the `bucket` before it, in shared memory:
// cs[k] belongs to particle tile0 - bucket + k.
__device__ __forceinline__ void load_shared_levels(const uint64_t* __restrict__ keys, int64_t n, int64_t tile0,
                                                   int bucket, int8_t* cs) {
  for (int k = threadIdx.x; k < kBuildTile + bucket; k += kBuildThreads) {
    const int64_t j = tile0 - bucket + k;
    int c = -1;
    if (j >= 0 && j + bucket < n) c = min(shared_levels(keys[j], keys[j + bucket]), kMaxDepth - 1);
    cs[k] = (int8_t)c;
  }
  __syncthreads();
}

struct Start {
  int d1, c, A;  // Internal nodes start at levels (d1, c]; A = deepest Internal level around the particle
  bool leaf;     // a leaf (level A + 1) starts here
};

__device__ __forceinline__ Start particle_start(const uint64_t* __restrict__ keys, int64_t n, int64_t i, int64_t tile0,
                                                int bucket, const int8_t* cs) {
  Start s{kMaxDepth, -1, -1, false};
  if (i < n) {
    const int k = (int)(i - tile0) + bucket;
    s.d1 = i == 0 ? -1 : shared_levels(keys[i - 1], keys[i]);
    s.c = cs[k];
    int A = -1;
    for (int w = 0; w <= bucket; w++) A = max(A, (int)cs[k - w]);
    s.A = A;
    s.leaf = s.d1 <= A;
  }
  return s;
}

__global__ void __launch_bounds__(kBuildThreads) tree_count(const uint64_t* __restrict__ keys, int64_t n, int bucket,
                                                           uint32_t* __restrict__ counts, int ntiles) {
  __shared__ int8_t cs[kBuildTile + 32];
  __shared__ uint32_t cnt[kLeafCol + 1];
  const int64_t tile0 = (int64_t)blockIdx.x * kBuildTile;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x <= kLeafCol) cnt[threadIdx.x] = 0;
  load_shared_levels(keys, n, tile0, bucket, cs);
  for (int r = 0; r < kBuildRounds; r++) {
    const Start s = particle_start(keys, n, tile0 + r * kBuildThreads + threadIdx.x, tile0, bucket, cs);
    const bool in = s.d1 < s.c;
    const int lo = __reduce_min_sync(0xffffffffu, in ? s.d1 + 1 : kMaxDepth);
    const int hi = __reduce_max_sync(0xffffffffu, in ? s.c : -1);
    for (int L = lo; L <= hi; L++) {
      const unsigned m = __ballot_sync(0xffffffffu, s.d1 < L && L <= s.c);
      if (lane == 0 && m) atomicAdd(&cnt[L], (uint32_t)__popc(m));
    }
    const unsigned m = __ballot_sync(0xffffffffu, s.leaf);
    if (lane == 0 && m) atomicAdd(&cnt[kLeafCol], (uint32_t)__popc(m));
  }
  __syncthreads();
  if (threadIdx.x <= kLeafCol) counts[(int64_t)threadIdx.x * ntiles + blockIdx.x] = cnt[threadIdx.x];
}

// Block L scans column L of the tiles' counts (exclusive, in place); totals[L].
constexpr int kColThreads = 512;
__global__ void __launch_bounds__(kColThreads) tree_scan(uint32_t* __restrict__ counts, int ntiles,
                                                         uint32_t* __restrict__ totals) {
  __shared__ uint32_t ws[kColThreads / 32];
  uint32_t* col = counts + (int64_t)blockIdx.x * ntiles;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int base = 0; base < ntiles; base += kColThreads) {
    const int i = base + threadIdx.x;
    const uint32_t v = i < ntiles ? col[i] : 0u;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    uint32_t before = carry, all = 0;
    for (int q = 0; q < kColThreads / 32; q++) {
      if (q < w) before += ws[q];
      all += ws[q];
    }
    if (i < ntiles) col[i] = before + inc - v;
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// First node of every level and the Internal nodes of the levels before it.
struct LevelBase {
  int32_t node[kMaxDepth + 2], internal[kMaxDepth + 1];
};
__device__ __forceinline__ void level_base(const uint32_t* __restrict__ totals, LevelBase& B) {
  int node = 0, in = 0, size = 1;
  for (int L = 0; L <= kMaxDepth; L++) {
    B.node[L] = node;
    B.internal[L] = in;
    node += size;
    const int t = L < kMaxDepth ? (int)totals[L] : 0;
    in += t;
    size = 8 * t;
  }
  B.node[kMaxDepth + 1] = node;
}

// inode[g] = (node, first child, first particle, level) of the g-th Internal
// node (level after level, key order), and buckets[] in DFS order.
__global__ void __launch_bounds__(kBuildThreads) tree_emit(Nodes nd, const uint64_t* __restrict__ keys, int64_t n,
                                                          int bucket, const uint32_t* __restrict__ counts, int ntiles,
                                                          const uint32_t* __restrict__ totals, int64_t cap,
                                                          int64_t nbuckets, int32_t* __restrict__ buckets,
                                                          unsigned* status) {
  __shared__ int8_t cs[kBuildTile + 32];
  __shared__ uint32_t seg[kLeafCol + 1][kBuildSegs];
  __shared__ LevelBase B;
  const int64_t tile0 = (int64_t)blockIdx.x * kBuildTile;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int k = threadIdx.x; k < (kLeafCol + 1) * kBuildSegs; k += kBuildThreads) (&seg[0][0])[k] = 0;
  if (threadIdx.x == 0) level_base(totals, B);
  load_shared_levels(keys, n, tile0, bucket, cs);
  Start s[kBuildRounds];
#pragma unroll
  for (int r = 0; r < kBuildRounds; r++) {
    s[r] = particle_start(keys, n, tile0 + r * kBuildThreads + threadIdx.x, tile0, bucket, cs);
    const bool in = s[r].d1 < s[r].c;
    const int lo = __reduce_min_sync(0xffffffffu, in ? s[r].d1 + 1 : kMaxDepth);
    const int hi = __reduce_max_sync(0xffffffffu, in ? s[r].c : -1);
    for (int L = lo; L <= hi; L++) {
      const unsigned m = __ballot_sync(0xffffffffu, s[r].d1 < L && L <= s[r].c);
      if (lane == 0) seg[L][r * kBuildWarps + w] = (uint32_t)__popc(m);
    }
    const unsigned m = __ballot_sync(0xffffffffu, s[r].leaf);
    if (lane == 0) seg[kLeafCol][r * kBuildWarps + w] = (uint32_t)__popc(m);
  }
  __syncthreads();
  for (int L = w; L <= kLeafCol; L += kBuildWarps) {  // exclusive prefix over the tile's segments, from the tile's own
    const uint32_t v = seg[L][lane];
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    seg[L][lane] = counts[(int64_t)L * ntiles + blockIdx.x] + inc - v;
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // the root
    nd.key[0] = 1ull;
    nd.type[0] = node_type_for(n, bucket, 0);
    nd.depth[0] = 0;
    nd.pstart[0] = 0;
    nd.pcount[0] = (int32_t)n;
    nd.parent[0] = -1;
    nd.fifo[0] = 0ull;
    if (n <= bucket) nd.first_child[0] = -1;
  }
#pragma unroll
  for (int r = 0; r < kBuildRounds; r++) {
    const Start q = s[r];
    const int64_t i = tile0 + r * kBuildThreads + threadIdx.x;
    const bool in = q.d1 < q.c;
    const uint64_t key = i < n ? keys[i] : 0ull;
    const int sg = r * kBuildWarps + w;
    // levels whose starts at or before i some lane needs: its own and its parent's
    int lo = in ? max(q.d1, 0) : kMaxDepth, hi = in ? q.c : -1;
    if (q.leaf && q.A >= 0) {
      lo = min(lo, q.A);
      hi = max(hi, q.A);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    int up = 0;     // starts of level L - 1 at or before i
    int leaf_up = 0;  // ... of level A
    for (int L = lo; L <= hi; L++) {
      const bool st = q.d1 < L && L <= q.c;
      const unsigned m = __ballot_sync(0xffffffffu, st);
      const int rank = (int)seg[L][sg] + __popc(m & lt);
      if (st) {
        const int g = B.internal[L] + rank;
        const int c0 = B.node[L + 1] + 8 * rank;
        const int node = L == 0 ? 0 : B.node[L] + 8 * (up - 1) + (int)((key >> (63 - 3 * L)) & 7u);
        if (node < 0 || (int64_t)c0 + 8 > cap) {  // never expected: the host sized the arrays from the totals
          atomicOr(status, kErrCapacity);
        } else {
          nd.first_child[node] = c0;
          nd.inode[g] = make_int4(node, c0, (int)i, L);
        }
      }
      up = rank + (st ? 1 : 0);
      if (L == q.A) leaf_up = up;
    }
    const unsigned m = __ballot_sync(0xffffffffu, q.leaf);
    if (q.leaf) {
      const int64_t b = (int64_t)seg[kLeafCol][sg] + __popc(m & lt);
      const int node =
          q.A < 0 ? 0 : B.node[q.A + 1] + 8 * (leaf_up - 1) + (int)((key >> (63 - 3 * (q.A + 1))) & 7u);
      if (b >= nbuckets || node < 0 || node >= cap) atomicOr(status, kErrCapacity);
      else buckets[b] = node;
    }
  }
}

// First index in [lo, n) whose key is >= v (keys[lo - 1] < v): doubling steps,
// then halving -- most nodes are a few steps long.
__device__ __forceinline__ int64_t first_ge(const uint64_t* __restrict__ keys, int64_t lo, int64_t n, uint64_t v) {
  int64_t step = 16, hi = lo + step;
  while (hi < n && keys[hi] < v) {
    lo = hi + 1;
    step <<= 1;
    hi = lo + step;
  }
  if (hi > n) hi = n;
  while (lo < hi) {
    const int64_t mid = lo + ((hi - lo) >> 1);
    if (keys[mid] >= v) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// Position of a leaf in the upward pass's FIFO (src/Subtree.h:352-361: leaves
// in DFS order, then empty leaves in DFS order) as an ordered number below 2^48:
// leaves by their first particle; empty leaves after all of them, by the
// particle gap they lie in and, inside one gap, in DFS order -- the trailing
// children along the path of the particle before the gap (deepest first), the
// children between the two paths, the leading children along the path of the
// particle after it.
__device__ __forceinline__ uint64_t fifo_of(int type, int64_t start, int64_t pstart, int64_t pfinish, int level, int c) {
  if (type == kTypeLeaf) return (uint64_t)start << 10;
  int sub = 200 + c;
  if (start == pfinish) sub = (kMaxDepth - level) * 8 + c;
  else if (start == pstart) sub = 256 + level * 8 + c;
  return (1ull << 47) | ((uint64_t)start << 10) | (uint64_t)sub;
}

// One thread per child: lanes 8e .. 8e + 7 write the children of one Internal
// node, each searching for its own end.
__global__ void __launch_bounds__(256) tree_children(Nodes nd, const uint64_t* __restrict__ keys, int64_t n, int bucket,
                                                     int64_t ninternal, int64_t cap, unsigned* status) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool live = (t >> 3) < ninternal;
  const int64_t g = live ? t >> 3 : ninternal - 1;
  const int c = (int)(t & 7), lane = threadIdx.x & 31;
  const int4 q = nd.inode[g];  // node, first child, first particle, level
  const int depth = q.w + 1;
  bool ok = q.x >= 0 && q.y >= 0 && (int64_t)q.y + 8 <= cap && q.z >= 0 && q.z < n && q.w >= 0 && q.w < kMaxDepth;
  int64_t end = 0, start = 0;
  uint64_t ck = 0;
  if (ok) {
    ck = ((keys[q.z] >> (63 - 3 * q.w)) << 3) | (uint64_t)c;
    const uint64_t v = (ck + 1) << (63 - 3 * depth);  // wraps to 0 behind the last key
    end = v == 0 ? n : first_ge(keys, q.z, n, v);
  }
  start = __shfl_up_sync(0xffffffffu, end, 1);
  const int64_t pfinish = __shfl_sync(0xffffffffu, end, (lane & 24) + 7);
  if (c == 0) start = q.z;
  const int cn = (int)(end - start);
  const int type = node_type_for(cn, bucket, depth);
  const unsigned in = __ballot_sync(0xffffffffu, ok && type == kTypeInternal);
  if (!live) return;
  if (!ok) {
    atomicOr(status, kErrCapacity);
    return;
  }
  const int64_t j = (int64_t)q.y + c;
  nd.key[j] = ck;
  nd.type[j] = type;
  nd.depth[j] = depth;
  nd.pstart[j] = (int32_t)start;
  nd.pcount[j] = cn;
  nd.parent[j] = q.x;
  if (type != kTypeInternal) {  // an Internal child's first_child was written with its inode
    nd.first_child[j] = -1;
    nd.fifo[j] = fifo_of(type, start, q.z, pfinish, q.w, c);
  }
  if (type == kTypeEmpty) {  // no particles: the moments an upward pass starts from
    Mom e{};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      e.lo[d] = DBL_MAX;
      e.hi[d] = -DBL_MAX;
    }
    nd.mom[j] = e;
    nd.count[j] = 0;
  }
  if (c == 0) {
    nd.npend[q.x] = __popc((in >> (lane & 24)) & 0xffu);
    nd.arrived[q.x] = 0;
  }
}

static inline unsigned blocks_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

int tree_columns() { return kLeafCol + 1; }
int tree_tiles(int64_t n) { return (int)((n + kBuildTile - 1) / kBuildTile); }

void launch_tree_count(const uint64_t* keys, int64_t n, int bucket, uint32_t* counts, uint32_t* totals,
                       cudaStream_t st) {
  const int tiles = tree_tiles(n);
  note_launch();
  tree_count<<<tiles, kBuildThreads, 0, st>>>(keys, n, bucket, counts, tiles);
  note_launch();
  tree_scan<<<kLeafCol + 1, kColThreads, 0, st>>>(counts, tiles, totals);
}

void launch_tree_emit(Nodes nd, const uint64_t* keys, int64_t n, int bucket, const uint32_t* counts,
                      const uint32_t* totals, int64_t ninternal, int64_t cap, int64_t nbuckets, int32_t* buckets,
                      unsigned* status, cudaStream_t st) {
  const int tiles = tree_tiles(n);
  note_launch();
  tree_emit<<<tiles, kBuildThreads, 0, st>>>(nd, keys, n, bucket, counts, tiles, totals, cap, nbuckets, buckets,
                                             status);
  if (ninternal > 0) {
    note_launch();
    tree_children<<<blocks_for(8 * ninternal), 256, 0, st>>>(nd, keys, n, bucket, ninternal, cap, status);
  }
}

}  // namespace pt
