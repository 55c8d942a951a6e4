// pt_walk.cuh -- the ordered warp-per-bucket tree walk of the FP64 traversal
// (and of interaction-list recording), plus the FP64-exact opening tests that
// every traversal shares.
//
// Semantics: TransposedDownTraverser::recurse (src/Traverser.h:154-217) for
// one target bucket is a pre-order depth-first walk from the root: a Leaf is
// handed to GravityVisitor::leaf (P2P, the bucket itself included), an
// Internal node is tested with GravityVisitor::open and either descended or
// handed to GravityVisitor::node (P2C), an EmptyLeaf is skipped.  Per target
// particle the interactions are applied in exactly that order.
//
// B200 mapping: one warp owns one bucket (lanes = target particles).  A step of the
// pre-order walk takes up to four opened nodes of a frame (the breadth-first one a
// single node, from the 64-byte records): lanes 8e .. 8e + 7 classify the children of
// the e-th in parallel (contiguous; their classification fields come from the
// sibling blocks, walk_sib_index) into P2P / P2C (quadrupole) / P2C (softened
// monopole, GravityVisitor::openSoftening) / open; four ballots give the per-child
// masks (a frame's bits: P2P 0-7, P2C quadrupole 8-15, P2C monopole 16-23, open
// 24-31).  The terminal children before the first opened child are handed to the
// evaluator in child order, the
// rest waits on a per-warp shared-memory stack (walk_preorder).  Every decision
// is warp-uniform.  The tests use
// __dadd_rn/__dmul_rn so that they evaluate identically (no FMA contraction)
// in every translation unit: all traversal forms see the same interactions.
#pragma once

#include "pt_internal.cuh"

namespace pt {

constexpr int kWalkStack = 128;  // pre-order walk: at most 4 entries more per level than it takes off
constexpr int kBfsQueue = 512;  // pending sibling frames of a breadth-first walk
constexpr unsigned kFull = 0xffffffffu;

// Child classes.
enum : int { kClsNone = 0, kClsP2P = 1, kClsQuad = 2, kClsOpen = 3, kClsMono = 4 };

// Squared gap between a box and a point as Space::intersect of the
// reference's utility submodule accumulates it (stand-in convention: per axis
// d = lo - c if positive, else c - hi if positive, else nothing; summed x, y,
// z).  Written with selects: an axis without a gap adds 0 * 0, which leaves
// the (non-negative) sum unchanged, so the value is the branchy form's bit for
// bit.  Space::intersect(box, centre, rsq) is gap <= rsq (GravityVisitor::open,
// :180, and ::openSoftening, :127).
__device__ __forceinline__ double box_gap2_exact(const double lo[3], const double hi[3], double cx, double cy,
                                                 double cz) {
  const double c[3] = {cx, cy, cz};
  double dsq = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double a = __dadd_rn(lo[k], -c[k]), b = __dadd_rn(c[k], -hi[k]);
    const double d = (a > 0) ? a : ((b > 0) ? b : 0.0);
    dsq = __dadd_rn(dsq, __dmul_rn(d, d));
  }
  return dsq;
}

// Squared distance from a point to a box (0 inside); conservative helper.
__device__ __forceinline__ double box_dist2(const double lo[3], const double hi[3], double cx, double cy,
                                            double cz) {
  double dsq = 0.0, d;
  if ((d = lo[0] - cx) > 0) dsq += d * d; else if ((d = cx - hi[0]) > 0) dsq += d * d;
  if ((d = lo[1] - cy) > 0) dsq += d * d; else if ((d = cy - hi[1]) > 0) dsq += d * d;
  if ((d = lo[2] - cz) > 0) dsq += d * d; else if ((d = cz - hi[2]) > 0) dsq += d * d;
  return dsq;
}

// GravityVisitor::openSoftening (:122-128): the softening spheres overlap, or
// the target bucket's box meets the source sphere of radius 2*soft; gap2 is
// box_gap2_exact of the bucket box and the source centre (the same gap the
// opening test measured).
__device__ __forceinline__ bool open_softening_gap(double scx, double scy, double scz, double ssoft, double tcx,
                                                   double tcy, double tcz, double tsoft, double gap2) {
  double r1 = __dmul_rn(2.0, ssoft), r2 = __dmul_rn(2.0, tsoft);
  double dx = __dadd_rn(scx, -tcx), dy = __dadd_rn(scy, -tcy), dz = __dadd_rn(scz, -tcz);
  double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  double rs = __dadd_rn(r1, r2);
  if (d2 <= __dmul_rn(rs, rs)) return true;
  return gap2 <= __dmul_rn(r1, r1);
}

// Whether a P2P leaf may hold a pair that GravityVisitor::leaf softens (or
// the target itself): the box gap between the target bucket's particle box
// and the leaf's centre (plus offset) is within the leaf's reach plus both
// sides' largest softening.  Conservative: a leaf for which it is false has
// every pair at r >= soft_i + soft_j > 0.  rec = the leaf's WalkRec.
__device__ __forceinline__ bool p2p_leaf_near(const WalkRec* __restrict__ walk, int leaf, const double lo[3],
                                              const double hi[3], double tsoft_max, double ox, double oy,
                                              double oz) {
  const double2* r = reinterpret_cast<const double2*>(walk + leaf);
  const double2 c01 = r[0], c2reach = r[1], smax = r[2];
  const double gap2 = box_gap2_exact(lo, hi, __dadd_rn(c01.x, ox), __dadd_rn(c01.y, oy), __dadd_rn(c2reach.x, oz));
  const double reach = c2reach.y + smax.x + tsoft_max;
  return !(gap2 > reach * reach);
}

struct BucketGeom {
  double lo[3], hi[3];  // target bucket's particle bbox (CentroidData::box)
  double cm[3];         // target bucket's centre of mass
  double soft;          // target bucket's mass-weighted softening
  double soft_max;      // max particle softening in the bucket
};

__device__ __forceinline__ void load_bucket_geom(const Mom* mom, int node, BucketGeom& g) {
  const Mom& q = mom[node];
  g.lo[0] = q.lo[0]; g.lo[1] = q.lo[1]; g.lo[2] = q.lo[2];
  g.hi[0] = q.hi[0]; g.hi[1] = q.hi[1]; g.hi[2] = q.hi[2];
  g.cm[0] = q.cm[0]; g.cm[1] = q.cm[1]; g.cm[2] = q.cm[2];
  g.soft = q.soft;
  g.soft_max = q.soft_max;
}

// Class of one node against the bucket (GravityVisitor::open / node).  The
// box gap of the node's centre (plus offset) serves both the opening test and
// openSoftening's second clause; it is returned in gap2 (-1 where it was not
// needed: leaves, empty nodes, nodes opened by their count).
// The same with the bucket box passed apart (lo, hi: e.g. held in registers).
__device__ __forceinline__ int classify_node_gap(const WalkRec& w, const double lo[3], const double hi[3],
                                                 const BucketGeom& g, double ox, double oy, double oz, double& gap2) {
  gap2 = -1.0;
  if (w.type == kTypeLeaf) return kClsP2P;
  if (w.type != kTypeInternal) return kClsNone;
  if (w.count <= kMinParticleNode) return kClsOpen;
  const double cx = __dadd_rn(w.cm[0], ox), cy = __dadd_rn(w.cm[1], oy), cz = __dadd_rn(w.cm[2], oz);
  gap2 = box_gap2_exact(lo, hi, cx, cy, cz);
  if (gap2 <= w.orsq) return kClsOpen;
  return open_softening_gap(cx, cy, cz, w.soft, g.cm[0], g.cm[1], g.cm[2], g.soft, gap2) ? kClsMono : kClsQuad;
}

// The same without a replica offset (the node's centre as it is).
__device__ __forceinline__ int classify_node_gap_nooff(const WalkRec& w, const double lo[3], const double hi[3],
                                                       const BucketGeom& g, double& gap2) {
  gap2 = -1.0;
  if (w.type == kTypeLeaf) return kClsP2P;
  if (w.type != kTypeInternal) return kClsNone;
  if (w.count <= kMinParticleNode) return kClsOpen;
  gap2 = box_gap2_exact(lo, hi, w.cm[0], w.cm[1], w.cm[2]);
  if (gap2 <= w.orsq) return kClsOpen;
  return open_softening_gap(w.cm[0], w.cm[1], w.cm[2], w.soft, g.cm[0], g.cm[1], g.cm[2], g.soft, gap2) ? kClsMono
                                                                                                       : kClsQuad;
}

__device__ __forceinline__ int classify_node_gap(const WalkRec& w, const BucketGeom& g, double ox, double oy,
                                                 double oz, double& gap2) {
  return classify_node_gap(w, g.lo, g.hi, g, ox, oy, oz, gap2);
}

__device__ __forceinline__ int classify_node(const WalkRec& w, const BucketGeom& g, double ox, double oy, double oz) {
  double gap2;
  return classify_node_gap(w, g, ox, oy, oz, gap2);
}

// Classify up to 8 nodes [c0, c0+nvalid) against the bucket; returns frame bits.
__device__ __forceinline__ uint32_t classify_children(const WalkRec* __restrict__ walk, int64_t nnodes, int c0,
                                                      int nvalid, const BucketGeom& g, double ox, double oy,
                                                      double oz, int lane, unsigned long long& n_open,
                                                      unsigned* status) {
  int code = kClsNone;
  bool internal = false;
  if (lane < nvalid) {
    int64_t idx = (int64_t)c0 + lane;
    if (c0 < 0 || idx >= nnodes) {
      atomicOr(status, kErrCapacity);
    } else {
      const WalkRec w = walk[idx];
      internal = (w.type == kTypeInternal);
      code = classify_node(w, g, ox, oy, oz);
    }
  }
  uint32_t pp = __ballot_sync(kFull, code == kClsP2P) & 0xffu;
  uint32_t pq = __ballot_sync(kFull, code == kClsQuad) & 0xffu;
  uint32_t pm = __ballot_sync(kFull, code == kClsMono) & 0xffu;
  uint32_t op = __ballot_sync(kFull, code == kClsOpen) & 0xffu;
  n_open += (unsigned long long)__popc(__ballot_sync(kFull, internal) & 0xffu);
  return pp | (pq << 8) | (pm << 16) | (op << 24);
}

// One stack entry of the pre-order walk: terminals of the frame above that come
// first (pc0, pbits), then a classified frame (its children from c0 on).
struct __align__(16) WalkSeg {
  int32_t pc0;
  uint32_t pbits;
  int32_t c0;
  uint32_t bits;
};

// The classification fields of node >= 1 from its sibling block.
__device__ __forceinline__ WalkRec load_sibling(const double2* __restrict__ walks, int64_t node) {
  const double2* sb = walks + walk_sib_index(node, 0);
  const double2 v0 = sb[0], v1 = sb[8], v2 = sb[16];
  WalkRec r;
  r.cm[0] = v0.x;
  r.cm[1] = v0.y;
  r.cm[2] = v1.x;
  r.orsq = v1.y;
  r.soft = v2.x;
  const int tc = __double2hiint(v2.y);
  r.first_child = __double2loint(v2.y);
  r.type = tc & 7;
  r.count = tc >> 3;
  return r;
}

// Walk the tree for one bucket in the reference's per-bucket order (pre-order).
// sink.emit(c0, pp, pq, pm, last) receives runs of terminals among the children
// from c0 on, in child order, and a last call with none.  A popped frame's first four opened children are
// classified together (lanes 8e .. 8e + 7 take the children of the e-th): all of
// them would be classified later anyway, so the tests are the same, the steps
// fewer.  The classified frames wait on the stack, each behind the terminals
// that precede it in its parent.  Returns false on stack overflow.
template <class Sink>
__device__ __forceinline__ bool walk_preorder(const WalkRec* __restrict__ walk, const double2* __restrict__ walks,
                                              int64_t nnodes, const BucketGeom& g, double ox, double oy, double oz,
                                              WalkSeg* stack, int lane, Sink& sink, unsigned long long& n_open,
                                              unsigned* status) {
  int c0 = 0;  // the root, tested as a one-child frame
  uint32_t bits = classify_children(walk, nnodes, 0, 1, g, ox, oy, oz, lane, n_open, status);
  int sp = 0;
  const int e = lane >> 3, c = lane & 7;
  int e0 = 0;        // terminals to emit: first child and masks (one call site: the
  uint32_t eb = 0u;  // evaluation is inlined into it)
  bool have = true, last = false;
  while (true) {
    if (eb | (uint32_t)last) sink.emit(e0, eb & 0xffu, (eb >> 8) & 0xffu, (eb >> 16) & 0xffu, last);
    if (last) break;
    if (!have) {
      if (sp == 0) {
        last = true;
        eb = 0u;
        continue;
      }
      --sp;
      const WalkSeg f = stack[sp];
      e0 = f.pc0;
      eb = f.pbits;
      c0 = f.c0;
      bits = f.bits;
      have = true;
      continue;
    }
    const uint32_t op = bits >> 24;
    const uint32_t low = op ? (op & (0u - op)) - 1u : 0xffu;  // the children before the first opened one
    e0 = c0;
    eb = bits & (low * 0x00010101u);
    have = op != 0u;
    if (!have) continue;
    // the e-th opened child of this frame, and the last of the four taken
    uint32_t o = op;
    for (int q = 0; q < e; q++) o &= o - 1u;
    const int k = o ? __ffs(o) - 1 : 8;
    const int klast = __reduce_max_sync(kFull, o ? k : -1);
    const int m = min(4, __popc(op));
    int fc = -1, code = kClsNone;
    bool internal = false;
    if (o) {
      const int64_t parent = (int64_t)c0 + k;
      fc = parent == 0 ? walk[0].first_child : __double2loint(walks[walk_sib_index(parent, 2)].y);
      const int64_t idx = (int64_t)fc + c;
      if (fc < 1 || idx >= nnodes) {
        atomicOr(status, kErrCapacity);
      } else {
        const WalkRec w = load_sibling(walks, idx);
        internal = (w.type == kTypeInternal);
        code = classify_node(w, g, ox, oy, oz);
      }
    }
    const unsigned pp = __ballot_sync(kFull, code == kClsP2P), pq = __ballot_sync(kFull, code == kClsQuad);
    const unsigned pm = __ballot_sync(kFull, code == kClsMono), po = __ballot_sync(kFull, code == kClsOpen);
    n_open += (unsigned long long)__popc(__ballot_sync(kFull, internal));
    // what is left of this frame behind the children taken, then the later
    // children's frames, each behind the terminals since the one before it
    const uint32_t above = 0xffu & ~((2u << klast) - 1u);
    const uint32_t rest = bits & (above * 0x01010101u);
    if (sp + m + 1 > kWalkStack) return false;
    __syncwarp();
    if (rest) {
      if (lane == 0) stack[sp] = WalkSeg{0, 0u, c0, rest};
      ++sp;
    }
    if (c == 0 && e >= 1 && e < m) {
      const int kp = 31 - __clz(op & ((1u << k) - 1u));  // the opened child before this one
      const uint32_t between = ((1u << k) - 1u) & ~((2u << kp) - 1u);
      const uint32_t b = ((pp >> (8 * e)) & 0xffu) | (((pq >> (8 * e)) & 0xffu) << 8) |
                         (((pm >> (8 * e)) & 0xffu) << 16) | (((po >> (8 * e)) & 0xffu) << 24);
      stack[sp + m - 1 - e] = WalkSeg{c0, bits & (between * 0x00010101u), fc, b};
    }
    sp += m - 1;
    __syncwarp();
    c0 = __shfl_sync(kFull, fc, 0);
    bits = (pp & 0xffu) | ((pq & 0xffu) << 8) | ((pm & 0xffu) << 16) | ((po & 0xffu) << 24);
  }
  return true;
}

// The same walk in BasicDownTraverser order (src/Traverser.h:296-330, the
// deque used first in, first out): breadth first per bucket.  Siblings stay
// consecutive in that order, so the unit of the queue is a frame -- the 8
// children of an opened node -- processed in child order, each opened child
// queuing its own frame at the back.  queue is a per-warp ring of qcap frames
// (first-child indices).  Returns false if the ring overflows.
template <class Sink>
__device__ __forceinline__ bool walk_bucket_bfs(const WalkRec* __restrict__ walk, int64_t nnodes,
                                                const BucketGeom& g, double ox, double oy, double oz,
                                                int32_t* queue, int qcap, int lane, Sink& sink,
                                                unsigned long long& n_open, unsigned* status) {
  int c0 = 0;  // the root, as a one-child frame
  uint32_t bits = classify_children(walk, nnodes, 0, 1, g, ox, oy, oz, lane, n_open, status);
  int head = 0, tail = 0;
  while (true) {
    const uint32_t pp = bits & 0xffu, pq = (bits >> 8) & 0xffu, pm = (bits >> 16) & 0xffu, op = bits >> 24;
    uint32_t all = pp | pq | pm | op;
    while (all) {  // runs of terminals between the opened children
      const uint32_t nxt = all & op, first = nxt & (0u - nxt);
      const uint32_t run = first ? all & (first - 1u) : all;
      if (run) sink.emit(c0, pp & run, pq & run, pm & run, false);
      all &= ~run;
      if (first) {
        if (tail - head >= qcap) return false;
        const int fc = walk[c0 + __ffs(first) - 1].first_child;
        __syncwarp();
        if (lane == 0) queue[tail % qcap] = fc;
        __syncwarp();
        ++tail;
        all &= ~first;
      }
    }
    if (head == tail) break;
    c0 = queue[head % qcap];
    ++head;
    bits = classify_children(walk, nnodes, c0, 8, g, ox, oy, oz, lane, n_open, status);
  }
  sink.emit(c0, 0u, 0u, 0u, true);
  return true;
}

// The next bucket index of a warp (lane 0 grabs, all lanes receive it).  With
// smq, the warps of one SM take consecutive buckets from a batch that the SM's
// queue holds, so the warps resident on an SM work on neighbouring buckets:
// their targets, results and most of their node records share cache lines.  (On
// the periodic 256^3 lattice pass, whose outer replica walks leave little work
// per bucket besides loading its targets and adding to its results, this
// measured 239.5 -> 214.4 ms; the Plummer pass at N = 2^24 is unchanged.)  A
// queue word is (batch start + 1) << 32 | next index; zero = no batch yet.
// The warp that draws index 0 of an empty queue, or the index one past the
// batch, takes a new batch from the global counter (keeping its first bucket);
// warps that draw past the batch meanwhile take single buckets.
__device__ __forceinline__ unsigned grab_bucket(unsigned* work, unsigned long long* smq, unsigned batch, int lane) {
  unsigned bi = 0;
  if (lane == 0) {
    if (batch <= 1u) {
      bi = atomicAdd(work, 1u);
    } else {
      unsigned sm;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
      unsigned long long* q = smq + (sm & 255u);
      const unsigned long long old = atomicAdd(q, 1ull);
      const unsigned hi = (unsigned)(old >> 32), idx = (unsigned)old;
      if (hi != 0u && idx < batch) {
        bi = hi - 1u + idx;
      } else if (hi == 0u ? idx == 0u : idx == batch) {
        bi = atomicAdd(work, batch);
        atomicExch(q, ((unsigned long long)(bi + 1u) << 32) | 1ull);
      } else {
        bi = atomicAdd(work, 1u);
      }
    }
  }
  return __shfl_sync(kFull, bi, 0);
}

// A bucket's P2C evaluations (list entries times targets) in bucket_work, before
// its P2P pairs are added.  Written by the P2C evaluation, which runs once per
// batch of replicas; the walk that writes the lists may be repeated.
__device__ __forceinline__ void add_p2c_work(const TravParams& P, int64_t b, int count, int ntot, int lane) {
  if (P.bucket_work && lane == 0) {
    unsigned long long wk = (unsigned long long)count * (unsigned long long)ntot;
    if (P.accumulate) wk += P.bucket_work[b];
    P.bucket_work[b] = wk;
  }
}

// Sink that only counts the interaction list of a bucket.
struct ListCounter {
  int64_t n;
  __device__ void emit(int, uint32_t pp, uint32_t pq, uint32_t pm, bool) { n += __popc(pp | pq | pm); }
};

}  // namespace pt
