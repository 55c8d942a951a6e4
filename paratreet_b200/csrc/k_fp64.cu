// k_fp64.cu -- FP64 kernels (this file is compiled with -fmad=false).
//
//  K6 upward pass
//     leaf_moments     CentroidData(particles, n, depth),
//                      examples/CentroidData.h:41-59, accumulating
//                      MultipoleMoments::operator+=(Particle) in particle order
//                      (examples/MultipoleMoments.h:274-353, non-HEXADECAPOLE)
//     upward_climb     Subtree::populateTree (src/Subtree.h:352-384): every
//                      parent combines its children with CentroidData::
//                      operator+= (examples/CentroidData.h:61-73,
//                      examples/MultipoleMoments.h:204-271, :458-469) in the
//                      order the reference's FIFO delivers them.  That order is
//                      reproduced without a queue: leaves hold FIFO rank
//                      (0, position) with all leaves before all empty leaves,
//                      each in DFS order (fifo_of, k_build.cu), and a parent's
//                      rank is (1 + chain, position) of its latest-ranked child -- parents enter the FIFO in the
//                      order their last child leaves it.
//     finalize         per-node traversal records (WalkRec, QuadRec).
//  K7 traverse_f64     warp-per-bucket walk (pt_walk.cuh) with the FP64
//                      GravityVisitor leaf / node terms, summed in the
//                      reference's order -- bit-identical to the reference
//                      built -DUSE_DOUBLE_FP.
//  K8 kick_perturb     Particle::kick + Particle::perturb
//                      (src/Particle.C:7-21) fused, and the leapfrog variant.
//  K9 direct_sum       FP64 spline direct sum (force-error yardstick).
#include <cfloat>

#include "pt_fp64.cuh"
#include "pt_internal.cuh"
#include "pt_walk.cuh"

namespace pt {

// Moments of one node held by eight lanes (r = lane & 7): lane r < 3 has centre
// coordinate r and the box along it, lane 3 the softening, lane r < 6 the second
// moment (quad_i, quad_j); the mass is on every lane.  A combine then takes one
// IEEE division per lane instead of four in a row on one lane, and the
// additions of the reference's moments stay in its order.
struct LaneMom {
  double mass, lin, quad, lo, hi;
};

__device__ __forceinline__ LaneMom lane_mom_clear() { return {0.0, 0.0, 0.0, DBL_MAX, -DBL_MAX}; }
// second moments in the order of Mom: xx xy xz yy yz zz
__device__ __forceinline__ int quad_i(int r) { return r < 3 ? 0 : r < 5 ? 1 : 2; }
__device__ __forceinline__ int quad_j(int r) { return r < 3 ? r : r == 3 ? 1 : 2; }

// The group's moments to the node's record.
__device__ __forceinline__ void lane_mom_store(Mom* __restrict__ out, const LaneMom& q, double radius, double reach,
                                               double soft_max, int r) {
  double* o = reinterpret_cast<double*>(out);  // mass cm soft radius | xx .. zz | lo hi | reach soft_max
  if (r < 4) o[1 + r] = q.lin;
  if (r < 6) o[6 + r] = q.quad;
  if (r < 3) {
    o[12 + r] = q.lo;
    o[15 + r] = q.hi;
  }
  if (r == 4) o[0] = q.mass;
  if (r == 5) o[5] = radius;
  if (r == 6) o[18] = reach;
  if (r == 7) o[19] = soft_max;
}
static_assert(sizeof(Mom) == 20 * sizeof(double), "lane_mom_store writes Mom's twenty doubles");

// CentroidData(particles, n, depth) of every bucket, four lanes per leaf: lane
// r < 3 centre coordinate r and the box along it, lane 3 the softening, each with
// one or two of the second moments; MultipoleMoments::operator+=(Particle),
// examples/MultipoleMoments.h:274-353, particle by particle.  (One thread per
// node, four divisions in a row per particle: 14 us at 10^4 and 15 at 10^5
// particles in buckets of 16, 51 us at 2^20, 504 us at 2^24 in buckets of 32; this
// 8, 10, 59 and 673 us: four times the warps for the same chain, which pays where
// the nodes are few.  Eight lanes with one second moment each: 934 us at 2^24.)
__global__ void __launch_bounds__(256) leaf_moments(Nodes nd, const int32_t* __restrict__ buckets, int64_t nbuckets,
                                                    Particles p, double4* __restrict__ src) {
  const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 2;
  if (g >= nbuckets) return;
  const int lane = threadIdx.x & 31, r = lane & 3;
  const unsigned gm = 0xfu << (lane & 28);
  const int node = buckets[g];
  const int s0 = nd.pstart[node], sn = nd.pcount[node];
  const double* const field = r == 0 ? p.x : r == 1 ? p.y : r == 2 ? p.z : p.soft;
  double mass = 0.0, lin = 0.0, lo = DBL_MAX, hi = -DBL_MAX, smax = 0.0;
  double qa = 0.0, qb = 0.0;  // xx xy xz yy by lane, and yz zz on lanes 0 and 1
  double v = field[s0], m = p.m[s0];
  for (int j = s0; j < s0 + sn; j++) {
    const double l2 = v, m2 = m, m1 = mass;
    if (j + 1 < s0 + sn) {
      v = field[j + 1];
      m = p.m[j + 1];
    }
    // the FP64 evaluation's source records (x, y, z, m)
    if (src) reinterpret_cast<double*>(src + j)[r] = r < 3 ? l2 : m2;
    if (l2 < lo) lo = l2;
    if (l2 > hi) hi = l2;
    smax = fmax(smax, l2);  // lane 3: the softening
    mass += m2;
    if (mass == 0.0) {
      lin = 0.5 * (lin + l2);
      continue;
    }
    const double old = lin;
    lin = (m1 * lin + m2 * l2) / mass;
    const double d = old - lin, e = l2 - lin;
    const double d0 = __shfl_sync(gm, d, 0, 4), d1 = __shfl_sync(gm, d, 1, 4), d2 = __shfl_sync(gm, d, 2, 4);
    const double e0 = __shfl_sync(gm, e, 0, 4), e1 = __shfl_sync(gm, e, 1, 4), e2 = __shfl_sync(gm, e, 2, 4);
    const bool yy = r == 3;
    qa += m1 * (yy ? d1 : d0) * (yy ? d1 : d);
    qa += m2 * (yy ? e1 : e0) * (yy ? e1 : e);
    qb += m1 * (r == 0 ? d1 : d2) * d2;
    qb += m2 * (r == 0 ? e1 : e2) * e2;
  }
  const double w = hi - lo;
  const double wx = __shfl_sync(gm, w, 0, 4), wy = __shfl_sync(gm, w, 1, 4), wz = __shfl_sync(gm, w, 2, 4);
  // not part of the reference's data: reach and max softening of the leaf,
  // used only to select the mixed form's unsoftened fast path
  const double cx = __shfl_sync(gm, lin, 0, 4), cy = __shfl_sync(gm, lin, 1, 4), cz = __shfl_sync(gm, lin, 2, 4);
  double r2max = 0.0;
  for (int j = s0 + r; j < s0 + sn; j += 4) {
    const double dx = p.x[j] - cx, dy = p.y[j] - cy, dz = p.z[j] - cz;
    r2max = fmax(r2max, dx * dx + dy * dy + dz * dz);
  }
  r2max = fmax(r2max, __shfl_xor_sync(gm, r2max, 2));
  r2max = fmax(r2max, __shfl_xor_sync(gm, r2max, 1));
  double* const o = reinterpret_cast<double*>(nd.mom + node);  // mass cm soft radius | xx .. zz | lo hi | reach soft_max
  o[1 + r] = lin;
  o[6 + r] = qa;
  if (r < 2) o[10 + r] = qb;
  if (r < 3) {
    o[12 + r] = lo;
    o[15 + r] = hi;
  } else {
    o[19] = smax;
  }
  if (r == 0) o[0] = mass;
  if (r == 1) o[5] = sn > 1 ? 0.5 * sqrt(wx * wx + wy * wy + wz * wz) : 1.0;
  if (r == 2) o[18] = sqrt(r2max);
  if (r == 0) nd.count[node] = sn;
}

// The upward pass over all levels in one launch: eight lanes per Internal node.
// The nodes without Internal children start; the group that brings a parent its
// last finished Internal child goes on with the parent (a counter per node, no
// waiting).  The children's moments are read in one round (lane c child c) and
// wait in shared memory while the group adds them (CentroidData::operator+= with
// MultipoleMoments::operator+=(MultipoleMoments)) in the order the reference's
// FIFO delivers them.  One launch per level, one thread per node and a load
// chain per child took 98 us at N = 4096 and 207 us at 2^20 (10-20 us per
// level); this form with every lane doing all of a combine 48 us at 4096; this 38.
constexpr int kClimbThreads = 128;
__global__ void __launch_bounds__(kClimbThreads) upward_climb(Nodes nd, int64_t ninternal) {
  __shared__ double kids[kClimbThreads / 8][8][19];  // odd stride: mass cm soft . | xx .. zz | lo hi, count
  const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
  if (g >= ninternal) return;
  const int lane = threadIdx.x & 31, r = lane & 7;
  const unsigned gm = 0xffu << (lane & 24);
  double(*K)[19] = kids[threadIdx.x >> 3];
  const int4 first = nd.inode[g];
  int node = first.x, c0 = first.y;
  if (nd.npend[node] != 0) return;
  while (true) {
    const int j = c0 + r;
    // past L1: another SM may have written the child in this launch
    const double2* m = reinterpret_cast<const double2*>(nd.mom + j);
    __syncwarp(gm);
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const double2 p = __ldcg(m + k);
      K[r][2 * k] = p.x;
      K[r][2 * k + 1] = p.y;
    }
    const int count = __ldcg(nd.count + j);
    const unsigned long long f = __ldcg(reinterpret_cast<const unsigned long long*>(nd.fifo) + j);
    int rank = 0;  // ascending FIFO position (all distinct)
#pragma unroll
    for (int o = 1; o < 8; o++) rank += __shfl_xor_sync(gm, f, o) < f;
    int cnt = count;
#pragma unroll
    for (int o = 4; o; o >>= 1) cnt += __shfl_xor_sync(gm, cnt, o);
    __syncwarp(gm);
    LaneMom q = lane_mom_clear();
    const int lin = 1 + min(r, 3), quad = 6 + min(r, 5), dim = min(r, 2);
    int src = 0;
    // first the serial chain of masses and centres (a division per child), then
    // the second moments, whose shuffles do not wait for one another
    double m1[8], m2[8], od[8], nw[8], qd[8];
    unsigned copy = 0, add = 0;
#pragma unroll
    for (int a = 0; a < 8; a++) {
      src = __ffs(__ballot_sync(gm, rank == a) & gm) - 1 - (lane & 24);
      const double* c = K[src];
      if (c[12 + dim] < q.lo) q.lo = c[12 + dim];
      if (c[15 + dim] > q.hi) q.hi = c[15 + dim];
      const double l2 = c[lin];
      m1[a] = q.mass;
      m2[a] = c[0];
      qd[a] = c[quad];
      od[a] = q.lin;
      q.mass += m2[a];
      if (q.mass == 0.0) {
        q.lin = 0.5 * (q.lin + l2);
      } else if (m1[a] == 0.0) {
        q.mass = m2[a];
        q.lin = l2;
        copy |= 1u << a;
      } else if (m2[a] != 0.0) {
        q.lin = (m1[a] * q.lin + m2[a] * l2) / q.mass;
        add |= 1u << a;
      }
      od[a] -= q.lin;
      nw[a] = l2 - q.lin;
    }
    const int qi = quad_i(r), qj = quad_j(r);
#pragma unroll
    for (int a = 0; a < 8; a++) {
      const double di = __shfl_sync(gm, od[a], qi, 8), dj = __shfl_sync(gm, od[a], qj, 8);
      const double ei = __shfl_sync(gm, nw[a], qi, 8), ej = __shfl_sync(gm, nw[a], qj, 8);
      if ((copy >> a) & 1u) q.quad = qd[a];
      if ((add >> a) & 1u) {
        q.quad += m1[a] * di * dj;
        q.quad += qd[a] + m2[a] * ei * ej;
      }
    }
    double e;
    {
      const double a = q.lin - q.lo, b = q.hi - q.lin;
      e = (a > b) ? a : b;
    }
    const double ex = __shfl_sync(gm, e, 0, 8), ey = __shfl_sync(gm, e, 1, 8), ez = __shfl_sync(gm, e, 2, 8);
    const double radius = cnt > 1 ? sqrt(ex * ex + ey * ey + ez * ez) : 1.0;
    const unsigned long long last = __shfl_sync(gm, f, src, 8);
    lane_mom_store(nd.mom + node, q, radius, 0.0, 0.0, r);
    if (r == 0) {
      nd.fifo[node] = (((last >> 48) + 1ull) << 48) | (last & ((1ull << 48) - 1ull));
      nd.count[node] = cnt;
    }
    const int parent = nd.parent[node];
    if (parent < 0) return;
    __threadfence();
    __syncwarp(gm);
    int go = 0;
    if (r == 0) {
      if (atomicAdd(nd.arrived + parent, 1) + 1 == nd.npend[parent]) {
        nd.arrived[parent] = 0;  // ready for the next upward pass over this tree
        go = 1;
      }
    }
    if (!__shfl_sync(gm, go, 0, 8)) return;
    __threadfence();
    node = parent;
    c0 = nd.first_child[node];
  }
}

__global__ void __launch_bounds__(256) finalize_records(Nodes nd, int64_t nnodes, double gfac, int want_f32) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nnodes) return;
  const Mom q = nd.mom[i];
  WalkRec w;
  w.cm[0] = q.cm[0]; w.cm[1] = q.cm[1]; w.cm[2] = q.cm[2];
  w.type = nd.type[i];
  if (w.type == kTypeLeaf) {
    w.reach = q.reach;
    w.soft_max = q.soft_max;
  } else {
    w.orsq = q.radius * q.radius * gfac;  // GravityVisitor::open, :164
    w.soft = q.soft;
  }
  w.first_child = nd.first_child[i];
  w.count = nd.count[i];
  w.pstart = nd.pstart[i];
  w.pcount = nd.pcount[i];
  w.pad = 0;
  nd.walk[i] = w;
  if (i >= 1) {
    nd.walks[walk_sib_index(i, 0)] = make_double2(w.cm[0], w.cm[1]);
    nd.walks[walk_sib_index(i, 1)] = make_double2(w.cm[2], w.orsq);
    nd.walks[walk_sib_index(i, 2)] = make_double2(w.soft, __hiloint2double((min(w.count, 1 << 27) << 3) | w.type, w.first_child));
  }
  QuadRec r;
  r.mass = q.mass; r.soft = q.soft;
  r.xx = q.xx; r.xy = q.xy; r.xz = q.xz; r.yy = q.yy; r.yz = q.yz; r.zz = q.zz;
  nd.quad[i] = r;
  if (want_f32) {
    QuadRecF rf;
    rf.mass = (float)q.mass; rf.soft = (float)q.soft;
    rf.xx = (float)q.xx; rf.xy = (float)q.xy; rf.xz = (float)q.xz;
    rf.yy = (float)q.yy; rf.yz = (float)q.yz; rf.zz = (float)q.zz;
    nd.quadf[i] = rf;
  }
}

// ---------------------------------------------------------------- traversal
// One warp per bucket.  The reference fixes the order in which each target adds
// its interactions, not the order in which the terms are computed, so a bucket's
// interactions are collected in walk order (up to 64 entries), their terms are
// computed for all targets by groups of lanes in parallel, and the sums then
// run over the entries in walk order:
//   terms  lane l of group l / nt is target l mod nt; the G = 32 / nt groups take
//          different entries.  A leaf's term is its own partial sum (the
//          reference's leaf() adds a leaf's pairs into a local first), in particle
//          order.  Leaves are taken by descending size, so the groups' loops are
//          of similar length; then quadrupole, then monopole nodes.
//   sums   the terms wait in shared memory as [entry][target][ax ay az pot]; lane
//          4 t + c adds component c of target t over the entries, in order.
// Bound by the FP64 pipe (45-80 operations per term, with the IEEE square roots
// and divisions) and by latency.  With one lane per target and nothing else (a
// bucket holds 4-10 particles, so 4-10 of 32 lanes worked) the 2^20 mixture took
// 84.8 ms and the 4096-particle Plummer 1.01 ms; this takes 27.6 and 0.6 ms.
//
// With fewer buckets than resident warps a pass takes as long as its longest
// bucket, so there the four warps of a CTA share one bucket (kTeam = 4): warp 0
// walks and adds the sums, and every warp computes the terms of a quarter of the
// collected entries.
constexpr int kTravWarps = 4;
constexpr int kF64Entries = 64;  // per warp
constexpr int kF64Ctas = 4;  // per SM: 128 registers; 5, 6 and 7 spill (35.8, 44 and 50 against 28.3 ms)
constexpr int kF64Terms = 256;  // (entry, target) terms held in shared memory, per warp
enum : int { kEntLeaf = 0, kEntQuad = 1, kEntMono = 2 };

template <int kTeam>
struct F64Work {
  double term[4 * kF64Terms * kTeam];
  BucketGeom geom;
  union {
    WalkSeg stack[kWalkStack];
    int32_t queue[kBfsQueue];  // basic-down order
  };
  int32_t ent[kF64Entries * kTeam];    // node | kind << 30, walk order
  int2 range[kF64Entries * kTeam];     // a leaf's first particle and count
  uint8_t order[kF64Entries * kTeam];  // a warp's entries by kind and size
  int cmd, t0, nt;                     // team: entries to evaluate (-1: leave) and their targets
  unsigned nsrc, npc;                  // source particles and nodes of the targets' entries
};

__device__ __forceinline__ void team_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kTravWarps * 32) : "memory"); }

// A particle's (x, y, z, m) record in one 256-bit load.
__device__ __forceinline__ double4 ld_src(const double4* p) {
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

template <int kTeam>
struct F64Eval {
  const TravParams* P;
  F64Work<kTeam>* w;
  int lane, nt, grp, G, cap, n;
  double xi, yi, zi, si;
  // sums of the (target, component) pairs lane + 32 h (4 t + c), and the
  // potential of those with c = 3
  double s[4], sp[4];
  int64_t lat;  // where the next list entry goes (recording)
  bool record;

  // The lane's target among the ntargets from t0 on.
  __device__ void targets(const TravParams& Q, F64Work<kTeam>& W, int t0, int ntargets, int l) {
    P = &Q;
    w = &W;
    lane = l;
    nt = ntargets;
    G = 32 / nt;
    grp = lane / nt;
    xi = yi = zi = si = 0.0;
    if (grp < G) {
      const int i = t0 + lane % nt;
      xi = Q.p.x[i];
      yi = Q.p.y[i];
      zi = Q.p.z[i];
      si = Q.p.soft[i];
    }
  }

  __device__ void begin(const TravParams& Q, F64Work<kTeam>& W, int t0, int ntargets, int l, int64_t rec) {
    targets(Q, W, t0, ntargets, l);
    cap = kTeam * min(kF64Entries, kF64Terms / nt);
    n = 0;
    record = rec >= 0;
    lat = rec;
    __syncwarp();
    if (lane == 0) {
      w->nsrc = w->npc = 0;
      if (kTeam > 1) {
        w->t0 = t0;
        w->nt = nt;
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 4; h++) {
      s[h] = sp[h] = 0.0;
      const int p = lane + 32 * h;
      if (Q.accumulate && p < 4 * nt) {  // later replica walks continue each particle's sums
        const int i = t0 + (p >> 2), c = p & 3;
        s[h] = c == 0 ? Q.p.ax[i] : c == 1 ? Q.p.ay[i] : c == 2 ? Q.p.az[i] : Q.p.potf[i];
        if (c == 3) sp[h] = Q.p.pot[i];
      }
    }
  }

  __device__ void store(int t0) {
    const Particles& q = P->p;
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int p = lane + 32 * h;
      if (p < 4 * nt) {
        const int i = t0 + (p >> 2), c = p & 3;
        double* const out = c == 0 ? q.ax : c == 1 ? q.ay : c == 2 ? q.az : q.potf;
        out[i] = s[h];
        if (c == 3) q.pot[i] = sp[h];
      }
    }
  }

  // Runs of terminals from the walk: children c0 + k, in child order.
  __device__ void emit(int c0, uint32_t pp, uint32_t pq, uint32_t pm, bool last) {
    const uint32_t run = pp | pq | pm;
    const int m = __popc(run);
    if (n + m > cap || last) flush();
    if (lane < 8 && ((run >> lane) & 1u)) {
      const int kind = ((pp >> lane) & 1u) ? kEntLeaf : ((pq >> lane) & 1u) ? kEntQuad : kEntMono;
      const int at = __popc(run & ((1u << lane) - 1u));
      w->ent[n + at] = (c0 + lane) | (kind << 30);
      if (record) {
        P->list_node[lat + at] = c0 + lane;
        P->list_kind[lat + at] = (int8_t)kind;
      }
    }
    lat += m;
    n += m;
  }

  // One entry of a recorded list.
  __device__ void push(int node, int kind) {
    if (n == cap) flush();
    if (lane == 0) w->ent[n] = node | (kind << 30);
    ++n;
  }

  // GravityVisitor::leaf, examples/GravityVisitor.h:144-160, over sn particles
  // from s0 on
  __device__ __forceinline__ void leaf_term(int s0, int sn, double v[4]) const {
    double pax = 0.0, pay = 0.0, paz = 0.0, ppf = 0.0;
    // two sources at a time: their chains of square root and division overlap,
    // the sums stay in particle order
    for (int j = 0; j < sn; j += 2) {
      const double4* rec = P->src + s0 + j;
      const double* so = P->p.soft + s0 + j;
      const bool two = j + 1 < sn;
      const double4 p = ld_src(rec), q = ld_src(two ? rec + 1 : rec);
      const double ph = so[0] + si, qh = so[two ? 1 : 0] + si;
      const double px = (p.x + P->ox) - xi, py = (p.y + P->oy) - yi, pz = (p.z + P->oz) - zi;
      const double qx = (q.x + P->ox) - xi, qy = (q.y + P->oy) - yi, qz = (q.z + P->oz) - zi;
      const double p2 = px * px + py * py + pz * pz, q2 = qx * qx + qy * qy + qz * qz;
      const double pr = sqrt(p2), qr = sqrt(q2);
      double pa = 1.0 / pr, qa = 1.0 / qr;
      double pb = pa * pa * pa, qb = qa * qa * qa;
      if (pr < ph || qr < qh) {
        if (p2 != 0) spline_f64(p2, ph, pa, pb);
        if (q2 != 0) spline_f64(q2, qh, qa, qb);
      }
      if (p2 != 0) {
        const double bm = pb * p.w;
        pax += px * bm;
        pay += py * bm;
        paz += pz * bm;
        ppf += -p.w * pa;
      }
      if (q2 != 0 && two) {
        const double bm = qb * q.w;
        pax += qx * bm;
        pay += qy * bm;
        paz += qz * bm;
        ppf += -q.w * qa;
      }
    }
    v[0] = pax;
    v[1] = pay;
    v[2] = paz;
    v[3] = ppf;
  }

  // GravityVisitor::node, examples/GravityVisitor.h:184-224 (non-HEXADECAPOLE)
  __device__ void quad_term(int node, double v[4]) const {
    const double2* wr = reinterpret_cast<const double2*>(P->walk + node);
    const double2 c01 = wr[0];
    const double cz = wr[1].x;
    const QuadRec q = P->quad[node];
    const double rx = (xi - c01.x) - P->ox;
    const double ry = (yi - c01.y) - P->oy;
    const double rz = (zi - cz) - P->oz;
    const double rsq = rx * rx + ry * ry + rz * rz;
    const double dir = 1.0 / sqrt(rsq);
    const double twoh = q.soft + si;
    double a, b, c, d;
    splineq_f64(dir, rsq, twoh, a, b, c, d);
    const double qx = q.xx * rx + q.xy * ry + q.xz * rz;
    const double qy = q.xy * rx + q.yy * ry + q.yz * rz;
    const double qz = q.xz * rx + q.yz * ry + q.zz * rz;
    const double qir = 0.5 * (qx * rx + qy * ry + qz * rz);
    const double tr = 0.5 * (q.xx + q.yy + q.zz);
    const double qir3 = b * q.mass + d * qir - c * tr;
    v[3] = -q.mass * a - c * qir + b * tr;
    v[0] = -qir3 * rx + c * qx;
    v[1] = -qir3 * ry + c * qy;
    v[2] = -qir3 * rz + c * qz;
  }

  // openSoftening held (decided in the walk): addGravity, :130-139
  __device__ void mono_term(int node, double v[4]) const {
    const WalkRec* wr = P->walk + node;
    const double mass = P->quad[node].mass;
    const double cx = wr->cm[0] + P->ox, cy = wr->cm[1] + P->oy, cz = wr->cm[2] + P->oz;
    const double dx = cx - xi, dy = cy - yi, dz = cz - zi;
    const double rsq = dx * dx + dy * dy + dz * dz;
    v[0] = v[1] = v[2] = v[3] = 0.0;
    if (rsq != 0) {
      const double f = mass / (rsq * sqrt(rsq));
      v[0] = dx * f;
      v[1] = dy * f;
      v[2] = dz * f;
      v[3] = -mass / sqrt(rsq);
    }
  }

  // The terms of the entries [e0, e1) (at most kF64Entries), by one warp.
  __device__ __forceinline__ void terms(int e0, int e1) {
    // kinds and leaf sizes of this lane's two entries
    int key[2];
    unsigned src = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int e = e0 + lane + 32 * h;
      key[h] = -1;
      if (e < e1) {
        const int x = w->ent[e], kind = (unsigned)x >> 30;
        if (kind == kEntLeaf) {
          const int4 r = *reinterpret_cast<const int4*>(&P->walk[x].count);  // count, pstart, pcount, pad
          w->range[e] = make_int2(r.y, r.z);
          src += (unsigned)r.z;
          key[h] = 1 + r.z;
        } else {
          key[h] = kind == kEntQuad ? 1 : 0;
        }
      }
    }
    const int m = e1 - e0;
    const int nnode = __popc(__ballot_sync(kFull, key[0] == 1 || key[0] == 0)) +
                      __popc(__ballot_sync(kFull, key[1] == 1 || key[1] == 0));
    const int nleaf = m - nnode;
    src = __reduce_add_sync(kFull, src);
    if (lane == 0) {
      if (kTeam > 1) {
        atomicAdd(&w->nsrc, src);
        atomicAdd(&w->npc, (unsigned)nnode);
      } else {
        w->nsrc += src;
        w->npc += (unsigned)nnode;
      }
    }
    // entries by descending key: one round per distinct key
    uint8_t* const order = w->order + e0;
    {
      const unsigned lt = (1u << lane) - 1u;
      int done = 0;
      int k0 = key[0], k1 = key[1];
      while (done < m) {
        const int top = __reduce_max_sync(kFull, max(k0, k1));
        const unsigned m0 = __ballot_sync(kFull, k0 == top), m1 = __ballot_sync(kFull, k1 == top);
        if (k0 == top) {
          order[done + __popc(m0 & lt)] = (uint8_t)(e0 + lane);
          k0 = -1;
        }
        if (k1 == top) {
          order[done + __popc(m0) + __popc(m1 & lt)] = (uint8_t)(e0 + lane + 32);
          k1 = -1;
        }
        done += __popc(m0) + __popc(m1);
      }
    }
    __syncwarp();
    if (grp < G) {
      const int t = lane % nt;
      int k = grp;
      for (; k < nleaf; k += G) {
        const int e = order[k];
        double v[4];
        leaf_term(w->range[e].x, w->range[e].y, v);
        double2* o = reinterpret_cast<double2*>(w->term + 4 * (e * nt + t));
        o[0] = make_double2(v[0], v[1]);
        o[1] = make_double2(v[2], v[3]);
      }
      for (; k < m; k += G) {
        const int e = order[k], x = w->ent[e];
        double v[4];
        if (((unsigned)x >> 30) == kEntQuad) quad_term(x & 0x3fffffff, v);
        else mono_term(x & 0x3fffffff, v);
        double2* o = reinterpret_cast<double2*>(w->term + 4 * (e * nt + t));
        o[0] = make_double2(v[0], v[1]);
        o[1] = make_double2(v[2], v[3]);
      }
    }
    __syncwarp();
  }

  // A team's share of n entries: those of warp q.
  __device__ __forceinline__ void share(int n_, int q) {
    const int per = (n_ + kTeam - 1) / kTeam, e0 = min(n_, q * per);
    terms(e0, min(n_, e0 + per));
  }

  // Evaluate the collected entries and add them to the sums (team: by warp 0,
  // whose threads alone hold the sums).
  __device__ void flush() {
    __syncwarp();
    if (kTeam > 1) {
      if (lane == 0) w->cmd = n;
      __syncwarp();
      team_barrier();
      share(n, 0);
      team_barrier();
    } else {
      terms(0, n);
    }
    const int per = 4 * nt;
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int p = lane + 32 * h;
      if (32 * h < per && p < per) {
        double a = s[h], b = sp[h];
        const double* v = w->term + p;
#pragma unroll 4
        for (int e = 0; e < n; e++, v += per) {
          const double t = *v;
          a += t;
          if (((unsigned)w->ent[e] >> 30) == kEntQuad) b += t;  // pot: quadrupole node() terms only
        }
        s[h] = a;
        sp[h] = b;
      }
    }
    n = 0;
    __syncwarp();
  }

  // The other warps of a team: evaluate shares until warp 0 sends them away.
  __device__ void help(const TravParams& Q, F64Work<kTeam>& W, int q, int l) {
    int last_t0 = -1;
    while (true) {
      team_barrier();
      const int m = *(volatile int*)&W.cmd;
      if (m < 0) break;
      const int t0 = *(volatile int*)&W.t0;
      if (t0 != last_t0) {
        targets(Q, W, t0, *(volatile int*)&W.nt, l);
        last_t0 = t0;
      }
      share(m, q);
      team_barrier();
    }
  }
};

// The bucket's walk in the handle's order; its geometry stays in shared memory
// (the terms need the registers).
template <bool kBfs, class Work, class Sink>
__device__ __forceinline__ bool walk_one(const TravParams& P, Work& W, int lane, Sink& sink,
                                         unsigned long long& opens) {
  if constexpr (kBfs)
    return walk_bucket_bfs(P.walk, P.nnodes, W.geom, P.ox, P.oy, P.oz, W.queue, kBfsQueue, lane, sink, opens, P.status);
  else
    return walk_preorder(P.walk, P.walks, P.nnodes, W.geom, P.ox, P.oy, P.oz, W.stack, lane, sink, opens, P.status);
}

template <bool kBfs, int kTeam>
__global__ void __launch_bounds__(kTravWarps * 32, kF64Ctas) traverse_f64(TravParams P, const Mom* __restrict__ mom) {
  __shared__ F64Work<kTeam> works[kTravWarps / kTeam];
  F64Work<kTeam>& W = works[(threadIdx.x >> 5) / kTeam];
  const int lane = threadIdx.x & 31;
  if (kTeam > 1 && threadIdx.x >= 32) {
    F64Eval<kTeam> ev;
    ev.help(P, W, threadIdx.x >> 5, lane);
    return;
  }
  unsigned long long c_pp = 0, c_pc = 0, c_open = 0;
  while (true) {
    const unsigned bi = grab_bucket(P.work, P.smq, P.batch, lane);
    int64_t b = P.b_begin + (int64_t)bi;
    if (b >= P.b_end) break;
    const int tnode = P.buckets[b];
    if (tnode < 0 || tnode >= P.nnodes) {
      if (lane == 0) atomicOr(P.status, kErrCapacity);
      continue;
    }
    __syncwarp();
    if (lane == 0) load_bucket_geom(mom, tnode, W.geom);
    __syncwarp();
    const int tbase = P.walk[tnode].pstart, ntot = P.walk[tnode].pcount;
    if (P.mode == 1) {  // count the interaction list only
      ListCounter rec{0};
      if (!walk_one<kBfs>(P, W, lane, rec, c_open) && lane == 0) atomicOr(P.status, kErrStack);
      if (lane == 0) P.list_count[b - P.b_begin] = rec.n;
      continue;
    }
    // A bucket holds more than 32 particles only when more than `bucket`
    // particles share one 63-bit key (depth-21 leaf); its targets are then
    // walked in chunks of 32 (the decisions depend on the bucket only).
    for (int tc = 0; tc < ntot; tc += 32) {
      const int t0 = tbase + tc, nt = min(32, ntot - tc);
      unsigned long long opens = 0;
      F64Eval<kTeam> ev;
      ev.begin(P, W, t0, nt, lane, P.mode == 2 && tc == 0 ? P.list_off[b - P.b_begin] : -1);
      if (!walk_one<kBfs>(P, W, lane, ev, opens) && lane == 0) atomicOr(P.status, kErrStack);
      ev.store(t0);
      if (tc == 0) c_open += opens;
      const unsigned long long pp = (unsigned long long)W.nsrc * (unsigned long long)nt;
      const unsigned long long pc = (unsigned long long)W.npc * (unsigned long long)nt;
      c_pp += pp;
      c_pc += pc;
      if (P.bucket_work && lane == 0) {  // this chunk's interactions, added to the bucket's
        unsigned long long wk = pp + pc;
        if (tc > 0 || P.accumulate) wk += P.bucket_work[b];
        P.bucket_work[b] = wk;
      }
    }
  }
  if (lane == 0) {
    atomicAdd(&P.counters[0], c_pp);
    atomicAdd(&P.counters[1], c_pc);
    atomicAdd(&P.counters[2], c_open);
  }
  if (kTeam > 1) {
    if (lane == 0) W.cmd = -1;
    __syncwarp();
    team_barrier();
  }
}

// Frozen-list replay: evaluates each bucket's recorded interaction list (in the
// recorded order, i.e. the walk's) with the FP64 evaluator, without walking.
// Used to differentiate the force pass for a fixed interaction list.
__global__ void __launch_bounds__(kTravWarps * 32, kF64Ctas) replay_f64(TravParams P) {
  __shared__ F64Work<1> works[kTravWarps];
  const int lane = threadIdx.x & 31;
  while (true) {
    const unsigned bi = grab_bucket(P.work, P.smq, P.batch, lane);
    const int64_t b = P.b_begin + (int64_t)bi;
    if (b >= P.b_end) break;
    const int tnode = P.buckets[b];
    const int tbase = P.walk[tnode].pstart, ntot = P.walk[tnode].pcount;
    const int64_t e0 = P.list_off[b - P.b_begin], e1 = P.list_off[b - P.b_begin + 1];
    for (int tc = 0; tc < ntot; tc += 32) {
      const int t0 = tbase + tc, nt = min(32, ntot - tc);
      F64Eval<1> ev;
      ev.begin(P, works[threadIdx.x >> 5], t0, nt, lane, -1);
      for (int64_t e = e0; e < e1; e++) {
        const int node = P.list_node[e];
        const int kind = P.list_kind[e];
        if (node < 0 || node >= P.nnodes) {
          if (lane == 0) atomicOr(P.status, kErrCapacity);
          continue;
        }
        ev.push(node, kind == 0 ? kEntLeaf : kind == 2 ? kEntMono : kEntQuad);
      }
      ev.flush();
      ev.store(t0);
    }
  }
}

// ---------------------------------------------------------------- integrate
// src/Particle.C:7-9 (kick) then :11-21 (perturb) for the same dt.
__global__ void __launch_bounds__(256) kick_perturb(Particles p, int64_t n, double dt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double ax = p.ax[i], ay = p.ay[i], az = p.az[i];
    double vx = p.vx[i], vy = p.vy[i], vz = p.vz[i];
    vx += ax * dt / 2;
    vy += ay * dt / 2;
    vz += az * dt / 2;
    vx += (ax * dt / 2);
    vy += (ay * dt / 2);
    vz += (az * dt / 2);
    p.x[i] += (vx * dt);
    p.y[i] += (vy * dt);
    p.z[i] += (vz * dt);
    p.vx[i] = vx;
    p.vy[i] = vy;
    p.vz[i] = vz;
  }
}

// Leapfrog halves: kick (v += a dt/2) and drift (x += v dt).
__global__ void __launch_bounds__(256) kick_half(Particles p, int64_t n, double dt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    p.vx[i] += p.ax[i] * dt / 2;
    p.vy[i] += p.ay[i] * dt / 2;
    p.vz[i] += p.az[i] * dt / 2;
  }
}
__global__ void __launch_bounds__(256) drift(Particles p, int64_t n, double dt) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    p.x[i] += (p.vx[i] * dt);
    p.y[i] += (p.vy[i] * dt);
    p.z[i] += (p.vz[i] * dt);
  }
}

// ---------------------------------------------------------------- direct sum
constexpr int kDirTile = 256;

__global__ void __launch_bounds__(kDirTile) direct_sum_f64(const double* __restrict__ x, const double* __restrict__ y,
                                                           const double* __restrict__ z, const double* __restrict__ m,
                                                           const double* __restrict__ soft, int64_t n,
                                                           const int32_t* __restrict__ tgt, int64_t nt, int nsplit,
                                                           double* __restrict__ part) {
  // grid: (target blocks, nsplit source slices); part[(slice * nt + t) * 4 + k]
  __shared__ double sx[kDirTile], sy[kDirTile], sz[kDirTile], sm[kDirTile], ss[kDirTile];
  int64_t t = blockIdx.x * (int64_t)kDirTile + threadIdx.x;
  bool ok = t < nt;
  int i = ok ? tgt[t] : 0;
  double xi = x[i], yi = y[i], zi = z[i], si = soft[i];
  double ax = 0.0, ay = 0.0, az = 0.0, pp = 0.0;
  int64_t per = (n + nsplit - 1) / nsplit;
  int64_t j0 = per * blockIdx.y, j1 = min(n, j0 + per);
  for (int64_t base = j0; base < j1; base += kDirTile) {
    __syncthreads();
    int64_t j = base + threadIdx.x;
    if (j < j1) { sx[threadIdx.x] = x[j]; sy[threadIdx.x] = y[j]; sz[threadIdx.x] = z[j]; sm[threadIdx.x] = m[j]; ss[threadIdx.x] = soft[j]; }
    __syncthreads();
    int cnt = (int)min((int64_t)kDirTile, j1 - base);
    for (int k = 0; k < cnt; k++) {
      double dx = sx[k] - xi, dy = sy[k] - yi, dz = sz[k] - zi;
      double rsq = dx * dx + dy * dy + dz * dz;
      if (rsq != 0) {
        double a, b;
        spline_f64(rsq, ss[k] + si, a, b);
        double bm = b * sm[k];
        ax += dx * bm;
        ay += dy * bm;
        az += dz * bm;
        pp += -sm[k] * a;
      }
    }
  }
  if (ok) {
    double* o = part + ((int64_t)blockIdx.y * nt + t) * 4;
    o[0] = ax; o[1] = ay; o[2] = az; o[3] = pp;
  }
}

// ---------------------------------------------------------------- launchers
static inline unsigned blocks_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

void launch_leaf_moments(Nodes nd, const int32_t* buckets, int64_t nbuckets, Particles p, double4* src,
                         cudaStream_t st) {
  if (nbuckets > 0) { note_launch(); leaf_moments<<<blocks_for(4 * nbuckets), 256, 0, st>>>(nd, buckets, nbuckets, p, src); }
}
void launch_upward(Nodes nd, int64_t ninternal, cudaStream_t st) {
  if (ninternal > 0) { note_launch(); upward_climb<<<blocks_for(8 * ninternal, kClimbThreads), kClimbThreads, 0, st>>>(nd, ninternal); }
}
void launch_finalize(Nodes nd, int64_t nnodes, double gfac, int want_f32, cudaStream_t st) {
  if (nnodes > 0) { note_launch(); finalize_records<<<blocks_for(nnodes), 256, 0, st>>>(nd, nnodes, gfac, want_f32); }
}
void launch_traverse_f64(const TravParams& P, const Mom* mom, int sms, cudaStream_t st) {
  const int grid = 16 * sms;
  note_launch();
  // Up to 24 buckets per SM (16 warps are resident), a CTA per bucket.  Plummer,
  // mixture and Hernquist spheres, buckets of 16, at 4,000 / 10,000 particles:
  // 0.65-0.72 -> 0.32-0.34 and 0.85-1.19 -> 0.68-0.86 ms (0.22 -> 0.13 and 0.41 ->
  // 0.32 the mixture); from 27 per SM on within 5% either way, and at 52 a warp
  // per bucket is the better one by a third.
  const bool team = P.mode != 1 && P.b_end - P.b_begin <= (int64_t)24 * sms;
  const int threads = kTravWarps * 32;
  if (P.bfs) {
    if (team) traverse_f64<true, kTravWarps><<<grid, threads, 0, st>>>(P, mom);
    else traverse_f64<true, 1><<<grid, threads, 0, st>>>(P, mom);
  } else {
    if (team) traverse_f64<false, kTravWarps><<<grid, threads, 0, st>>>(P, mom);
    else traverse_f64<false, 1><<<grid, threads, 0, st>>>(P, mom);
  }
}
void launch_replay_f64(const TravParams& P, int grid, cudaStream_t st) {
  note_launch();
  replay_f64<<<grid, kTravWarps * 32, 0, st>>>(P);
}
void launch_kick_perturb(Particles p, int64_t n, double dt, int grid, cudaStream_t st) {
  note_launch();
  kick_perturb<<<grid, 256, 0, st>>>(p, n, dt);
}
void launch_kick_half(Particles p, int64_t n, double dt, int grid, cudaStream_t st) {
  note_launch();
  kick_half<<<grid, 256, 0, st>>>(p, n, dt);
}
void launch_drift(Particles p, int64_t n, double dt, int grid, cudaStream_t st) {
  note_launch();
  drift<<<grid, 256, 0, st>>>(p, n, dt);
}
void launch_direct_sum(const double* x, const double* y, const double* z, const double* m, const double* soft,
                       int64_t n, const int32_t* tgt, int64_t nt, int nsplit, double* part, cudaStream_t st) {
  dim3 grid(blocks_for(nt, kDirTile), nsplit);
  note_launch();
  direct_sum_f64<<<grid, kDirTile, 0, st>>>(x, y, z, m, soft, n, tgt, nt, nsplit, part);
}

}  // namespace pt
