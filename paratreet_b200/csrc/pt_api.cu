// pt_api.cu -- the C ABI (include/pt_gravity.h): handle, device buffers and the
// per-pass orchestration of the kernels.
//
// One force pass (pt_compute_forces) runs, on the handle's stream:
//   K1 bbox + universe -> K2 keys -> K3 radix sort -> K4 permute
//   -> K5 octree build, all levels at once (+ bucket DFS order)
//   -> K6 leaf moments + upward pass + traversal records
//   -> K7 traversal (FP64 or mixed), optionally with interaction lists.
// The host reads back the tree's node counts (to size the node arrays) and the
// status word; everything else stays on the device.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/pt_gravity.h"
#include "pt_launch.h"

using namespace pt;

// What a pass writes for the host, and the counters' copy from before a list walk
// (restored if the walk is repeated with larger pools).
struct Words {
  unsigned long long counters[3], lcur[3], saved[3], list_total;
  unsigned status, ticket;
  uint32_t total[kMaxDepth + 1];
};

constexpr size_t kPage = 4096;

struct pt_handle {
  pt_config cfg{};
  std::string err;
  int sms = 148;
  cudaStream_t stream = nullptr;
  cudaStream_t own_stream = nullptr;

  int64_t alloc_limit = 0;  // largest device allocation (pt_set_alloc_limit; 0: no limit)
  int64_t n = 0, cap_n = 0;
  Particles p{};
  unsigned char* slab = nullptr;  // every per-particle array below, one allocation
  double* tmp[8]{};               // the other half of the permutation (free between passes)
  int32_t* tmp_i = nullptr;
  uint64_t* key_alt = nullptr;
  uint32_t *idx = nullptr, *idx_alt = nullptr;
  unsigned sort_tag = 1;  // the next sort's first look-back tag
  size_t sort_bytes = 0;
  unsigned char* sort_scratch = nullptr;  // onesweep histograms, tile counters, look-back words
  uint32_t* tree_counts = nullptr;  // per tile of particles: Internal nodes by level, leaves
  uint32_t* d_total = nullptr;      // their sums
  double* bbox_partial = nullptr;
  int bbox_blocks = 0;
  double* d_uni = nullptr;  // 12 doubles
  // small device words in one block (Words), so that one copy brings the host all
  // it reads back, into pinned memory
  Words* d_words = nullptr;
  Words* pin = nullptr;
  bool pinned = false;
  unsigned* d_status = nullptr;
  unsigned* d_ticket = nullptr;  // CTAs that finished the bounding box (0 between passes)
  unsigned long long* d_counters = nullptr;  // 3
  unsigned* d_work = nullptr;
  unsigned long long* d_vmax2 = nullptr;
  double4* src = nullptr;  // (x, y, z, m) per particle, sorted order (FP64 walk and replay)
  int64_t cap_src = 0;
  float4* srcf = nullptr;
  float* softf = nullptr;
  int64_t cap_srcf = 0;

  Nodes nd{};
  unsigned char* node_slab = nullptr;  // the node arrays, one allocation
  int64_t node_cap = 0, nnodes = 0, ninternal = 0;
  int depth = 0;  // deepest level of the tree
  int32_t* buckets = nullptr;
  unsigned long long* bucket_work = nullptr;  // interactions per bucket of the last pass
  int64_t nbuckets = 0, cap_buckets = 0;

  int64_t* list_count = nullptr;
  int64_t* list_off = nullptr;
  int32_t* list_node = nullptr;
  int8_t* list_kind = nullptr;
  int64_t list_total = 0, list_cap = 0, list_nb = 0;  // list_nb = recorded buckets + 1
  int64_t list_off_cap = 0;                              // entries of list_count / list_off
  bool lists_valid = false;
  bool tp_lists_valid = false;  // the two-phase pools hold the last pass's lists of every bucket

  double* dsum = nullptr;  // direct-sum scratch (caller-order copies + partials)
  int64_t dsum_cap = 0;

  // two-phase mixed traversal: list pools and per-bucket list descriptors
  bool two_phase = true;  // PT_MIXED_FUSED=1 selects the fused walk + evaluate kernel
  int32_t *pool_pc = nullptr, *pool_pp = nullptr;
  unsigned long long cap_pc = 0, cap_pp = 0;    // allocated entries of each pool
  bool pool_reps = false;       // ... with a byte per entry behind them
  int rep_batch = kMaxReps;     // replicas a mixed periodic pass takes in one batch
  unsigned long long want_pc = 0, want_pp = 0;  // entries the next pass should have
  int64_t *l_pc_start = nullptr, *l_pp_start = nullptr;
  int32_t *l_pc_count = nullptr, *l_pp_count = nullptr;
  int64_t l_nb_cap = 0;
  unsigned long long* d_lcur = nullptr;  // [0] P2C cursor, [1] P2P cursor, [2] longest list
  unsigned long long* d_queue = nullptr;  // bucket queues (kQueueWords each) of up to three kernels
  unsigned l_region = 32768;  // entries per warp region of the list pools

  double* sph = nullptr;  // SPH density pass: density, ball^2 (2n), neighbours (k n int32 + k n double)
  int64_t sph_cap = 0, sph_nbr_cap = 0;
  int32_t* sph_nbr = nullptr;
  double* sph_nd2 = nullptr;
  double* sph_list_d = nullptr;  // neighbour-search scratch: per-warp lists
  int32_t* sph_list_i = nullptr;
  int64_t sph_list_cap = 0;
  double* sph_state = nullptr;  // SPH step: u, u_pred, v_pred (caller order, 5 N), sorted v_pred (3 N)
  int64_t sph_state_cap = 0;

  double4* d_htab = nullptr;  // Ewald reciprocal table (h vector, hCfac)
  int64_t htab_cap = 0;
  double* ewd = nullptr;  // Ewald direct-sum scratch
  int64_t ewd_cap = 0;

  cudaEvent_t ev[7]{};
  long long sort_spin_limit = 1LL << 21;  // pt_set_sort_spin_limit
  pt_counters last{};
  double last_dt = 0.0;
  bool have_forces = false;     // a force pass ran since the particles were set
  bool forces_current = false;  // ... and the positions have not moved since
  bool keys_valid = false;      // the keys are sorted and line up with the particles
  bool trav_range_partial = false;

  double* adj = nullptr;  // adjoint scratch: cotangent (3N) and gradients (4N), sorted + caller order,
                          // then pt_adjoint's caller-order input and output (7N)
  int64_t adj_cap = 0;
  double* chain = nullptr;  // pt_chain_grad's states and checkpoints
  int64_t chain_cap = 0;
  double* nadj = nullptr;  // 10 adjoint values per node
  int64_t nadj_cap = 0;
};

namespace pt {
namespace {

// Scratch owned by one call (freed on every return path).
struct DevBuf {
  double* p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
};
std::atomic<unsigned long long> g_launches{0};
}
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
unsigned long long launches_so_far() { return g_launches.load(std::memory_order_relaxed); }
}  // namespace pt

namespace {

// A bucket queue: the global counter's word, then 256 words of per-SM batches.
constexpr int kQueueWords = 257;

void use_queue(pt_handle* h, TravParams& P, int k) {
  P.work = reinterpret_cast<unsigned*>(h->d_queue + k * kQueueWords);
  P.smq = h->d_queue + k * kQueueWords + 1;
}

// Buckets per batch of an SM: 32, or less where the SMs would not each see a
// few batches.  A batch belongs to its SM: with 32 for 2112 buckets, 66 SMs took
// everything, one warp each (the others had found the counter at its end and
// left), and the walk of the 10,000-particle Plummer took 391 us.
unsigned bucket_batch(const pt_handle* h, int64_t nb) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(32, nb / ((int64_t)h->sms * 64)));
}

int fail(pt_handle* h, int code, const std::string& msg) {
  if (h) h->err = msg;
  return code;
}

#define CK(call)                                                                               \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) {                                                                   \
      cudaGetLastError(); /* or the next launch's check reports this error again */            \
      return fail(h, (e_ == cudaErrorMemoryAllocation) ? PT_E_NOMEM : PT_E_CUDA,               \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                         \
    }                                                                                          \
  } while (0)

#define CKR(expr)              \
  do {                         \
    int r_ = (expr);           \
    if (r_ != PT_OK) return r_; \
  } while (0)

// cudaMalloc within the handle's limit.
template <typename T>
cudaError_t device_malloc(const pt_handle* h, T** ptr, size_t bytes) {
  // a refused allocation asks for more than any device has, so that the runtime's
  // error state is that of a failed call
  if (h->alloc_limit > 0 && bytes > (size_t)h->alloc_limit) bytes = (size_t)1 << 62;
  return cudaMalloc((void**)ptr, bytes);
}

template <typename T>
int dalloc(pt_handle* h, T** ptr, size_t count) {
  if (*ptr) {
    cudaFree(*ptr);
    *ptr = nullptr;
  }
  if (count == 0) count = 1;
  CK(device_malloc(h, ptr, count * sizeof(T)));
  return PT_OK;
}

// Room for `need` elements in each of the arrays that share the capacity `cap`,
// with `want` of them where they are allocated anew and that fits.  The old arrays
// go first, so the capacity is 0 until all of the new ones are there: after a refused
// allocation the next call allocates again instead of using a null array.
template <typename... T>
int reserve(pt_handle* h, int64_t& cap, int64_t need, int64_t want, T**... arrays) {
  if (need <= cap) return PT_OK;
  cap = 0;
  int rc = PT_OK;
  for (const int64_t count : {std::max(need, want), need}) {
    (void)(((rc = dalloc(h, arrays, (size_t)count)) == PT_OK) && ...);
    if (rc == PT_OK) cap = count;
    if (rc != PT_E_NOMEM || count == need) break;
  }
  return rc;
}

int zero_queue(pt_handle* h) {
  CK(cudaMemsetAsync(h->d_queue, 0, kQueueWords * sizeof(unsigned long long), h->stream));
  return PT_OK;
}

template <typename T>
void dfree(T*& ptr) {
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
}

int grid_for(const pt_handle* h, int64_t n) {
  int64_t g = (n + 255) / 256;
  int64_t cap = (int64_t)h->sms * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

int ensure_particles(pt_handle* h, int64_t n) {
  if (n <= h->cap_n && h->p.x) return PT_OK;
  const int64_t c = (std::max<int64_t>(n, 1) + 31) / 32 * 32;  // every array starts on a 128-byte boundary
  h->cap_n = h->n = 0;
  h->have_forces = h->forces_current = h->lists_valid = false;
  h->p = Particles{};
  const size_t sort_bytes = (sort_scratch_bytes(c) + 255) / 256 * 256;
  const size_t count_bytes = ((size_t)tree_columns() * tree_tiles(c) * sizeof(uint32_t) + 255) / 256 * 256;
  CKR(dalloc(h, &h->slab, (size_t)c * (21 * 8 + 2 * 8 + 4 * 4) + sort_bytes + count_bytes));
  unsigned char* at = h->slab;
  auto take = [&](auto** ptr, size_t bytes) {
    *ptr = reinterpret_cast<std::remove_reference_t<decltype(*ptr)>>(at);
    at += bytes;
  };
  h->sort_scratch = at;
  at += sort_bytes;
  take(&h->tree_counts, count_bytes);
  double** dbl[] = {&h->p.y, &h->p.z, &h->p.vx, &h->p.vy, &h->p.vz, &h->p.m, &h->p.soft,
                    &h->p.ax, &h->p.ay, &h->p.az, &h->p.pot, &h->p.potf};
  for (auto pp : dbl) take(pp, c * sizeof(double));
  for (auto& t : h->tmp) take(&t, c * sizeof(double));
  take(&h->p.order, c * sizeof(int32_t));
  take(&h->tmp_i, c * sizeof(int32_t));
  take(&h->p.key, c * sizeof(uint64_t));
  take(&h->key_alt, c * sizeof(uint64_t));
  take(&h->idx, c * sizeof(uint32_t));
  take(&h->idx_alt, c * sizeof(uint32_t));
  take(&h->p.x, c * sizeof(double));
  CK(cudaMemsetAsync(h->sort_scratch, 0, sort_bytes, h->stream));
  h->sort_tag = 1;
  h->sort_bytes = sort_bytes;
  h->cap_n = c;
  return PT_OK;
}

// Room for `need` nodes; the arrays hold nothing that outlives a build.  One
// allocation for all of them: a new handle's first pass made 17 here.
int grow_nodes(pt_handle* h, int64_t need) {
  if (need <= h->node_cap) return PT_OK;
  const int64_t nc = std::max<int64_t>(need + need / 4, 1024);
  Nodes o{};
  size_t bytes = 0;
  unsigned char* base = nullptr;  // null: count the bytes
  auto take = [&](auto** ptr, size_t count) {
    if (base) *ptr = reinterpret_cast<std::remove_reference_t<decltype(*ptr)>>(base + bytes);
    bytes += (count * sizeof(**ptr) + 255) / 256 * 256;
  };
  auto take_all = [&]() {
    bytes = 0;
    take(&o.mom, nc);
    take(&o.walk, nc);
    take(&o.walks, walk_sib_size(nc));
    take(&o.quad, nc);
    take(&o.quadf, nc);
    take(&o.inode, nc / 8 + 1);
    take(&o.key, nc);
    take(&o.fifo, nc);
    take(&o.type, nc);
    take(&o.depth, nc);
    take(&o.pstart, nc);
    take(&o.pcount, nc);
    take(&o.parent, nc);
    take(&o.first_child, nc);
    take(&o.count, nc);
    take(&o.npend, nc);
    take(&o.arrived, nc);
  };
  take_all();
  h->node_cap = 0;
  h->nd = Nodes{};
  CKR(dalloc(h, &h->node_slab, bytes));
  base = h->node_slab;
  take_all();
  h->nd = o;
  h->node_cap = nc;
  return PT_OK;
}

// The small words, as they stand after the work issued so far (synchronises).
int read_words(pt_handle* h) {
  CK(cudaMemcpyAsync(h->pin, h->d_words, sizeof(Words), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PT_OK;
}

// read_words and the status among them.
int read_status(pt_handle* h) {
  CKR(read_words(h));
  const unsigned st = h->pin->status;
  if (st) {
    CK(cudaMemsetAsync(h->d_status, 0, sizeof(unsigned), h->stream));
    std::string m = "device status:";
    if (st & kErrNonFinite) m += " non-finite particle position;";
    if (st & kErrStack) m += " traversal stack overflow;";
    if (st & kErrCapacity) m += " capacity exceeded;";
    if (st & kErrAdjointSoftened) m += " adjoint met a softened quadrupole term (not differentiated);";
    if (st & kErrSort) m += " radix sort look-back timed out;";
    if (st & kErrPool) m += " interaction-list pools exhausted;";
    if (st & kErrSphNonFinite) m += " SPH pressure term not finite (a ball of zero radius: N = 1 or coincident particles);";
    return fail(h, (st & kErrNonFinite) ? PT_E_NONFINITE : PT_E_DEVICE, m);
  }
  return PT_OK;
}

// K1..K4: universe, keys, sort, permute.
int keys_and_sort(pt_handle* h) {
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  const int g = grid_for(h, n);
  h->keys_valid = false;
  launch_bbox(h->p.x, h->p.y, h->p.z, n, h->bbox_partial, h->bbox_blocks, h->d_ticket, h->d_uni, h->d_status, st);
  launch_keys(h->p.x, h->p.y, h->p.z, n, h->d_uni, h->p.key, h->idx, g, st);
  CK(cudaGetLastError());
  CK(cudaEventRecord(h->ev[1], st));
  if (h->sort_tag + 8 > sort_tags()) {
    CK(cudaMemsetAsync(h->sort_scratch, 0, h->sort_bytes, st));
    h->sort_tag = 1;
  }
  const int where = radix_sort_pairs(h->p.key, h->idx, h->key_alt, h->idx_alt, n, h->sort_scratch, h->d_status,
                                     h->sms, h->sort_spin_limit, h->sort_tag, st);
  if (where < 0) return fail(h, PT_E_CUDA, "radix sort: could not set the shared-memory attribute");
  h->sort_tag += 8;
  if (where == 1) {
    std::swap(h->p.key, h->key_alt);
    std::swap(h->idx, h->idx_alt);
  }
  // a look-back that gave up leaves indices that are not a permutation: the
  // permutation then leaves every particle where it is, and build_tree, which
  // reads the status word, stops the pass
  PermuteArrays A{};
  double** fields[] = {&h->p.x, &h->p.y, &h->p.z, &h->p.vx, &h->p.vy, &h->p.vz, &h->p.m, &h->p.soft};
  for (int f = 0; f < 8; f++) {
    A.in[f] = *fields[f];
    A.out[f] = h->tmp[f];
  }
  A.order_in = h->p.order;
  A.order_out = h->tmp_i;
  launch_permute(A, h->idx, n, h->d_status, g, st);
  for (int f = 0; f < 8; f++) std::swap(*fields[f], h->tmp[f]);
  std::swap(h->p.order, h->tmp_i);
  CK(cudaGetLastError());
  CK(cudaEventRecord(h->ev[2], st));
  return PT_OK;
}

// K5: octree build and bucket order.
int build_tree(pt_handle* h) {
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  launch_tree_count(h->p.key, n, h->cfg.bucket, h->tree_counts, h->d_total, st);
  CKR(read_status(h));  // synchronises; a failed sort ends the pass here
  // the particles are in a new order from here on: results of an earlier pass no
  // longer line up with it
  h->have_forces = h->forces_current = h->lists_valid = h->tp_lists_valid = false;
  h->keys_valid = true;
  const uint32_t* tot = h->pin->total;  // Internal nodes of each level, leaves
  int64_t ni = 0;
  int depth = 0;
  for (int l = 0; l < kMaxDepth; l++) {
    ni += tot[l];
    if (tot[l]) depth = l + 1;
  }
  const int64_t nl = tot[kMaxDepth];
  h->nnodes = h->nbuckets = 0;
  CKR(grow_nodes(h, 1 + 8 * ni));
  // an eighth of headroom: the bucket count drifts from pass to pass as the
  // particles move, and a cudaFree on every new maximum would stall the device
  CKR(reserve(h, h->cap_buckets, nl, nl + nl / 8 + 64, &h->buckets, &h->bucket_work));
  h->nnodes = 1 + 8 * ni;
  h->ninternal = ni;
  h->depth = depth;
  h->nbuckets = nl;
  launch_tree_emit(h->nd, h->p.key, n, h->cfg.bucket, h->tree_counts, h->d_total, ni, h->node_cap, nl, h->buckets,
                   h->d_status, st);
  CK(cudaGetLastError());
  CK(cudaEventRecord(h->ev[3], st));
  return PT_OK;
}

int ensure_src(pt_handle* h) { return reserve(h, h->cap_src, h->cap_n, h->cap_n, &h->src); }

// K6: moments, upward pass, traversal records.
int upward(pt_handle* h, bool walk = true) {
  cudaStream_t st = h->stream;
  // the FP64 walk reads source records (a mixed pass takes it only to record
  // lists, or where its list pools do not fit)
  const bool want_src = walk && (h->cfg.precision != PT_MIXED || h->cfg.record_lists);
  if (want_src) CKR(ensure_src(h));
  launch_leaf_moments(h->nd, h->buckets, h->nbuckets, h->p, want_src ? h->src : nullptr, st);
  launch_upward(h->nd, h->ninternal, st);
  const double gfac = (4.0 / 3.0) / (h->cfg.theta * h->cfg.theta);  // GravityVisitor.h:14,18
  const int mixed = h->cfg.precision == PT_MIXED;
  launch_finalize(h->nd, h->nnodes, gfac, mixed, st);
  if (mixed) {
    CKR(reserve(h, h->cap_srcf, h->cap_n, h->cap_n, &h->srcf, &h->softf));
    launch_prep_sources(h->buckets, h->nbuckets, h->nd.walk, h->p, h->srcf, h->softf, st);
  }
  CK(cudaGetLastError());
  CK(cudaEventRecord(h->ev[4], st));
  return PT_OK;
}

// The Ewald correction of a periodic pass (examples/Gravity.C:45-48 calls
// LeafEwaldFn on every leaf after the replica walks).  The host builds the
// reciprocal table from the root's moments as EwaldData::EwaldInit does
// (examples/Ewald.C:80-163, QEVAL at (hx, hy, hz) with the odd gamma terms
// zeroed: hCfac = -g2 Qmir - g0 M, hSfac = 0), then one thread per particle of
// the buckets [b0, b1) adds the real-space and reciprocal sums.
int ewald_correction_pass(pt_handle* h, int64_t b0, int64_t b1) {
  cudaStream_t st = h->stream;
  Mom root;
  CK(cudaMemcpyAsync(&root, h->nd.mom, sizeof(Mom), cudaMemcpyDeviceToHost, st));
  int32_t pb[2] = {0, 0};
  int32_t pe[2] = {0, 0};
  if (b1 > b0) {
    int32_t nb0 = 0, nb1 = 0;
    CK(cudaMemcpyAsync(&nb0, h->buckets + b0, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&nb1, h->buckets + (b1 - 1), sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    CK(cudaMemcpyAsync(pb, &h->nd.walk[nb0].pstart, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(pe, &h->nd.walk[nb1].pstart, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  }
  CK(cudaStreamSynchronize(st));
  const double L = h->cfg.period;
  const double hcut = h->cfg.ewald_hcut;
  const int hReps = (int)std::ceil(hcut);
  const double alpha = 2.0 / L;
  const double k4 = M_PI * M_PI / (alpha * alpha * L * L);
  std::vector<double4> tab;
  for (int hx = -hReps; hx <= hReps; ++hx)
    for (int hy = -hReps; hy <= hReps; ++hy)
      for (int hz = -hReps; hz <= hReps; ++hz) {
        const int h2 = hx * hx + hy * hy + hz * hz;
        if (h2 == 0) continue;
        if (h2 > hcut * hcut) continue;
        // h and -h have the same coefficient and add the same: the first of the
        // two in this order stands for both
        if (hx > 0 || (hx == 0 && (hy > 0 || (hy == 0 && hz > 0)))) continue;
        const double g0 = std::exp(-k4 * h2) / (M_PI * h2 * L);
        const double g1 = 2 * M_PI / L * g0;
        const double g2 = -2 * M_PI / L * g1;
        const double Qmirx = (1.0 / 1.0) * (root.xz * hz + root.xy * hy + root.xx * hx);
        const double Qmiry = (1.0 / 1.0) * (root.yz * hz + root.xy * hx + root.yy * hy);
        const double Qmirz = (1.0 / 1.0) * (root.yz * hy + root.xz * hx + root.zz * hz);
        const double Qmir = (1.0 / 2.0) * (Qmirx * hx + Qmiry * hy + Qmirz * hz);
        double mfacc = 0.0;
        mfacc -= g2 * Qmir;
        mfacc -= g0 * root.mass;
        tab.push_back(make_double4(2 * M_PI / L * hx, 2 * M_PI / L * hy, 2 * M_PI / L * hz, 2.0 * mfacc));
      }
  CKR(reserve(h, h->htab_cap, (int64_t)tab.size(), (int64_t)tab.size(), &h->d_htab));
  if (!tab.empty())
    CK(cudaMemcpyAsync(h->d_htab, tab.data(), tab.size() * sizeof(double4), cudaMemcpyHostToDevice, st));
  EwaldRoot R{};
  R.cm[0] = root.cm[0];
  R.cm[1] = root.cm[1];
  R.cm[2] = root.cm[2];
  R.mass = root.mass;
  R.xx = root.xx;
  R.xy = root.xy;
  R.xz = root.xz;
  R.yy = root.yy;
  R.yz = root.yz;
  R.zz = root.zz;
  R.L = L;
  R.rcut = h->cfg.ewald_rcut;
  R.n_replicas = h->cfg.n_replicas;
  R.n_h = (int)tab.size();
  const int64_t i0 = pb[0], i1 = (b1 > b0) ? (int64_t)pe[0] + pe[1] : i0;
  launch_ewald_correction(h->p, i0, i1, R, h->d_htab, st);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(st));  // the host table must outlive the copy
  return PT_OK;
}

// The offset of replica r in the order of the loop of examples/Gravity.C:35-41.
void replica_offset(const pt_handle* h, int r, TravParams& P) {
  const int nr = h->cfg.n_replicas, w = 2 * nr + 1;
  P.ox = (r / (w * w) - nr) * h->cfg.period;
  P.oy = (r / w % w - nr) * h->cfg.period;
  P.oz = (r % w - nr) * h->cfg.period;
}

// Two-phase mixed evaluation: walk_lists writes every bucket's interaction
// list to the pools, then eval_p2c2 and eval_p2p evaluate them.  Pools are
// sized from the previous pass with a quarter of headroom (a bucket whose list
// outgrows its warp's region moves it to a new region inside the walk); only
// a pass whose lists fill a pool is repeated (counters restored) with pools
// twice as large, which happens at most on the first passes of a handle.
constexpr int kFewerReplicas = 1;  // run_two_phase: no room for a batch's lists, h->rep_batch is smaller now
int run_two_phase(pt_handle* h, TravParams& P) {
  cudaStream_t st = h->stream;
  const int64_t nb = P.b_end - P.b_begin;
  if (nb <= 0) return PT_OK;
  if (nb > h->l_nb_cap) {
    const int64_t cap = nb + nb / 8 + 64;  // headroom, as for the bucket arrays
    h->l_nb_cap = 0;
    CKR(dalloc(h, &h->l_pc_start, 3 * cap));  // two arrays of starts, two of 32-bit counts
    h->l_pp_start = h->l_pc_start + cap;
    h->l_pc_count = reinterpret_cast<int32_t*>(h->l_pp_start + cap);
    h->l_pp_count = h->l_pc_count + cap;
    h->l_nb_cap = cap;
  }
  const int wgrid = (int)std::max<int64_t>(1, std::min<int64_t>(walk_lists_grid(h->sms), (nb + 3) / 4));
  CK(cudaMemcpyAsync(h->d_words->saved, h->d_counters, sizeof(h->d_words->saved), cudaMemcpyDeviceToDevice, st));
  auto restore_counters = [&]() {
    return cudaMemcpyAsync(h->d_counters, h->d_words->saved, sizeof(h->d_words->saved), cudaMemcpyDeviceToDevice, st);
  };
  auto fewer_replicas = [&]() {  // the lists of so many do not fit
    h->rep_batch = P.rep_count / 2;
    h->want_pc = h->want_pp = 0;
    return kFewerReplicas;
  };
  ListParams L{};
  for (int attempt = 0;; attempt++) {
    const unsigned region = h->l_region;
    const unsigned long long slack = (unsigned long long)wgrid * 4 * region;
    const unsigned long long need_pc =
        std::max<unsigned long long>(h->want_pc, 1024ull * nb + slack);
    const unsigned long long need_pp =
        std::max<unsigned long long>(h->want_pp, 256ull * nb + slack);
    // an entry, and where a batch has several replicas its replica (a byte)
    const bool reps = P.rep_count > 1;
    if (need_pc > h->cap_pc || need_pp > h->cap_pp || (reps && !h->pool_reps)) {
      // a quarter of headroom, so that the pass-to-pass variation of the
      // reserved regions does not free and map the multi-GB pools again
      // (which costs more than a whole pass); without room for it, the bare need
      dfree(h->pool_pc);
      dfree(h->pool_pp);
      h->cap_pc = h->cap_pp = 0;
      unsigned long long alloc_pc = need_pc + need_pc / 4, alloc_pp = need_pp + need_pp / 4;
      const size_t per = sizeof(int32_t) + (reps ? 1 : 0);
      if (device_malloc(h, &h->pool_pc, alloc_pc * per) != cudaSuccess ||
          device_malloc(h, &h->pool_pp, alloc_pp * per) != cudaSuccess) {
        cudaGetLastError();
        dfree(h->pool_pc);
        dfree(h->pool_pp);
        alloc_pc = need_pc;
        alloc_pp = need_pp;
      }
      if ((!h->pool_pc && device_malloc(h, &h->pool_pc, need_pc * per) != cudaSuccess) ||
          (!h->pool_pp && device_malloc(h, &h->pool_pp, need_pp * per) != cudaSuccess)) {
        cudaGetLastError();
        dfree(h->pool_pc);
        dfree(h->pool_pp);
        CK(restore_counters());
        if (reps) return fewer_replicas();
        // no room for the lists: this handle evaluates with the fused kernel from now on
        h->two_phase = false;
        CKR(zero_queue(h));
        if (h->cfg.precision == PT_FP64_LISTS) launch_traverse_f64(P, h->nd.mom, h->sms, st);
        else launch_traverse_mixed(P, h->nd.mom, h->sms * 16, st);
        CK(cudaGetLastError());
        return PT_OK;
      }
      h->cap_pc = alloc_pc;
      h->cap_pp = alloc_pp;
      h->pool_reps = reps;
    }
    L.pc_pool = h->pool_pc;
    L.pp_pool = h->pool_pp;
    if (reps) {
      L.pc_rep = reinterpret_cast<uint8_t*>(h->pool_pc + h->cap_pc);
      L.pp_rep = reinterpret_cast<uint8_t*>(h->pool_pp + h->cap_pp);
    }
    L.cursor = h->d_lcur;
    L.cap_pc = h->cap_pc;
    L.cap_pp = h->cap_pp;
    L.region = region;
    L.thresh = region / 8;
    L.pc_start = h->l_pc_start;
    L.pc_count = h->l_pc_count;
    L.pp_start = h->l_pp_start;
    L.pp_count = h->l_pp_count;
    L.max_len = reinterpret_cast<unsigned*>(h->d_lcur + 2);
    CK(cudaMemsetAsync(h->d_lcur, 0, 3 * sizeof(unsigned long long), st));
    CK(cudaMemsetAsync(h->d_queue, 0, 3 * kQueueWords * sizeof(unsigned long long), st));
    TravParams A = P;
    use_queue(h, A, 0);
    launch_walk_lists(A, L, h->nd.mom, wgrid, st);
    CK(cudaGetLastError());
    CKR(read_words(h));
    unsigned status = h->pin->status;
    const unsigned long long* cur = h->pin->lcur;
    // the cursors count reserved regions (also refused ones): at most the pool size is used
    const unsigned long long used_pc = std::min(cur[0], h->cap_pc), used_pp = std::min(cur[1], h->cap_pp);
    if (!(status & kErrPool)) {
      // next pass: room for this pass's regions and a sixteenth more (a pool is
      // allocated a quarter larger than asked for, so it serves the next passes
      // as it is: asking for a quarter more here made every handle's second pass
      // allocate again, 129 instead of 90 ms at N = 2^24)
      h->want_pc = std::max<unsigned long long>(h->want_pc, used_pc + used_pc / 16);
      h->want_pp = std::max<unsigned long long>(h->want_pp, used_pp + used_pp / 16);
      break;
    }
    if (attempt >= 6) return fail(h, PT_E_NOMEM, "interaction lists outgrow their pools");
    // repeat the walk with larger pools (the cursors under-count the need: warps
    // stop reserving once their pool is full)
    status &= ~kErrPool;
    CK(cudaMemcpyAsync(h->d_status, &status, sizeof(unsigned), cudaMemcpyHostToDevice, st));
    CK(restore_counters());
    if (attempt >= 6) return reps ? fewer_replicas() : fail(h, PT_E_NOMEM, "interaction lists outgrow their pools");
    h->want_pc = std::max(2 * h->cap_pc, cur[0] + cur[0] / 2);
    h->want_pp = std::max(2 * h->cap_pp, cur[1] + cur[1] / 2);
  }
  TravParams E = P;
  use_queue(h, E, 1);
  TravParams F = P;  // the P2P evaluation's
  use_queue(h, F, 2);
  if (h->cfg.precision == PT_FP64_LISTS) launch_eval_lists_f64(E, L, h->nd.mom, h->sms * 16, st, F.work);
  else launch_eval_lists(E, F, L, h->nd.mom, h->sms, st);
  CK(cudaGetLastError());
  h->tp_lists_valid = (P.b_begin == 0 && P.b_end == h->nbuckets && !h->cfg.periodic);
  return PT_OK;
}

int run_traversal(pt_handle* h, TravParams& P, int grid) {
  const bool lists_form = h->cfg.precision == PT_MIXED || h->cfg.precision == PT_FP64_LISTS;
  if (lists_form && P.mode == 0 && h->two_phase) return run_two_phase(h, P);
  if (h->cfg.precision == PT_MIXED && P.mode != 1)
    launch_traverse_mixed(P, h->nd.mom, grid, h->stream);
  else launch_traverse_f64(P, h->nd.mom, h->sms, h->stream);
  CK(cudaGetLastError());
  return PT_OK;
}

// CSR lists (list_off / list_node / list_kind, kinds 0 P2P, 1 quadrupole,
// 2 monopole) of every bucket from the two-phase pools of the pass just
// made: per bucket its P2P leaves, then its P2C nodes, in the two-phase
// walk's order.
int lists_from_pools(pt_handle* h) {
  cudaStream_t st = h->stream;
  const int64_t nb = h->nbuckets;
  CKR(reserve(h, h->list_off_cap, nb + 1, nb + nb / 8 + 64, &h->list_count, &h->list_off));
  // list_count is the scan's scratch here (the FP64 form's counting walk uses it)
  launch_list_offsets(h->l_pc_count, h->l_pp_count, nb, h->list_count, h->list_off, &h->d_words->list_total, st);
  CK(cudaGetLastError());
  CKR(read_words(h));
  h->list_total = (int64_t)h->pin->list_total;
  CKR(reserve(h, h->list_cap, h->list_total, h->list_total + h->list_total / 8, &h->list_node, &h->list_kind));
  launch_pools_to_csr(h->pool_pc, h->pool_pp, h->l_pc_start, h->l_pc_count, h->l_pp_start, h->l_pp_count, nb,
                      h->list_off, h->list_node, h->list_kind, st);
  CK(cudaGetLastError());
  h->list_nb = nb + 1;
  h->lists_valid = true;
  return PT_OK;
}

int traverse(pt_handle* h, int64_t b0, int64_t b1) {
  cudaStream_t st = h->stream;
  b0 = std::max<int64_t>(0, std::min(b0, h->nbuckets));
  b1 = std::max<int64_t>(b0, std::min(b1, h->nbuckets));
  h->trav_range_partial = !(b0 == 0 && b1 == h->nbuckets);
  if (h->trav_range_partial) {
    double* arrs[] = {h->p.ax, h->p.ay, h->p.az, h->p.pot, h->p.potf};
    for (auto a : arrs) CK(cudaMemsetAsync(a, 0, h->n * sizeof(double), st));
  }
  TravParams P{};
  P.p = h->p;
  P.walk = h->nd.walk;
  P.walks = h->nd.walks;
  P.quad = h->nd.quad;
  P.quadf = h->nd.quadf;
  P.srcf = h->srcf;
  P.src = h->src;
  P.softf = h->softf;
  P.buckets = h->buckets;
  P.b_begin = b0;
  P.b_end = b1;
  P.ox = P.oy = P.oz = 0.0;
  P.bucket_work = h->bucket_work;
  P.bfs = (h->cfg.traversal == PT_BASIC_DOWN) ? 1 : 0;
  if (h->nbuckets > 0) CK(cudaMemsetAsync(h->bucket_work, 0, h->nbuckets * sizeof(unsigned long long), st));
  P.nnodes = h->nnodes;
  P.counters = h->d_counters;
  P.status = h->d_status;
  use_queue(h, P, 0);
  P.batch = bucket_batch(h, b1 - b0);
  const int grid = h->sms * 16;
  CK(cudaMemsetAsync(h->d_counters, 0, 3 * sizeof(unsigned long long), st));
  const int64_t nb = b1 - b0;
  h->lists_valid = false;
  h->tp_lists_valid = false;
  // The two-phase forms record a full pass's lists from their own pools
  // (lists_from_pools, after the pass); the FP64 form records them in the
  // reference's walk order with a counting and a recording walk.
  const bool two_phase_record = h->cfg.record_lists && nb > 0 && h->two_phase && !h->cfg.periodic &&
                                b0 == 0 && b1 == h->nbuckets &&
                                (h->cfg.precision == PT_MIXED || h->cfg.precision == PT_FP64_LISTS);
  if (h->cfg.record_lists && nb > 0 && !two_phase_record) {
    CKR(reserve(h, h->list_off_cap, nb + 1, nb + 1, &h->list_count, &h->list_off));
    h->list_nb = nb + 1;
    P.mode = 1;
    P.list_count = h->list_count;
    CKR(zero_queue(h));
    CKR(run_traversal(h, P, grid));
    std::vector<int64_t> cnt(nb), off(nb + 1);
    CK(cudaMemcpyAsync(cnt.data(), h->list_count, nb * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    off[0] = 0;
    for (int64_t i = 0; i < nb; i++) off[i + 1] = off[i] + cnt[i];
    h->list_total = off[nb];
    CKR(reserve(h, h->list_cap, h->list_total, h->list_total, &h->list_node, &h->list_kind));
    CK(cudaMemcpyAsync(h->list_off, off.data(), (nb + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(h->d_counters, 0, 3 * sizeof(unsigned long long), st));
    P.mode = 2;
    P.list_off = h->list_off;
    P.list_node = h->list_node;
    P.list_kind = h->list_kind;
    if (h->cfg.precision == PT_MIXED || h->cfg.precision == PT_FP64_LISTS) {
      // lists come from the FP64 walk (identical for every form); then the two-phase pass
      P.mode = 2;
      CKR(zero_queue(h));
      launch_traverse_f64(P, h->nd.mom, h->sms, st);  // records lists (and FP64 forces)
      CK(cudaMemsetAsync(h->d_counters, 0, 3 * sizeof(unsigned long long), st));
      P.mode = 0;
    }
    h->lists_valid = true;
  } else {
    P.mode = 0;
  }
  CK(cudaEventRecord(h->ev[5], st));
  // examples/Gravity.C:32-46: one walk, or (2n+1)^3 replica walks with
  // GravityVisitor offsets (X, Y, Z) * L in that loop order; every walk after
  // the first continues each particle's sums
  const int nr = h->cfg.periodic ? h->cfg.n_replicas : 0;
  const int reps = (2 * nr + 1) * (2 * nr + 1) * (2 * nr + 1);
  // the mixed two-phase form takes the replicas in batches of up to kMaxReps, of
  // fewer where the lists of so many do not fit; the others one by one
  int per = 1;
  P.rep_n = nr;
  P.period = h->cfg.period;
  for (int r = 0; r < reps; r += per) {
    const bool lists_form = (h->cfg.precision == PT_MIXED || h->cfg.precision == PT_FP64_LISTS) && h->two_phase;
    per = h->cfg.precision == PT_MIXED && lists_form ? std::min(h->rep_batch, reps - r) : 1;
    if (h->cfg.periodic) replica_offset(h, r, P);
    P.rep_first = r;
    P.rep_count = reps > 1 && lists_form ? per : 0;
    P.accumulate = r > 0;
    CKR(zero_queue(h));
    const int rc = run_traversal(h, P, grid);
    if (rc == kFewerReplicas) per = 0;  // the same replicas again
    else CKR(rc);
  }
  if (h->cfg.periodic) CKR(ewald_correction_pass(h, b0, b1));
  CK(cudaEventRecord(h->ev[6], st));
  if (two_phase_record && h->tp_lists_valid) CKR(lists_from_pools(h));
  return PT_OK;
}

int forces(pt_handle* h, int64_t b0, int64_t b1) {
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles: call pt_set_particles first");
  const unsigned long long launches0 = launches_so_far();
  cudaStream_t st = h->stream;
  CK(cudaEventRecord(h->ev[0], st));
  if (h->n == 0) {
    h->nnodes = 0;
    h->nbuckets = 0;
    h->have_forces = true;
    h->forces_current = true;
    return PT_OK;
  }
  CKR(keys_and_sort(h));
  CKR(build_tree(h));
  CKR(upward(h));
  int rc = traverse(h, b0, b1);
  if (rc == PT_OK) rc = read_status(h);
  if (rc != PT_OK) {
    h->lists_valid = h->tp_lists_valid = false;
    return rc;
  }
  const unsigned long long* c = h->pin->counters;
  pt_counters& k = h->last;
  k.n_pp = c[0];
  k.n_pc = c[1];
  k.n_open = c[2];
  k.n_nodes = h->nnodes;
  k.n_buckets = h->nbuckets;
  k.depth = h->depth;
  k.launches = (int32_t)(launches_so_far() - launches0);
  CK(cudaEventElapsedTime(&k.ms_keys, h->ev[0], h->ev[1]));
  CK(cudaEventElapsedTime(&k.ms_sort, h->ev[1], h->ev[2]));
  CK(cudaEventElapsedTime(&k.ms_build, h->ev[2], h->ev[3]));
  CK(cudaEventElapsedTime(&k.ms_upward, h->ev[3], h->ev[4]));
  CK(cudaEventElapsedTime(&k.ms_traverse, h->ev[5], h->ev[6]));
  CK(cudaEventElapsedTime(&k.ms_total, h->ev[0], h->ev[6]));
  h->have_forces = true;
  h->forces_current = true;
  return PT_OK;
}

// examples/Gravity.C:63-67 with v_max from src/Subtree.h:164-170.
int timestep(pt_handle* h, double* dt) {
  cudaStream_t st = h->stream;
  CK(cudaMemsetAsync(h->d_vmax2, 0, sizeof(unsigned long long), st));
  launch_vmax2(h->p.vx, h->p.vy, h->p.vz, h->n, h->d_vmax2, grid_for(h, h->n), st);
  unsigned long long bits = 0;
  double uni[6];
  CK(cudaMemcpyAsync(&bits, h->d_vmax2, sizeof(bits), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(uni, h->d_uni, sizeof(uni), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  double v2;
  std::memcpy(&v2, &bits, sizeof(v2));
  double vmax = std::sqrt(v2);
  double len = uni[3] - uni[0];
  double t = len / vmax / std::cbrt((double)h->n);
  *dt = std::min(t, h->cfg.dt_max);
  return PT_OK;
}

// Sorted arrays to the caller's, in the caller's order (null outputs are left
// out): each array is scattered to a buffer of its own, so that only the end is
// waited for.
int unpermute_all(pt_handle* h, const double* const* dsrc, double* const* host_out, int count) {
  const int g = grid_for(h, h->n);
  for (int k = 0; k < count; k++) {
    if (!host_out[k]) continue;
    double* const t = h->tmp[k];
    launch_scatter_f64(dsrc[k], t, h->p.order, h->n, g, h->stream);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(host_out[k], t, h->n * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  }
  CK(cudaStreamSynchronize(h->stream));
  return PT_OK;
}

int set_particles_impl(pt_handle* h, int64_t n, const double* const src[8], cudaMemcpyKind kind) {
  if (n < 0 || n > (int64_t)INT32_MAX - 64) return fail(h, PT_E_ARG, "particle count out of range");
  for (int i = 0; i < 8 && n > 0; i++)
    if (!src[i]) return fail(h, PT_E_ARG, "null particle array");
  CKR(ensure_particles(h, n));
  if (n != h->n) h->rep_batch = kMaxReps;
  h->n = n;
  double* dst[8] = {h->p.x, h->p.y, h->p.z, h->p.vx, h->p.vy, h->p.vz, h->p.m, h->p.soft};
  for (int i = 0; i < 8 && n > 0; i++)
    CK(cudaMemcpyAsync(dst[i], src[i], n * sizeof(double), kind, h->stream));
  launch_iota_i32(h->p.order, n, grid_for(h, n), h->stream);
  CK(cudaGetLastError());
  h->have_forces = false;
  h->forces_current = false;
  h->lists_valid = false;
  return PT_OK;
}

}  // namespace

extern "C" {

int pt_abi_version(void) { return PT_ABI_VERSION; }

int pt_config_default(pt_config* c) {
  if (!c) return PT_E_ARG;
  std::memset(c, 0, sizeof(*c));
  c->theta = 0.7;
  c->bucket = 16;
  c->precision = PT_FP64;
  c->integrator = PT_KKD;
  c->dt_max = 1e-5;
  c->device = 0;
  c->record_lists = 0;
  c->periodic = 0;
  c->n_replicas = 0;
  c->period = 1.0;
  c->ewald_rcut = 2.6;  // fEwCut, examples/Ewald.h:26
  c->ewald_hcut = 2.8;  // dEwhCut, examples/Ewald.C:86
  return PT_OK;
}

int pt_create(const pt_config* cfg, pt_handle** out) {
  if (!cfg || !out) return PT_E_ARG;
  *out = nullptr;
  if (!(cfg->theta > 0.0) || cfg->bucket < 1 || cfg->bucket > 32) return PT_E_ARG;
  if (cfg->precision != PT_FP64 && cfg->precision != PT_MIXED && cfg->precision != PT_FP64_LISTS) return PT_E_ARG;
  if (cfg->traversal != PT_TRANSPOSED_DOWN && cfg->traversal != PT_BASIC_DOWN) return PT_E_ARG;
  if (cfg->integrator != PT_KKD && cfg->integrator != PT_KDK) return PT_E_ARG;
  if (cfg->periodic && (!(cfg->period > 0.0) || cfg->n_replicas < 0 || cfg->n_replicas > 8 ||
                        !(cfg->ewald_rcut > 0.0) || cfg->ewald_rcut > 8.0 || !(cfg->ewald_hcut >= 0.0) ||
                        cfg->ewald_hcut > 16.0 || cfg->record_lists))
    return PT_E_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return PT_E_CUDA;
  if (cfg->device < 0 || cfg->device >= ndev) return PT_E_ARG;
  pt_handle* h = new pt_handle();
  h->cfg = *cfg;
  auto bail = [&](int code) {
    pt_destroy(h);
    return code;
  };
  if (cudaSetDevice(cfg->device) != cudaSuccess) return bail(PT_E_CUDA);
  // (the one attribute: cudaGetDeviceProperties takes 2.5 ms)
  if (cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, cfg->device) != cudaSuccess)
    return bail(PT_E_CUDA);
  if (const char* v = std::getenv("PT_MIXED_FUSED")) h->two_phase = std::atoi(v) == 0;
  if (cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking) != cudaSuccess) return bail(PT_E_CUDA);
  h->stream = h->own_stream;
  for (auto& e : h->ev)
    if (cudaEventCreate(&e) != cudaSuccess) return bail(PT_E_CUDA);
  h->bbox_blocks = h->sms * 4;
  if (dalloc(h, &h->bbox_partial, 6 * (size_t)h->bbox_blocks) != PT_OK) return bail(PT_E_NOMEM);
  if (dalloc(h, &h->d_uni, 12) != PT_OK) return bail(PT_E_NOMEM);
  if (dalloc(h, &h->d_words, 1) != PT_OK) return bail(PT_E_NOMEM);
  // a page registered in place takes 0.35 ms, cudaMallocHost 1-3 ms
  static_assert(sizeof(Words) <= kPage, "the words are one page");
  h->pin = static_cast<Words*>(std::aligned_alloc(kPage, kPage));
  if (!h->pin) return bail(PT_E_NOMEM);
  h->pinned = cudaHostRegister(h->pin, kPage, cudaHostRegisterDefault) == cudaSuccess;
  if (!h->pinned) cudaGetLastError();  // the copies work from pageable memory too
  h->d_status = &h->d_words->status;
  h->d_ticket = &h->d_words->ticket;
  h->d_counters = h->d_words->counters;
  h->d_lcur = h->d_words->lcur;
  h->d_total = h->d_words->total;
  if (dalloc(h, &h->d_work, 1) != PT_OK) return bail(PT_E_NOMEM);
  if (dalloc(h, &h->d_queue, 3 * kQueueWords) != PT_OK) return bail(PT_E_NOMEM);
  if (dalloc(h, &h->d_vmax2, 1) != PT_OK) return bail(PT_E_NOMEM);
  // (on the handle's stream: it does not wait for the default stream's work)
  if (cudaMemsetAsync(h->d_words, 0, sizeof(Words), h->own_stream) != cudaSuccess ||
      cudaStreamSynchronize(h->own_stream) != cudaSuccess)
    return bail(PT_E_CUDA);
  *out = h;
  return PT_OK;
}

int pt_destroy(pt_handle* h) {
  if (!h) return PT_OK;
  cudaSetDevice(h->cfg.device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  dfree(h->slab); dfree(h->bbox_partial); dfree(h->d_uni);
  dfree(h->d_words); dfree(h->d_work); dfree(h->d_vmax2); dfree(h->src); dfree(h->srcf); dfree(h->softf);
  dfree(h->node_slab);
  dfree(h->buckets); dfree(h->bucket_work); dfree(h->list_count); dfree(h->list_off); dfree(h->list_node);
  dfree(h->list_kind); dfree(h->dsum); dfree(h->adj); dfree(h->nadj); dfree(h->chain); dfree(h->d_htab); dfree(h->ewd); dfree(h->sph); dfree(h->sph_nbr); dfree(h->sph_nd2);
  dfree(h->sph_list_d); dfree(h->sph_list_i); dfree(h->sph_state);
  dfree(h->pool_pc); dfree(h->pool_pp); dfree(h->l_pc_start);
  dfree(h->d_queue);
  for (auto& e : h->ev)
    if (e) cudaEventDestroy(e);
  if (h->pinned) cudaHostUnregister(h->pin);
  std::free(h->pin);
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
  delete h;
  return PT_OK;
}

const char* pt_last_error(const pt_handle* h) { return h ? h->err.c_str() : "null handle"; }

int pt_set_stream(pt_handle* h, void* stream) {
  if (!h) return PT_E_ARG;
  h->stream = stream ? (cudaStream_t)stream : h->own_stream;
  return PT_OK;
}

int pt_set_theta(pt_handle* h, double theta) {
  if (!h || !(theta > 0.0)) return PT_E_ARG;
  h->cfg.theta = theta;
  return PT_OK;
}

int pt_set_precision(pt_handle* h, int precision) {
  if (!h || (precision != PT_FP64 && precision != PT_MIXED && precision != PT_FP64_LISTS)) return PT_E_ARG;
  h->cfg.precision = precision;
  return PT_OK;
}

int pt_set_sort_spin_limit(pt_handle* h, int64_t polls) {
  if (!h || polls < 0) return PT_E_ARG;
  h->sort_spin_limit = (long long)polls;
  return PT_OK;
}

int pt_set_list_region(pt_handle* h, int64_t entries) {
  if (!h || entries < 64 || entries > (1 << 30)) return PT_E_ARG;
  h->l_region = (unsigned)entries;
  return PT_OK;
}

int pt_set_alloc_limit(pt_handle* h, int64_t bytes) {
  if (!h || bytes < 0) return PT_E_ARG;
  h->alloc_limit = bytes;
  return PT_OK;
}

int pt_set_particles(pt_handle* h, int64_t n, const double* x, const double* y, const double* z, const double* vx,
                     const double* vy, const double* vz, const double* m, const double* soft) {
  if (!h) return PT_E_ARG;
  cudaSetDevice(h->cfg.device);
  const double* src[8] = {x, y, z, vx, vy, vz, m, soft};
  CKR(set_particles_impl(h, n, src, cudaMemcpyHostToDevice));
  CK(cudaStreamSynchronize(h->stream));
  return PT_OK;
}

int pt_set_particles_device(pt_handle* h, int64_t n, const double* x, const double* y, const double* z,
                            const double* vx, const double* vy, const double* vz, const double* m,
                            const double* soft) {
  if (!h) return PT_E_ARG;
  cudaSetDevice(h->cfg.device);
  const double* src[8] = {x, y, z, vx, vy, vz, m, soft};
  return set_particles_impl(h, n, src, cudaMemcpyDeviceToDevice);
}

int64_t pt_num_particles(const pt_handle* h) { return h ? h->n : -1; }

int pt_compute_forces(pt_handle* h) {
  if (!h) return PT_E_ARG;
  cudaSetDevice(h->cfg.device);
  return forces(h, 0, INT64_MAX);
}

int pt_compute_forces_range(pt_handle* h, int64_t b0, int64_t b1) {
  if (!h || b0 < 0 || b1 < b0) return PT_E_ARG;
  cudaSetDevice(h->cfg.device);
  return forces(h, b0, b1);
}

int pt_get_accel(pt_handle* h, double* ax, double* ay, double* az, double* pot, double* pot_full) {
  if (!h) return PT_E_ARG;
  if (!h->have_forces) return fail(h, PT_E_STATE, "no force pass yet");
  if (h->n == 0) return PT_OK;
  cudaSetDevice(h->cfg.device);
  const double* src[5] = {h->p.ax, h->p.ay, h->p.az, h->p.pot, h->p.potf};
  double* dst[5] = {ax, ay, az, pot, pot_full};
  return unpermute_all(h, src, dst, 5);
}

int pt_device_accel(pt_handle* h, double** ax, double** ay, double** az, double** pot, double** pot_full,
                    const int32_t** order) {
  if (!h) return PT_E_ARG;
  if (ax) *ax = h->p.ax;
  if (ay) *ay = h->p.ay;
  if (az) *az = h->p.az;
  if (pot) *pot = h->p.pot;
  if (pot_full) *pot_full = h->p.potf;
  if (order) *order = h->p.order;
  return PT_OK;
}

// Density pass on a rebuilt tree; leaves density and ball^2 (sorted order) in
// h->sph and, with want_nbr, the neighbour lists in h->sph_nbr / h->sph_nd2.
// h->sph holds 7 N doubles: density, ball^2, and the pressure pass's u, ax,
// ay, az, PdV.
static int sph_density_device(pt_handle* h, bool want_nbr) {
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  const int k = sph_k();
  CKR(keys_and_sort(h));
  CKR(build_tree(h));
  CKR(upward(h, false));
  CKR(reserve(h, h->sph_cap, 7 * n, 7 * n, &h->sph));
  if (want_nbr) CKR(reserve(h, h->sph_nbr_cap, n * k, n * k, &h->sph_nbr, &h->sph_nd2));
  // per-warp candidate lists of the neighbour search: 32 targets x 32 entries
  const int kgrid = h->sms * 7;
  const int64_t slots = sph_knn_slots(kgrid);
  CKR(reserve(h, h->sph_list_cap, slots * 1024, slots * 1024, &h->sph_list_d, &h->sph_list_i));
  CK(cudaMemsetAsync(h->d_work, 0, sizeof(unsigned), st));
  launch_sph_density(h->p, n, h->nd.mom, h->nd.walk, h->buckets, h->nbuckets, h->nnodes, h->sph, h->sph + n,
                     want_nbr ? h->sph_nbr : nullptr, want_nbr ? h->sph_nd2 : nullptr, h->sph_list_d,
                     h->sph_list_i, h->d_work, h->d_status, kgrid, st);
  CK(cudaGetLastError());
  return read_status(h);
}

int pt_sph_density(pt_handle* h, double* density, double* ball_sq, int32_t* nbr, double* nbr_d2) {
  if (!h || ((nbr == nullptr) != (nbr_d2 == nullptr))) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  const int k = sph_k();
  if (n == 0) return PT_OK;
  const bool want_nbr = nbr != nullptr;
  CKR(sph_density_device(h, want_nbr));
  const double* src[2] = {h->sph, h->sph + n};
  double* dst[2] = {density, ball_sq};
  CKR(unpermute_all(h, src, dst, 2));
  if (want_nbr) {
    // neighbours of sorted particle i -> caller order, each list sorted by (d2, caller index)
    std::vector<int32_t> hn((size_t)n * k), order(n);
    std::vector<double> hd((size_t)n * k);
    CK(cudaMemcpyAsync(hn.data(), h->sph_nbr, hn.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(hd.data(), h->sph_nd2, hd.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(order.data(), h->p.order, n * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::vector<std::pair<double, int32_t>> row(k);
    for (int64_t i = 0; i < n; i++) {
      int m = 0;
      for (int e = 0; e < k; e++) {
        const int32_t j = hn[(size_t)i * k + e];
        if (j >= 0) row[m++] = {hd[(size_t)i * k + e], order[j]};
      }
      std::sort(row.begin(), row.begin() + m);
      const int64_t c = order[i];
      for (int e = 0; e < k; e++) {
        nbr[c * k + e] = e < m ? row[e].second : -1;
        nbr_d2[c * k + e] = e < m ? row[e].first : -1.0;
      }
    }
  }
  return PT_OK;
}

int pt_sph_pressure(pt_handle* h, const double* u, double* density, double* ax, double* ay, double* az,
                    double* pdv) {
  if (!h || !u) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  if (n == 0) return PT_OK;
  CKR(sph_density_device(h, true));
  double* us = h->sph + 2 * n;
  double* out = h->sph + 3 * n;  // ax, ay, az, PdV
  CK(cudaMemcpyAsync(h->tmp[0], u, n * sizeof(double), cudaMemcpyHostToDevice, st));
  launch_gather_by_order(h->tmp[0], us, h->p.order, n, grid_for(h, n), st);
  CK(cudaMemsetAsync(out, 0, 4 * n * sizeof(double), st));
  launch_sph_pressure(h->p, h->sph, h->sph + n, us, h->sph_nbr, h->sph_nd2, n, out, out + n, out + 2 * n,
                      out + 3 * n, h->d_status, h->sms * 16, st);
  CK(cudaGetLastError());
  CKR(read_status(h));
  double* dst[5] = {density, ax, ay, az, pdv};
  const double* src[5] = {h->sph, out, out + n, out + 2 * n, out + 3 * n};
  return unpermute_all(h, src, dst, 5);
}

// nsteps iterations of the SPH example: density pass, pressure pass with the
// predicted energies and velocities, then kick + perturb with the SPH updates.
// dt = max_timestep (examples/SPH.C getTimestep).  The caller-order state
// (u, u_pred, v_pred) stays on the device across the steps; the sorted copies
// the pressure pass reads are gathered by p.order after each re-sort.
int pt_sph_step(pt_handle* h, int nsteps, double* u, double* u_pred, double* vpx, double* vpy, double* vpz) {
  if (!h || nsteps < 0 || !u || !u_pred || !vpx || !vpy || !vpz) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  if (!(h->cfg.dt_max > 0.0)) return fail(h, PT_E_ARG, "dt_max must be positive");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  if (n == 0 || nsteps == 0) return PT_OK;
  CKR(reserve(h, h->sph_state_cap, 8 * n, 8 * n, &h->sph_state));
  double* cs = h->sph_state;  // caller order: u, u_pred, vpx, vpy, vpz
  double* vps = cs + 5 * n;   // sorted v_pred
  double* in[5] = {u, u_pred, vpx, vpy, vpz};
  for (int k = 0; k < 5; k++) CK(cudaMemcpyAsync(cs + k * n, in[k], n * sizeof(double), cudaMemcpyHostToDevice, st));
  const int g = grid_for(h, n);
  const double dt = h->cfg.dt_max;
  for (int s = 0; s < nsteps; s++) {
    CKR(sph_density_device(h, true));  // re-sorts the particles, builds the tree, density + neighbours
    double* us = h->sph + 2 * n;
    double* out = h->sph + 3 * n;  // ax, ay, az, PdV
    launch_gather_by_order(cs + n, us, h->p.order, n, g, st);
    for (int d = 0; d < 3; d++) launch_gather_by_order(cs + (2 + d) * n, vps + d * n, h->p.order, n, g, st);
    CK(cudaMemsetAsync(out, 0, 4 * n * sizeof(double), st));
    Particles q = h->p;  // the pressure pass reads velocity_predicted
    q.vx = vps;
    q.vy = vps + n;
    q.vz = vps + 2 * n;
    launch_sph_pressure(q, h->sph, h->sph + n, us, h->sph_nbr, h->sph_nd2, n, out, out + n, out + 2 * n,
                        out + 3 * n, h->d_status, h->sms * 16, st);
    CK(cudaGetLastError());
    CKR(read_status(h));  // a failed pressure pass leaves the particles as they were
    launch_sph_kick_perturb(h->p, out, out + n, out + 2 * n, out + 3 * n, cs, cs + n, cs + 2 * n, cs + 3 * n,
                            cs + 4 * n, n, dt, g, st);
    CK(cudaGetLastError());
    CKR(read_status(h));
    h->last_dt = dt;
  }
  double* outs[5] = {u, u_pred, vpx, vpy, vpz};
  for (int k = 0; k < 5; k++) CK(cudaMemcpyAsync(outs[k], cs + k * n, n * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return PT_OK;
}

int pt_get_bucket_work(pt_handle* h, uint64_t* work) {
  if (!h || !work) return PT_E_ARG;
  if (!h->have_forces) return fail(h, PT_E_STATE, "no force pass yet");
  if (h->nbuckets == 0) return PT_OK;
  cudaSetDevice(h->cfg.device);
  CK(cudaMemcpyAsync(work, h->bucket_work, h->nbuckets * sizeof(uint64_t), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PT_OK;
}

int pt_advance(pt_handle* h, double* dt_out) {
  if (!h) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  if (!h->have_forces || !h->forces_current) return fail(h, PT_E_STATE, "no force pass at the current positions");
  cudaSetDevice(h->cfg.device);
  double dt = 0.0;
  if (h->n > 0) {
    CKR(timestep(h, &dt));
    launch_kick_perturb(h->p, h->n, dt, grid_for(h, h->n), h->stream);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->stream));
  }
  h->last_dt = dt;
  h->forces_current = false;
  if (dt_out) *dt_out = dt;
  return PT_OK;
}

int pt_step(pt_handle* h, int nsteps) {
  if (!h || nsteps < 0) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  cudaSetDevice(h->cfg.device);
  const int g = grid_for(h, h->n);
  for (int s = 0; s < nsteps; s++) {
    if (h->cfg.integrator == PT_KKD) {
      CKR(forces(h, 0, INT64_MAX));
      double dt;
      CKR(timestep(h, &dt));
      h->last_dt = dt;
      launch_kick_perturb(h->p, h->n, dt, g, h->stream);
      CK(cudaGetLastError());
      h->forces_current = false;
    } else {
      if (!h->forces_current) CKR(forces(h, 0, INT64_MAX));
      double dt;
      CKR(timestep(h, &dt));
      h->last_dt = dt;
      launch_kick_half(h->p, h->n, dt, g, h->stream);
      launch_drift(h->p, h->n, dt, g, h->stream);
      CK(cudaGetLastError());
      CKR(forces(h, 0, INT64_MAX));
      launch_kick_half(h->p, h->n, dt, g, h->stream);
      CK(cudaGetLastError());
    }
  }
  CK(cudaStreamSynchronize(h->stream));
  return PT_OK;
}

int pt_get_state(pt_handle* h, double* x, double* y, double* z, double* vx, double* vy, double* vz) {
  if (!h) return PT_E_ARG;
  if (h->n == 0) return PT_OK;
  cudaSetDevice(h->cfg.device);
  const double* src[6] = {h->p.x, h->p.y, h->p.z, h->p.vx, h->p.vy, h->p.vz};
  double* dst[6] = {x, y, z, vx, vy, vz};
  return unpermute_all(h, src, dst, 6);
}

int pt_last_dt(const pt_handle* h, double* dt) {
  if (!h || !dt) return PT_E_ARG;
  *dt = h->last_dt;
  return PT_OK;
}

int pt_get_keys(pt_handle* h, uint64_t* keys) {
  if (!h || !keys) return PT_E_ARG;
  if (!h->have_forces) return fail(h, PT_E_STATE, "no force pass yet");
  if (h->n == 0) return PT_OK;
  if (!h->keys_valid) return fail(h, PT_E_STATE, "the keys were lost in a failed pass");
  cudaSetDevice(h->cfg.device);
  launch_scatter_u64(h->p.key, h->key_alt, h->p.order, h->n, grid_for(h, h->n), h->stream);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(keys, h->key_alt, h->n * sizeof(uint64_t), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PT_OK;
}

int pt_get_universe(pt_handle* h, double* lo3, double* hi3) {
  if (!h || !lo3 || !hi3) return PT_E_ARG;
  double u[6];
  CK(cudaMemcpyAsync(u, h->d_uni, sizeof(u), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int d = 0; d < 3; d++) {
    lo3[d] = u[d];
    hi3[d] = u[3 + d];
  }
  return PT_OK;
}

int pt_get_tree_size(pt_handle* h, int64_t* n_nodes, int64_t* n_buckets) {
  if (!h) return PT_E_ARG;
  if (n_nodes) *n_nodes = h->nnodes;
  if (n_buckets) *n_buckets = h->nbuckets;
  return PT_OK;
}

int pt_get_tree(pt_handle* h, uint64_t* keys, int32_t* ints4, double* dbls18) {
  if (!h) return PT_E_ARG;
  const int64_t nn = h->nnodes;
  if (nn == 0) return PT_OK;
  cudaStream_t st = h->stream;
  std::vector<int32_t> type(nn), depth(nn), count(nn);
  std::vector<Mom> mom(nn);
  if (keys) CK(cudaMemcpyAsync(keys, h->nd.key, nn * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(type.data(), h->nd.type, nn * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(depth.data(), h->nd.depth, nn * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(count.data(), h->nd.count, nn * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(mom.data(), h->nd.mom, nn * sizeof(Mom), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  for (int64_t i = 0; i < nn; i++) {
    if (ints4) {
      ints4[4 * i + 0] = type[i];
      ints4[4 * i + 1] = depth[i];
      ints4[4 * i + 2] = count[i];
      ints4[4 * i + 3] = (type[i] == kTypeInternal) ? 8 : 0;
    }
    if (dbls18) {
      const Mom& q = mom[i];
      double* d = dbls18 + 18 * i;
      d[0] = q.mass; d[1] = q.cm[0]; d[2] = q.cm[1]; d[3] = q.cm[2]; d[4] = q.soft; d[5] = q.radius;
      d[6] = q.xx; d[7] = q.xy; d[8] = q.xz; d[9] = q.yy; d[10] = q.yz; d[11] = q.zz;
      d[12] = q.lo[0]; d[13] = q.lo[1]; d[14] = q.lo[2]; d[15] = q.hi[0]; d[16] = q.hi[1]; d[17] = q.hi[2];
    }
  }
  return PT_OK;
}

int pt_get_bucket_keys(pt_handle* h, uint64_t* keys) {
  if (!h || !keys) return PT_E_ARG;
  const int64_t nb = h->nbuckets;
  if (nb == 0) return PT_OK;
  std::vector<int32_t> b(nb);
  std::vector<uint64_t> nk(h->nnodes);
  CK(cudaMemcpyAsync(b.data(), h->buckets, nb * sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(nk.data(), h->nd.key, h->nnodes * sizeof(uint64_t), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int64_t i = 0; i < nb; i++) keys[i] = nk[b[i]];
  return PT_OK;
}

int pt_get_lists_size(pt_handle* h, int64_t* total) {
  if (!h || !total) return PT_E_ARG;
  if (!h->lists_valid) return fail(h, PT_E_STATE, "no interaction lists recorded (config.record_lists)");
  *total = h->list_total;
  return PT_OK;
}

int pt_get_lists(pt_handle* h, int64_t* offsets, uint64_t* keys, int32_t* kinds) {
  if (!h) return PT_E_ARG;
  if (!h->lists_valid) return fail(h, PT_E_STATE, "no interaction lists recorded (config.record_lists)");
  const int64_t nb = h->list_nb - 1, tot = h->list_total;
  std::vector<int64_t> off(nb + 1);
  std::vector<int32_t> node(tot);
  std::vector<int8_t> kind(tot);
  std::vector<uint64_t> nk(h->nnodes);
  cudaStream_t st = h->stream;
  CK(cudaMemcpyAsync(off.data(), h->list_off, (nb + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  if (tot) {
    CK(cudaMemcpyAsync(node.data(), h->list_node, tot * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(kind.data(), h->list_kind, tot * sizeof(int8_t), cudaMemcpyDeviceToHost, st));
  }
  CK(cudaMemcpyAsync(nk.data(), h->nd.key, h->nnodes * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (offsets)
    for (int64_t i = 0; i <= nb; i++) offsets[i] = off[i];
  for (int64_t i = 0; i < tot; i++) {
    if (keys) keys[i] = nk[node[i]];
    if (kinds) kinds[i] = kind[i] ? 1 : 0;  // node() entries, softened or not, are kind 1
  }
  return PT_OK;
}

int pt_get_list_digests(pt_handle* h, int which, uint64_t* digest, int64_t* count) {
  if (!h || (which != 0 && which != 1)) return PT_E_ARG;
  const int64_t nb = h->nbuckets;
  if (which == 0 && !(h->lists_valid && !h->trav_range_partial && h->list_nb - 1 == nb))
    return fail(h, PT_E_STATE, "no interaction lists recorded for every bucket (config.record_lists)");
  if (which == 1 && !h->tp_lists_valid)
    return fail(h, PT_E_STATE, "the last pass was not a two-phase mixed pass over every bucket");
  if (nb == 0) return PT_OK;
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  DevBuf buf;
  CK(device_malloc(h, &buf.p, 2 * nb * sizeof(double)));
  unsigned long long* d_dig = reinterpret_cast<unsigned long long*>(buf.p);
  int64_t* d_cnt = reinterpret_cast<int64_t*>(buf.p + nb);
  if (which == 0)
    launch_digest_recorded(h->list_off, h->list_node, h->list_kind, nb, d_dig, d_cnt, st);
  else
    launch_digest_two_phase(h->pool_pc, h->pool_pp, h->l_pc_start, h->l_pc_count, h->l_pp_start, h->l_pp_count, nb,
                            d_dig, d_cnt, st);
  CK(cudaGetLastError());
  if (digest) CK(cudaMemcpyAsync(digest, d_dig, nb * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  if (count) CK(cudaMemcpyAsync(count, d_cnt, nb * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  return PT_OK;
}

int pt_get_counters(pt_handle* h, pt_counters* c) {
  if (!h || !c) return PT_E_ARG;
  *c = h->last;
  return PT_OK;
}

int pt_direct_sum(pt_handle* h, int64_t nt, const int32_t* targets, double* ax, double* ay, double* az,
                  double* pot) {
  if (!h || nt < 0 || (nt > 0 && !targets)) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  const int64_t n = h->n;
  if (nt == 0 || n == 0) return PT_OK;
  for (int64_t t = 0; t < nt; t++)
    if (targets[t] < 0 || targets[t] >= n) return fail(h, PT_E_ARG, "target index out of range");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int tb = (int)((nt + 255) / 256);
  int nsplit = std::max(1, std::min(256, (4 * h->sms + tb - 1) / tb));
  if (n < 4096) nsplit = 1;
  const int64_t need = 5 * n + 4 * nt * nsplit + nt;
  CKR(reserve(h, h->dsum_cap, need, need, &h->dsum));
  // caller-order copies of x, y, z, m, soft
  const double* src[5] = {h->p.x, h->p.y, h->p.z, h->p.m, h->p.soft};
  for (int k = 0; k < 5; k++) launch_scatter_f64(src[k], h->dsum + k * n, h->p.order, n, grid_for(h, n), st);
  int32_t* dt = reinterpret_cast<int32_t*>(h->dsum + 5 * n + 4 * nt * nsplit);
  CK(cudaMemcpyAsync(dt, targets, nt * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  double* part = h->dsum + 5 * n;
  launch_direct_sum(h->dsum, h->dsum + n, h->dsum + 2 * n, h->dsum + 3 * n, h->dsum + 4 * n, n, dt, nt, nsplit,
                    part, st);
  CK(cudaGetLastError());
  std::vector<double> hp((size_t)4 * nt * nsplit);
  CK(cudaMemcpyAsync(hp.data(), part, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  for (int64_t t = 0; t < nt; t++) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int sl = 0; sl < nsplit; sl++)
      for (int k = 0; k < 4; k++) s[k] += hp[((size_t)sl * nt + t) * 4 + k];
    if (ax) ax[t] = s[0];
    if (ay) ay[t] = s[1];
    if (az) az[t] = s[2];
    if (pot) pot[t] = s[3];
  }
  return PT_OK;
}

// FP64 periodic (Ewald) direct sum: alpha = 4/L, real-space images within
// 1.5 L (erfc(6) ~ 2e-17), reciprocal |h|^2 <= 64 (exp(-pi^2 64/16) ~ 7e-18),
// the spline kernel for the nearest image within soft_i + soft_j, and the
// background and self terms in the potential.
int pt_ewald_direct_sum(pt_handle* h, int64_t nt, const int32_t* targets, double* ax, double* ay, double* az,
                        double* pot) {
  if (!h || nt < 0 || (nt > 0 && !targets)) return PT_E_ARG;
  if (!h->p.x) return fail(h, PT_E_STATE, "no particles");
  if (!(h->cfg.period > 0.0)) return fail(h, PT_E_ARG, "period must be positive");
  const int64_t n = h->n;
  if (nt == 0 || n == 0) return PT_OK;
  for (int64_t t = 0; t < nt; t++)
    if (targets[t] < 0 || targets[t] >= n) return fail(h, PT_E_ARG, "target index out of range");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const double L = h->cfg.period, V = L * L * L;
  const double alpha = 4.0 / L, rcut = 1.5 * L;
  const int hmax = 8;
  std::vector<double4> kv;
  for (int hx = -hmax; hx <= hmax; hx++)
    for (int hy = -hmax; hy <= hmax; hy++)
      for (int hz = -hmax; hz <= hmax; hz++) {
        const int h2 = hx * hx + hy * hy + hz * hz;
        if (h2 == 0 || h2 > hmax * hmax) continue;
        const double kx = 2 * M_PI / L * hx, ky = 2 * M_PI / L * hy, kz = 2 * M_PI / L * hz;
        const double k2 = kx * kx + ky * ky + kz * kz;
        kv.push_back(make_double4(kx, ky, kz, 4 * M_PI / V * std::exp(-k2 / (4 * alpha * alpha)) / k2));
      }
  const int nk = (int)kv.size();
  kv.push_back(make_double4(0.0, 0.0, 0.0, 0.0));  // k = 0: total mass
  const int tb = (int)((nt + 127) / 128);
  int nsplit = std::max(1, std::min(256, (4 * h->sms + tb - 1) / tb));
  if (n < 4096) nsplit = 1;
  // doubles: caller-order x y z m soft (5n) | partials (4 nt nsplit) | recip out (4 nt) | S (2 nk + 2)
  //          | k vectors (4 (nk + 1), 32-byte aligned) | targets (int32, nt / 2 + 1 doubles)
  const int64_t off_part = 5 * n, off_rec = off_part + 4 * nt * nsplit, off_S = off_rec + 4 * nt;
  const int64_t off_kv = (off_S + 2 * (nk + 1) + 3) / 4 * 4;
  const int64_t off_tgt = off_kv + 4 * (nk + 1);
  const int64_t need = off_tgt + nt / 2 + 1;
  CKR(reserve(h, h->ewd_cap, need, need, &h->ewd));
  double* c = h->ewd;
  const double* src[5] = {h->p.x, h->p.y, h->p.z, h->p.m, h->p.soft};
  for (int k = 0; k < 5; k++) launch_scatter_f64(src[k], c + k * n, h->p.order, n, grid_for(h, n), st);
  double* part = c + off_part;
  double* rec = c + off_rec;
  double* S = c + off_S;
  double4* dkv = reinterpret_cast<double4*>(c + off_kv);
  int32_t* dt = reinterpret_cast<int32_t*>(c + off_tgt);
  CK(cudaMemcpyAsync(dkv, kv.data(), kv.size() * sizeof(double4), cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dt, targets, nt * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  launch_ewald_structure(c, c + n, c + 2 * n, c + 3 * n, n, dkv, nk + 1, S, st);
  launch_ewald_real(c, c + n, c + 2 * n, c + 3 * n, c + 4 * n, n, dt, nt, nsplit, L, alpha, rcut, part, st);
  launch_ewald_recip(c, c + n, c + 2 * n, c + 3 * n, dt, nt, dkv, nk, S, alpha, V, rec, st);
  CK(cudaGetLastError());
  std::vector<double> hp((size_t)4 * nt * nsplit), hr((size_t)4 * nt);
  CK(cudaMemcpyAsync(hp.data(), part, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(hr.data(), rec, hr.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  for (int64_t t = 0; t < nt; t++) {
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
    for (int sl = 0; sl < nsplit; sl++)
      for (int k = 0; k < 4; k++) s4[k] += hp[((size_t)sl * nt + t) * 4 + k];
    for (int k = 0; k < 4; k++) s4[k] += hr[4 * t + k];
    if (ax) ax[t] = s4[0];
    if (ay) ay[t] = s4[1];
    if (az) az[t] = s4[2];
    if (pot) pot[t] = s4[3];
  }
  return PT_OK;
}

}  // extern "C"

// ---------------------------------------------------------------- differentiation
namespace {

int ensure_adjoint(pt_handle* h) {
  const int64_t need = 21 * std::max<int64_t>(h->n, 1);
  CKR(reserve(h, h->adj_cap, need, need, &h->adj));
  const int64_t nneed = 10 * std::max<int64_t>(h->nnodes, 1);
  return reserve(h, h->nadj_cap, nneed, nneed, &h->nadj);
}

bool lists_cover_all(const pt_handle* h) {
  return h->lists_valid && !h->trav_range_partial && h->list_nb - 1 == h->nbuckets;
}

// Leaf moments, upward pass and traversal records on the existing topology.
int recompute_moments(pt_handle* h) {
  cudaStream_t st = h->stream;
  CKR(ensure_src(h));
  launch_leaf_moments(h->nd, h->buckets, h->nbuckets, h->p, h->src, st);
  launch_upward(h->nd, h->ninternal, st);
  const double gfac = (4.0 / 3.0) / (h->cfg.theta * h->cfg.theta);
  launch_finalize(h->nd, h->nnodes, gfac, h->cfg.precision == PT_MIXED, st);
  CK(cudaGetLastError());
  return PT_OK;
}

// Gradient of sum_i cot_i . a_i for the recorded lists.  cot: caller order,
// device; outputs: caller order, device (gx, gy, gz, gm; added into when
// accumulate is set).
int adjoint_device(pt_handle* h, const double* cx, const double* cy, const double* cz, double* gx, double* gy,
                   double* gz, double* gm, bool accumulate) {
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  const int g = grid_for(h, n);
  CKR(ensure_adjoint(h));
  double* cs = h->adj;       // 3N sorted cotangent
  double* gs = h->adj + 3 * n;  // 4N sorted gradient
  double* tmp = h->adj + 7 * n;  // 4N caller-order gradient
  launch_gather_by_order(cx, cs, h->p.order, n, g, st);
  launch_gather_by_order(cy, cs + n, h->p.order, n, g, st);
  launch_gather_by_order(cz, cs + 2 * n, h->p.order, n, g, st);
  CK(cudaMemsetAsync(gs, 0, 4 * n * sizeof(double), st));
  CK(cudaMemsetAsync(h->nadj, 0, 10 * h->nnodes * sizeof(double), st));
  CK(cudaMemsetAsync(h->d_work, 0, sizeof(unsigned), st));
  AdjParams A{};
  A.p = h->p;
  A.walk = h->nd.walk;
  A.quad = h->nd.quad;
  A.mom = h->nd.mom;
  A.parent = h->nd.parent;
  A.buckets = h->buckets;
  A.nbuckets = h->nbuckets;
  A.nnodes = h->nnodes;
  A.list_off = h->list_off;
  A.list_node = h->list_node;
  A.list_kind = h->list_kind;
  A.cax = cs;
  A.cay = cs + n;
  A.caz = cs + 2 * n;
  A.gx = gs;
  A.gy = gs + n;
  A.gz = gs + 2 * n;
  A.gm = gs + 3 * n;
  A.nadj = h->nadj;
  A.work = h->d_work;
  A.status = h->d_status;
  launch_adjoint(A, h->sms, st);
  CK(cudaGetLastError());
  double* outs[4] = {gx, gy, gz, gm};
  for (int k = 0; k < 4; k++) {
    if (!outs[k]) continue;
    if (accumulate) {
      launch_scatter_f64(gs + k * n, tmp + k * n, h->p.order, n, g, st);
      launch_axpy1(n, 1.0, tmp + k * n, outs[k], g, st);
    } else {
      launch_scatter_f64(gs + k * n, outs[k], h->p.order, n, g, st);
    }
  }
  CK(cudaGetLastError());
  return read_status(h);
}

}  // namespace

extern "C" {

int pt_forces_frozen(pt_handle* h, const double* x, const double* y, const double* z, const double* m) {
  if (!h) return PT_E_ARG;
  if (!lists_cover_all(h)) return fail(h, PT_E_STATE, "needs a full force pass with config.record_lists");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  const int g = grid_for(h, n);
  CKR(ensure_adjoint(h));
  const double* src[4] = {x, y, z, m};
  double* dst[4] = {h->p.x, h->p.y, h->p.z, h->p.m};
  for (int k = 0; k < 4; k++) {
    if (!src[k]) continue;
    CK(cudaMemcpyAsync(h->adj, src[k], n * sizeof(double), cudaMemcpyHostToDevice, st));
    launch_gather_by_order(h->adj, dst[k], h->p.order, n, g, st);
  }
  CKR(recompute_moments(h));
  TravParams P{};
  P.p = h->p;
  P.walk = h->nd.walk;
  P.walks = h->nd.walks;
  P.quad = h->nd.quad;
  P.src = h->src;
  P.buckets = h->buckets;
  P.b_begin = 0;
  P.b_end = h->nbuckets;
  P.nnodes = h->nnodes;
  P.list_off = h->list_off;
  P.list_node = h->list_node;
  P.list_kind = h->list_kind;
  P.status = h->d_status;
  use_queue(h, P, 0);
  P.batch = bucket_batch(h, h->nbuckets);
  CKR(zero_queue(h));
  launch_replay_f64(P, h->sms * 16, st);
  CK(cudaGetLastError());
  return read_status(h);
}

int pt_adjoint(pt_handle* h, const double* cax, const double* cay, const double* caz, double* gx, double* gy,
               double* gz, double* gm) {
  if (!h || !cax || !cay || !caz) return PT_E_ARG;
  if (!lists_cover_all(h)) return fail(h, PT_E_STATE, "needs a full force pass with config.record_lists");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  if (n == 0) return PT_OK;
  CKR(ensure_adjoint(h));
  double* buf = h->adj + 14 * n;  // caller-order cotangent (3N) and gradients (4N), kept by the handle
  const double* hin[3] = {cax, cay, caz};
  for (int k = 0; k < 3; k++) {
    CK(cudaMemcpyAsync(buf + k * n, hin[k], n * sizeof(double), cudaMemcpyHostToDevice, st));
  }
  int rc = adjoint_device(h, buf, buf + n, buf + 2 * n, buf + 3 * n, buf + 4 * n, buf + 5 * n, buf + 6 * n, false);
  if (rc == PT_OK) {
    double* hout[4] = {gx, gy, gz, gm};
    for (int k = 0; k < 4; k++)
      if (hout[k]) CK(cudaMemcpyAsync(hout[k], buf + (3 + k) * n, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
  }
  return rc;
}

}  // extern "C"

// ---------------------------------------------------------------- K-step chain
namespace {

// Caller-order state -> particle arrays (order reset to identity).
int load_state(pt_handle* h, const double* X, const double* V, const double* M, const double* S) {
  const int64_t n = h->n;
  const double* src[8] = {X, X + n, X + 2 * n, V, V + n, V + 2 * n, M, S};
  return set_particles_impl(h, n, src, cudaMemcpyDeviceToDevice);
}

// Force pass with interaction lists; accelerations in caller order into A (3N).
int chain_forces(pt_handle* h, double* A) {
  const int saved = h->cfg.record_lists;
  h->cfg.record_lists = 1;
  const int rc = forces(h, 0, INT64_MAX);
  h->cfg.record_lists = saved;
  CKR(rc);
  const int64_t n = h->n;
  const int g = grid_for(h, n);
  launch_scatter_f64(h->p.ax, A, h->p.order, n, g, h->stream);
  launch_scatter_f64(h->p.ay, A + n, h->p.order, n, g, h->stream);
  launch_scatter_f64(h->p.az, A + 2 * n, h->p.order, n, g, h->stream);
  CK(cudaGetLastError());
  return PT_OK;
}

}  // namespace

extern "C" int pt_chain_grad(pt_handle* h, int nsteps, double dt, int ckpt_every, const double* yx, const double* yy,
                             const double* yz, double* loss, double* gx, double* gy, double* gz, double* gvx,
                             double* gvy, double* gvz, double* gm) {
  if (!h || nsteps < 1 || !(dt > 0.0) || !yx || !yy || !yz) return PT_E_ARG;
  if (!h->p.x || h->n == 0) return fail(h, PT_E_STATE, "no particles");
  cudaSetDevice(h->cfg.device);
  cudaStream_t st = h->stream;
  const int64_t n = h->n;
  const int g = grid_for(h, n);
  const int K = nsteps;
  int C = ckpt_every > 0 ? ckpt_every : std::max(1, (int)std::lround(std::sqrt((double)K)));
  if (C > K) C = K;
  const int nck = (K + C - 1) / C;
  // layout (doubles): X0 V0 M0 S0 | X V A | Y | xb vb mb pend | ckpt (nck x 6N) | seg ((C+1) x 3N)
  const int64_t off_X0 = 0, off_V0 = 3 * n, off_M0 = 6 * n, off_S0 = 7 * n, off_X = 8 * n, off_V = 11 * n,
                off_A = 14 * n, off_Y = 17 * n, off_xb = 20 * n, off_vb = 23 * n, off_mb = 26 * n, off_pd = 27 * n,
                off_ck = 30 * n, off_seg = off_ck + (int64_t)nck * 6 * n;
  const int64_t total = off_seg + (int64_t)(C + 1) * 3 * n;
  CKR(reserve(h, h->chain_cap, total, total, &h->chain));
  double* B = h->chain;
  double *X0 = B + off_X0, *V0 = B + off_V0, *M0 = B + off_M0, *S0 = B + off_S0, *X = B + off_X, *V = B + off_V,
         *A = B + off_A, *Y = B + off_Y, *xb = B + off_xb, *vb = B + off_vb, *mb = B + off_mb, *pd = B + off_pd,
         *ck = B + off_ck, *seg = B + off_seg;
  // initial state in caller order (the arrays may be key-sorted by an earlier pass)
  const double* cur[8] = {h->p.x, h->p.y, h->p.z, h->p.vx, h->p.vy, h->p.vz, h->p.m, h->p.soft};
  double* dst0[8] = {X0, X0 + n, X0 + 2 * n, V0, V0 + n, V0 + 2 * n, M0, S0};
  for (int k = 0; k < 8; k++) launch_scatter_f64(cur[k], dst0[k], h->p.order, n, g, st);
  const double* hy[3] = {yx, yy, yz};
  for (int k = 0; k < 3; k++) CK(cudaMemcpyAsync(Y + k * n, hy[k], n * sizeof(double), cudaMemcpyHostToDevice, st));
  auto copy3 = [&](double* d, const double* s) {
    return cudaMemcpyAsync(d, s, 3 * n * sizeof(double), cudaMemcpyDeviceToDevice, st);
  };
  // one KDK step from (X, V) with A = a(X) on entry; A = a(X') on exit
  auto kdk = [&]() -> int {
    launch_axpy3(n, 0.5 * dt, A, A + n, A + 2 * n, V, V + n, V + 2 * n, g, st);
    launch_axpy3(n, dt, V, V + n, V + 2 * n, X, X + n, X + 2 * n, g, st);
    CKR(load_state(h, X, V, M0, S0));
    CKR(chain_forces(h, A));
    launch_axpy3(n, 0.5 * dt, A, A + n, A + 2 * n, V, V + n, V + 2 * n, g, st);
    return PT_OK;
  };

  // forward, keeping (X, V) every C steps
  CK(copy3(X, X0));
  CK(copy3(V, V0));
  CKR(load_state(h, X, V, M0, S0));
  CKR(chain_forces(h, A));
  for (int s = 0; s < K; s++) {
    if (s % C == 0) {
      CK(copy3(ck + (int64_t)(s / C) * 6 * n, X));
      CK(copy3(ck + (int64_t)(s / C) * 6 * n + 3 * n, V));
    }
    CKR(kdk());
  }
  // loss = 0.5 sum |x_K - y|^2 and its gradient
  {
    std::vector<double> hx(3 * n);
    CK(cudaMemcpyAsync(hx.data(), X, 3 * n * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    double L = 0.0;
    for (int k = 0; k < 3; k++)
      for (int64_t i = 0; i < n; i++) {
        const double d = hx[k * n + i] - hy[k][i];
        L += d * d;
      }
    if (loss) *loss = 0.5 * L;
  }
  CK(copy3(xb, X));
  launch_axpy3(n, -1.0, Y, Y + n, Y + 2 * n, xb, xb + n, xb + 2 * n, g, st);
  CK(cudaMemsetAsync(vb, 0, 3 * n * sizeof(double), st));
  CK(cudaMemsetAsync(mb, 0, n * sizeof(double), st));
  CK(cudaMemsetAsync(pd, 0, 3 * n * sizeof(double), st));

  // backward, segment by segment, recomputing each segment's positions
  for (int c = nck - 1; c >= 0; c--) {
    const int s0 = c * C, s1 = std::min(s0 + C, K);
    CK(copy3(X, ck + (int64_t)c * 6 * n));
    CK(copy3(V, ck + (int64_t)c * 6 * n + 3 * n));
    CK(copy3(seg, X));
    CKR(load_state(h, X, V, M0, S0));
    CKR(chain_forces(h, A));
    for (int s = s0; s < s1; s++) {
      CKR(kdk());
      CK(copy3(seg + (int64_t)(s + 1 - s0) * 3 * n, X));
    }
    for (int s = s1 - 1; s >= s0; s--) {
      // the point x_{s+1}: a(x_{s+1}) feeds v_{s+1} (and v_h of step s+1, already in pd)
      launch_axpy3(n, 0.5 * dt, vb, vb + n, vb + 2 * n, pd, pd + n, pd + 2 * n, g, st);
      if (s + 1 < K) {
        CKR(load_state(h, seg + (int64_t)(s + 1 - s0) * 3 * n, V, M0, S0));
        CKR(chain_forces(h, A));
        CKR(adjoint_device(h, pd, pd + n, pd + 2 * n, xb, xb + n, xb + 2 * n, mb, true));
      }
      // x_{s+1} = x_s + dt v_h ; v_h = v_s + dt/2 a(x_s)
      launch_axpy3(n, dt, xb, xb + n, xb + 2 * n, vb, vb + n, vb + 2 * n, g, st);
      CK(cudaMemsetAsync(pd, 0, 3 * n * sizeof(double), st));
      launch_axpy3(n, 0.5 * dt, vb, vb + n, vb + 2 * n, pd, pd + n, pd + 2 * n, g, st);
    }
  }
  // the point x_0
  CKR(load_state(h, X0, V0, M0, S0));
  CKR(chain_forces(h, A));
  CKR(adjoint_device(h, pd, pd + n, pd + 2 * n, xb, xb + n, xb + 2 * n, mb, true));
  double* hout[7] = {gx, gy, gz, gvx, gvy, gvz, gm};
  const double* dsrc[7] = {xb, xb + n, xb + 2 * n, vb, vb + n, vb + 2 * n, mb};
  for (int k = 0; k < 7; k++)
    if (hout[k]) CK(cudaMemcpyAsync(hout[k], dsrc[k], n * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  // leave the handle at the initial state (with its force pass)
  return PT_OK;
}
