// k_sort.cu -- K3 stable LSD radix sort of the 64-bit SFC keys with a uint32
// payload (onesweep) and K4 particle permutation.
//
// Replaces std::sort(particles) (src/Subtree.h:281, Particle::operator<
// src/Particle.C:61-79), which moves ~170-byte AoS particles; here only the
// 12-byte (key, index) pairs move and the FP64 SoA is gathered once.
//
// Onesweep (one read and one write of the pairs per 8-bit digit):
//   histogram  one pass over the keys builds all eight 256-bin digit
//              histograms (shared-memory atomics, then global atomics), and
//              one small kernel turns each into exclusive digit offsets;
//   pass       per digit, each CTA claims the next tile (4096 keys; 1024 up to 2^19
//              keys) from an atomic counter (so every earlier tile is already running), ranks its
//              keys stably with __match_any_sync (lane order = key order in a
//              round, rounds and warps in order), publishes its per-digit
//              counts, and resolves the counts of all earlier tiles by
//              decoupled look-back on 64-bit status words (tag | flag | count;
//              a word of another tag is one an earlier pass left, so the words
//              are cleared only when the tags start over).  The
//              ranked tile is staged in shared memory and written out with
//              consecutive threads on consecutive destinations.
// The look-back only waits on tiles that claimed their index earlier and
// publish their counts before waiting on anything, so it always ends; the spin
// is still bounded (spin_limit polls of an unpublished tile, 2^21 by default)
// and reports kErrSort instead of hanging.  A look-back cut short under-counts a
// digit's exclusive prefix: its own pass still writes inside [0, n), but leaves
// slots of the output as they were, and a later pass may then hold more keys of
// a digit than the histogram of the original keys says, whose destinations run
// past n.  A tile's keys of such a digit go to the front of the output.  The output
// is not a permutation: the caller checks the status word before it uses the
// sorted indices.
#include <algorithm>

#include "pt_internal.cuh"

namespace pt {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Rounds of 32 keys per warp: 4096 keys per CTA, or 1024 where that leaves SMs
// without a CTA (a pass then waits for one CTA's 16 serial rounds).
constexpr int kSortRounds = 16, kSortRoundsSmall = 4;
constexpr int64_t kSortSmallMax = 1 << 19;
constexpr unsigned long long kFlagAggregate = 1ull << 32;
constexpr unsigned long long kFlagInclusive = 2ull << 32;
constexpr int kTagShift = 34;
// pass tags 1 .. kTags - 1; 0 = memory as it was cleared.  A clear every 127 sorts
// costs nothing to speak of, and an ordinary run starts the tags over.
constexpr unsigned kTags = 1u << 10;

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// All eight digit histograms in one read of the keys.
__global__ void __launch_bounds__(kSortThreads) radix_histograms(const uint64_t* __restrict__ keys, int64_t n,
                                                                 uint32_t* __restrict__ ghist) {
  __shared__ uint32_t h[8][256];
  for (int i = threadIdx.x; i < 8 * 256; i += kSortThreads) (&h[0][0])[i] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)kSortThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kSortThreads) {
    const uint64_t k = keys[i];
#pragma unroll
    for (int p = 0; p < 8; p++) atomicAdd(&h[p][(k >> (8 * p)) & 0xff], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 8 * 256; i += kSortThreads) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(&ghist[i], c);
  }
}

// Exclusive scan of each 256-bin histogram in place (block p = digit pass p).
__global__ void __launch_bounds__(256) radix_digit_offsets(uint32_t* __restrict__ ghist) {
  __shared__ uint32_t ws[8];
  uint32_t* g = ghist + blockIdx.x * 256;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t v = g[threadIdx.x];
  uint32_t inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  uint32_t base = 0;
  for (int q = 0; q < w; q++) base += ws[q];
  g[threadIdx.x] = base + inc - v;
}

template <int kRounds>
struct OnesweepShared {
  uint32_t wh[kSortWarps][256];  // per-warp digit counts, then their warp prefixes
  uint32_t dstart[256];          // tile-local start of each digit
  uint32_t gbase[256];           // global destination of each digit's first key of this tile
  uint32_t wsum[kSortWarps];
  int tile;
  uint64_t key[kSortThreads * kRounds];
  uint32_t val[kSortThreads * kRounds];
};

template <int kRounds>
__global__ void __launch_bounds__(kSortThreads, 2) radix_onesweep(const uint64_t* __restrict__ kin,
                                                                  const uint32_t* __restrict__ vin,
                                                                  uint64_t* __restrict__ kout,
                                                                  uint32_t* __restrict__ vout, int64_t n, int shift,
                                                                  const uint32_t* __restrict__ gofs,
                                                                  uint32_t* __restrict__ counter,
                                                                  unsigned long long* __restrict__ look,
                                                                  unsigned* __restrict__ status, long long spin_limit,
                                                                  unsigned tag) {
  constexpr int kTile = kSortThreads * kRounds;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Shared = OnesweepShared<kRounds>;
  Shared& S = *reinterpret_cast<Shared*>(smem_raw);
  const unsigned long long mine = (unsigned long long)tag << kTagShift;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortThreads) (&S.wh[0][0])[i] = 0;
  if (threadIdx.x == 0) S.tile = (int)atomicAdd(counter, 1u);
  __syncthreads();
  const int tile = S.tile;
  const int64_t tbase = (int64_t)tile * kTile;
  const int64_t base = tbase + (int64_t)w * (32 * kRounds);
  uint64_t k[kRounds];
  uint32_t v[kRounds];
  uint32_t rank[kRounds];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < kRounds; r++) {
    const int64_t i = base + r * 32 + lane;
    const bool ok = i < n;
    k[r] = ok ? kin[i] : 0ull;
    v[r] = ok ? vin[i] : 0u;
    const uint32_t d = ok ? (uint32_t)((k[r] >> shift) & 0xff) : (256u + lane);
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    uint32_t before = 0;
    if (ok) before = S.wh[w][d];
    rank[r] = before + __popc(peers & lt);
    __syncwarp();
    if (ok && (31 - __clz(peers)) == lane) S.wh[w][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // thread d: the tile's count of digit d and the warp prefixes
  const int d = threadIdx.x;
  uint32_t total = 0;
  for (int q = 0; q < kSortWarps; q++) {
    const uint32_t t = S.wh[q][d];
    S.wh[q][d] = total;
    total += t;
  }
  unsigned long long* my = look + (int64_t)tile * 256 + d;
  uint32_t excl = 0;
  if (tile == 0) {
    st_relaxed_u64(my, mine | kFlagInclusive | total);
  } else {
    st_relaxed_u64(my, mine | kFlagAggregate | total);
    // decoupled look-back over the earlier tiles
    int64_t pt = tile - 1;
    long long spins = 0;
    while (pt >= 0) {
      const unsigned long long s = ld_relaxed_u64(look + pt * 256 + d);
      const unsigned long long f = (s >> kTagShift) == tag ? s & (3ull << 32) : 0ull;
      if (f == 0) {
        if (++spins > spin_limit) {
          atomicOr(status, kErrSort);
          break;
        }
        __nanosleep(32);
        continue;
      }
      excl += (uint32_t)s;
      if (f == kFlagInclusive) break;
      pt--;
    }
    st_relaxed_u64(my, mine | kFlagInclusive | (unsigned long long)(excl + total));
  }
  // a destination past n, only behind a pass whose look-back gave up: the keys go to
  // the front instead (a test of every key's destination cost 12% of a pass)
  uint32_t first = gofs[d] + excl;
  if ((int64_t)first + total > n) {
    atomicOr(status, kErrSort);
    first = 0;
  }
  S.gbase[d] = first;
  // tile-local digit starts: exclusive scan of total over the 256 digits
  {
    uint32_t inc = total;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) S.wsum[w] = inc;
    __syncthreads();
    uint32_t b = 0;
    for (int q = 0; q < w; q++) b += S.wsum[q];
    S.dstart[d] = b + inc - total;
  }
  __syncthreads();
  // stage the ranked tile in shared memory
#pragma unroll
  for (int r = 0; r < kRounds; r++) {
    const int64_t i = base + r * 32 + lane;
    if (i < n) {
      const uint32_t dd = (uint32_t)((k[r] >> shift) & 0xff);
      const uint32_t pos = S.dstart[dd] + S.wh[w][dd] + rank[r];
      S.key[pos] = k[r];
      S.val[pos] = v[r];
    }
  }
  __syncthreads();
  const int cnt = (int)min((int64_t)kTile, n - tbase);
  for (int i = threadIdx.x; i < cnt; i += kSortThreads) {
    const uint64_t key = S.key[i];
    const uint32_t dd = (uint32_t)((key >> shift) & 0xff);
    const uint32_t dst = S.gbase[dd] + ((uint32_t)i - S.dstart[dd]);
    kout[dst] = key;
    vout[dst] = S.val[i];
  }
}

// ---------------------------------------------------------------- small sort
// Up to kRankMax keys: every key's place is the number of keys before it, counted
// against all of them (n^2 comparisons cost less than eight dependent digit
// passes, figures below).  A CTA places 64 keys, two
// per lane, its warps taking every 16th group of 16 keys.
constexpr int kRankThreads = 512;
constexpr int kRankWarps = kRankThreads / 32;
constexpr int kRankGroup = 16;
// sort and permutation by size, rank sort against digit passes: 4096 19 / 70 us,
// 10,000 38 / 81, 12,345 46 / 81, 16,000 56 / 82
constexpr int64_t kRankMax = 16384;

__global__ void __launch_bounds__(kRankThreads) rank_sort(const uint64_t* __restrict__ kin, uint64_t* __restrict__ kout,
                                                         uint32_t* __restrict__ vout, int64_t n) {
  __shared__ unsigned part[kRankWarps][64];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int base = blockIdx.x * 64, m = (int)n;
  uint64_t k[2];
  unsigned before[2] = {0, 0};
#pragma unroll
  for (int u = 0; u < 2; u++) k[u] = base + 32 * u + lane < m ? kin[base + 32 * u + lane] : ~0ull;
  // keys at lower indices come first when equal: all keys of a group below the
  // CTA's 64 count with <=, those above with <
  for (int g = kRankGroup * w; g < m; g += kRankGroup * kRankWarps) {
    uint64_t q[kRankGroup];
    if (g + kRankGroup <= m) {
#pragma unroll
      for (int h = 0; h < kRankGroup; h += 2) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(kin + g + h);
        q[h] = a.x;
        q[h + 1] = a.y;
      }
    } else {  // past the end: a key that counts for none
#pragma unroll
      for (int h = 0; h < kRankGroup; h++) q[h] = g + h < m ? kin[g + h] : ~0ull;
    }
    if (g + kRankGroup <= base) {
#pragma unroll
      for (int h = 0; h < kRankGroup; h++) {
        before[0] += q[h] <= k[0];
        before[1] += q[h] <= k[1];
      }
    } else if (g >= base + 64) {
#pragma unroll
      for (int h = 0; h < kRankGroup; h++) {
        before[0] += q[h] < k[0];
        before[1] += q[h] < k[1];
      }
    } else {
#pragma unroll
      for (int h = 0; h < kRankGroup; h++) {
        before[0] += q[h] < k[0] || (q[h] == k[0] && g + h < base + lane);
        before[1] += q[h] < k[1] || (q[h] == k[1] && g + h < base + 32 + lane);
      }
    }
  }
  part[w][lane] = before[0];
  part[w][32 + lane] = before[1];
  __syncthreads();
  const int i = base + (int)threadIdx.x;
  if (threadIdx.x < 64 && i < m) {
    unsigned r = 0;
#pragma unroll
    for (int q = 0; q < kRankWarps; q++) r += part[q][threadIdx.x];
    kout[r] = kin[i];
    vout[r] = (uint32_t)i;
  }
}

// ---------------------------------------------------------------- sort driver
namespace {
size_t align256(size_t b) { return (b + 255) / 256 * 256; }

template <int kRounds>
bool onesweep_passes(uint64_t* ka, uint32_t* va, uint64_t* kb, uint32_t* vb, int64_t n, const uint32_t* ghist,
                     uint32_t* counters, unsigned long long* look, unsigned* status, long long spin_limit, unsigned tag,
                     cudaStream_t st) {
  constexpr size_t kBytes = sizeof(OnesweepShared<kRounds>);
  static_assert(kBytes <= 227 * 1024, "onesweep tile exceeds shared memory");
  const int tiles = (int)((n + kSortThreads * kRounds - 1) / (kSortThreads * kRounds));
  if (cudaFuncSetAttribute(radix_onesweep<kRounds>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBytes) !=
      cudaSuccess)
    return false;
  for (int pass = 0; pass < 8; pass++) {
    note_launch();
    radix_onesweep<kRounds><<<tiles, kSortThreads, kBytes, st>>>(ka, va, kb, vb, n, 8 * pass, ghist + 256 * pass,
                                                                 counters + pass, look, status, spin_limit,
                                                                 tag + (unsigned)pass);
    uint64_t* tk = ka; ka = kb; kb = tk;
    uint32_t* tv = va; va = vb; vb = tv;
  }
  return true;
}

bool small_tiles(int64_t n) { return n <= kSortSmallMax; }
int64_t sort_tiles(int64_t n) {
  const int64_t tile = kSortThreads * (small_tiles(n) ? kSortRoundsSmall : kSortRounds);
  return std::max<int64_t>((n + tile - 1) / tile, 1);
}
}  // namespace

// Scratch of radix_sort_pairs for up to n keys: eight digit histograms, eight
// tile counters, and one 64-bit look-back word per (tile, digit); the caller
// clears it once, and again when it starts the tags over.
size_t sort_scratch_bytes(int64_t n) {
  const int64_t tiles = std::max(sort_tiles(n), sort_tiles(std::min(n, kSortSmallMax)));
  return align256(8 * 256 * sizeof(uint32_t)) + align256(8 * sizeof(uint32_t)) +
         align256((size_t)tiles * 256 * sizeof(unsigned long long));
}

unsigned sort_tags() { return kTags; }

// Sorts the keys k0 with their indices; (k0, v0) or (k1, v1) hold the result
// (returns 0 or 1, -1 on an error).  tag: the first of eight tags no sort on this
// scratch has used since it was cleared, 1 .. kTags - 8.
int radix_sort_pairs(uint64_t* k0, uint32_t* v0, uint64_t* k1, uint32_t* v1, int64_t n, void* scratch,
                     unsigned* status, int sms, long long spin_limit, unsigned tag, cudaStream_t st) {
  if (n <= 1) return 0;  // v0 holds the identity
  if (n <= kRankMax) {
    note_launch();
    rank_sort<<<(unsigned)((n + 63) / 64), kRankThreads, 0, st>>>(k0, k1, v1, n);
    return 1;
  }
  unsigned char* b = static_cast<unsigned char*>(scratch);
  uint32_t* ghist = reinterpret_cast<uint32_t*>(b);
  uint32_t* counters = reinterpret_cast<uint32_t*>(b + align256(8 * 256 * sizeof(uint32_t)));
  unsigned long long* look = reinterpret_cast<unsigned long long*>(
      b + align256(8 * 256 * sizeof(uint32_t)) + align256(8 * sizeof(uint32_t)));
  cudaMemsetAsync(ghist, 0, align256(8 * 256 * sizeof(uint32_t)) + align256(8 * sizeof(uint32_t)), st);
  note_launch();
  radix_histograms<<<(unsigned)std::min<int64_t>(sms * 4, (n + 2047) / 2048), kSortThreads, 0, st>>>(k0, n, ghist);
  note_launch();
  radix_digit_offsets<<<8, 256, 0, st>>>(ghist);
  const bool ok = small_tiles(n)
                      ? onesweep_passes<kSortRoundsSmall>(k0, v0, k1, v1, n, ghist, counters, look, status, spin_limit, tag, st)
                      : onesweep_passes<kSortRounds>(k0, v0, k1, v1, n, ghist, counters, look, status, spin_limit, tag, st);
  return ok ? 0 : -1;  // 8 passes: the result is back in (k0, v0)
}

// ---------------------------------------------------------------- permute
// All nine particle arrays through one read of the sorted indices.  With a status
// bit set (a sort that gave up leaves no permutation; a non-finite position) every
// particle stays where it is: the arrays keep a consistent state.
__global__ void __launch_bounds__(256) permute_particles(PermuteArrays a, const uint32_t* __restrict__ idx, int64_t n,
                                                        const unsigned* __restrict__ status) {
  const bool keep = *status != 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = keep ? i : (int64_t)idx[i];
    double v[8];
#pragma unroll
    for (int f = 0; f < 8; f++) v[f] = a.in[f][j];
    const int32_t o = a.order_in[j];
#pragma unroll
    for (int f = 0; f < 8; f++) a.out[f][i] = v[f];
    a.order_out[i] = o;
  }
}

void launch_permute(const PermuteArrays& a, const uint32_t* idx, int64_t n, const unsigned* status, int grid,
                    cudaStream_t st) {
  note_launch();
  permute_particles<<<grid, 256, 0, st>>>(a, idx, n, status);
}

}  // namespace pt
