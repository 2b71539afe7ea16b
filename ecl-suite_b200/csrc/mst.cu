// Minimum spanning forest (ECL-MST contract).
//
// Result contract (src/racefree/egr-input/MST/ECL-MST_10-atomic.cu): each
// undirected edge is represented by its v<n CSR entry j (:203) and ordered by
// the 64-bit key (weight << 32) | j (:248); with unique keys the minimum
// spanning forest is unique, so in_mst[] and the total weight equal cpuMST's
// Kruskal result (:112-154) bit for bit.  Light edges (weight <= a sampled
// threshold) are contracted first, then the rest (:331-360); any threshold
// gives the same forest.
//
// B200 design:
//  * mst_threshold: one block of mst_init samples 1024 weights and picks
//    the quantile that leaves ~0.75 n (1.5 n in a sparse graph) light CSR
//    entries, with no host round trip; below 4 entries a vertex there is one
//    pass over all entries instead of a light and a heavy one;
//  * mst_scan: builds a worklist of int4 {a, b, weight, j} from the CSR in
//    tiles of 256 entries a warp, whatever rows they belong to; appends are
//    staged per warp in shared memory and reserved in the global list with one
//    atomic per ~kStage entries;
//    the heavy pass drops entries whose endpoints are already joined (the
//    forest is flattened by pointer jumping first, so a root is one load);
//  * mst_boruvka: ALL Boruvka rounds in one cooperative persistent launch, three
//    phases a round with a bounded grid barrier after each: relabel the
//    edges and lower both roots' keys, hook every root along its smallest
//    edge, flatten the new trees.  Hooking writes one parent per root and
//    flattening keeps every tree one level deep, so finding an edge's roots
//    is one load each and no phase reads what it writes: the loads are plain
//    ones that L1 serves.  Per-round sizes live in a counter array, so no
//    counter is ever reset concurrently with its use.  The last, short rounds
//    are run by one block.
#include <algorithm>

#include "csr_bins.cuh"
#include "fill.cuh"
#include "flat_scan.cuh"
#include "grid_sync.cuh"
#include "solvers.cuh"

namespace ecl {
namespace {

using namespace dev;
typedef unsigned long long u64;

constexpr int kTPB = 256;
constexpr int kMaxRounds = 64;
// Light entries aimed at, in multiples of n: 0.75 from this average degree on,
// 1.5 below.  Rounds whose list does not shrink cost most; in a sparse random
// graph the light edges have to join most vertices (about n of them) before
// the heavy pass drops the bulk of its entries in the scan, while a power-law
// graph's hubs do that with few.  Measured, 0.75 / 1.5 / 2: G(3 M, 12 M) 1.94 /
// 1.02 / 0.95 ms, G(1 M, 3 M) 0.65 / 0.50 / 0.45, G(150 k, 600 k) 0.274 / 0.272 /
// 0.269, R-MAT-22 of degree 7 0.83 / 0.89 / 0.98, of degree 15 (scale 20) 0.455 /
// 0.443 / 0.472, of degree 30 1.67 / 1.69 / 1.78.
constexpr int kDenseDegree = 16;
constexpr int kSamples = 1024;

struct MSTCtl {
  GridBarrier bar;
  int wlcount[2][kMaxRounds + 2];    // [pass][round] sizes of the edge list
  int rootcount[2][kMaxRounds + 2];  // [pass][round] roots that may still have edges
  int threshold;
  u64 total;
  // %globaltimer when each pass started and after each of its barriers
  // (phases A, B and C of round r end at [3r + 1], [3r + 2] and [3r + 3]): a
  // per-round time profile that costs one store per barrier.
  u64 stamp[2][3 * kMaxRounds + 2];
};

__device__ __forceinline__ u64 mst_now() {
  u64 t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// parent[v] = root(v) between the passes, so the heavy scan reads each
// entry's root with one load.  Pointer jumping: each thread rewrites only its
// own parent[v], stepping to the parent of its current target, which its own
// thread is shortening at the same time (a vertex is a root iff it is its own
// parent; hooks may point either way in the ids).
__global__ void __launch_bounds__(kTPB) mst_flatten(int n, int* __restrict__ parent) {
  dep_wait();
  for (int v = blockIdx.x * kTPB + threadIdx.x; v < n; v += gridDim.x * kTPB) {
    int p = ld(&parent[v]);
    if (p == v) continue;
    int pp;
    while ((pp = ld(&parent[p])) != p) {
      st(&parent[v], pp);
      p = pp;
    }
  }
}

// Threshold = the k-th smallest of kSamples sampled weights, k chosen so the
// light pass keeps about light_factor * n of the m entries (the reference
// aims at 3n, ECL-MST_10-atomic.cu:450-459; the batched engine's autotuner
// may pick another factor -- the forest does not depend on it).
__device__ void mst_threshold(int n, int m, const int* eweight, MSTCtl* ctl, float light_factor) {
  __shared__ int s[kSamples];
  for (int t = threadIdx.x; t < kSamples; t += kTPB)
    s[t] = __ldg(&eweight[ecl_hash((unsigned)t * 2654435761u + 12345u) % (unsigned)m]);
  __syncthreads();
  for (int k = 2; k <= kSamples; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < kSamples / 2; i += kTPB) {
        const int t = 2 * i - (i & (j - 1)), p = t + j;  // the i-th pair j apart
        const int a = s[t], b = s[p];
        const bool up = (t & k) == 0;
        if ((a > b) == up) {
          s[t] = b;
          s[p] = a;
        }
      }
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) {
    const double frac = (double)light_factor * (double)n / (double)m;
    ctl->threshold = s[min(kSamples - 1, (int)(frac * kSamples))];
  }
}

// Also finds the rows of the scans' tiles (and so checks the CSR rows once: a
// malformed row raises ECL_ERR_BAD_GRAPH).  With a light pass to come, the
// first block finds its threshold meanwhile (in a launch of its own this took
// 7 to 10 us).
__global__ void __launch_bounds__(kTPB) mst_init(int n, int m, const int* __restrict__ nindex, int* __restrict__ parent,
                                                 u64* __restrict__ minv, int* __restrict__ tilerow,
                                                 const int* __restrict__ eweight, MSTCtl* __restrict__ ctl,
                                                 float light_factor, bool filter, Status* __restrict__ status) {
  dep_wait();
  if (filter && blockIdx.x == 0) {
    mst_threshold(n, m, eweight, ctl, light_factor);
    return;
  }
  const int first = ((int)blockIdx.x - filter) * kTPB + threadIdx.x, stride = ((int)gridDim.x - filter) * kTPB;
  for (int v = first; v < n; v += stride) {
    // race-free: thread-owned init, no reader in this launch
    parent[v] = v;
    minv[v] = ~0ull;
  }
  if (m > 0) flat_rows_range(n, m, nindex, tilerow, first & ~31, stride, status);
}

// Slots per warp in the shared-memory staging of worklist appends.
constexpr int kStage = 128;
// Worklists are 16 B per edge (100 MB each for R-MAT-22's light edges):
// they are written and read with evict-first hints so parent[] and the key
// arrays, which Boruvka reads at random, stay in L2.
typedef WarpStage<int4, kStage, true> Stage;

// More v<n entries than the worklist holds: an asymmetric graph flagged
// symmetric.
__device__ __forceinline__ void mst_overflow(bool overflow, Status* status) {
  if (__any_sync(kFull, overflow) && (threadIdx.x & 31) == 0) raise(status, ECL_ERR_BAD_GRAPH, -2);
}

// The worklist entries of a pass, from one pass over the CSR in tiles of 256
// entries a warp (flat_scan.cuh): the v < u entries of light weight, as they
// are; or, for the heavy pass, those whose ends lie in different components,
// as their roots.  The heavy pass loads an entry's root first and its weight
// only for entries between two components: the light pass joined the ends of
// every light entry (and checked every weight), so those are all heavy, and
// the ~80 % of entries inside one component cost no weight load.  parent[] is
// flat and not written in this launch, so its loads are read-only ones that L1
// serves.  Bound by instructions (about 450 a tile in the light scan, 650 in
// the heavy one) at the half of the warps that 48 and 64 registers leave: the
// entries and weights alone would take 0.13 ms at R-MAT-22 (128 M entries).
// The light scan takes 0.29 ms with five blocks an SM and 0.31 with four, the
// heavy one 0.54 with four and 0.55 with five (spilled registers).  One bit a
// vertex for "in the largest tree", looked up before the roots, did not make
// it faster (0.53 -> 0.53): the gathers are not the bound.  Before the flat
// tiles, rows per lane / warp / chunk record in two launches: light 0.55 ms,
// heavy (with the flattening) 0.86; 1000 vertices, 12 k entries: 36 us and 50,
// now 9 and 13.
template <bool kLight>
__global__ void __launch_bounds__(kTPB, kLight ? 5 : 4) mst_scan(FlatCsr g, bool vec, const int* __restrict__ eweight,
                                                 const int* parent, int4* __restrict__ wl, int cap, bool filter,
                                                 MSTCtl* ctl, Status* __restrict__ status) {
  dep_wait();
  __shared__ int4 stage_buf[kTPB / 32][kStage];
  __shared__ __align__(16) int s_mark[kTPB / 32][kFlatTile];
  const int wid = threadIdx.x >> 5;
  const int thr = filter ? ctl->threshold : 0x7fffffff;
  int* cnt = &ctl->wlcount[kLight ? 0 : 1][0];
  Stage stg{stage_buf[wid]};
  bool overflow = false;
  const int stop = min(g.m, __ldg(&g.nindex[g.n]));
  const int tiles = flat_tiles(g.m);
  for (int t = blockIdx.x * (kTPB / 32) + wid; t < tiles; t += gridDim.x * (kTPB / 32))
    flat_tile(g, stop, vec, t, s_mark[wid], [&](int e0, const int (&row)[kFlatLane], const int (&u)[kFlatLane]) {
      unsigned want = 0;  // bit k: entry k may be kept
#pragma unroll
      for (int k = 0; k < kFlatLane; k++) {
        if ((unsigned)u[k] >= (unsigned)g.n)
          raise(status, ECL_ERR_BAD_GRAPH, u[k]);
        else if (row[k] >= 0 && u[k] > row[k])
          want |= 1u << k;
      }
      int a[kFlatLane], b[kFlatLane], w[kFlatLane];
      if (!kLight) {
#pragma unroll
        for (int k = 0; k < kFlatLane; k++) b[k] = (want >> k) & 1u ? parent[u[k]] : -1;  // race-free: not written in this launch
#pragma unroll
        for (int k = 0; k < kFlatLane; k++) {
          a[k] = -1;
          if (!((want >> k) & 1u)) continue;
          a[k] = k > 0 && row[k] == row[k - 1] && a[k - 1] >= 0 ? a[k - 1] : parent[row[k]];  // race-free: as above
          if (a[k] == b[k]) want &= ~(1u << k);
        }
      }
      if (kLight && vec && want && e0 <= g.m - kFlatLane) {
        const int4 x = __ldcs(reinterpret_cast<const int4*>(eweight + e0));
        const int4 y = __ldcs(reinterpret_cast<const int4*>(eweight + e0 + 4));
        w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w, w[4] = y.x, w[5] = y.y, w[6] = y.z, w[7] = y.w;
      } else {
#pragma unroll
        for (int k = 0; k < kFlatLane; k++) w[k] = (want >> k) & 1u ? __ldcs(&eweight[e0 + k]) : 0;
      }
#pragma unroll
      for (int k = 0; k < kFlatLane; k++) {
        bool keep = (want >> k) & 1u;
        if (keep && w[k] < 0) {
          raise(status, ECL_ERR_BAD_GRAPH, e0 + k);
          keep = false;
        }
        if (kLight) keep = keep && w[k] <= thr;
        if (!keep) want &= ~(1u << k);
      }
      stg.template push_some<kFlatLane>(
          want, [&](int k) { return make_int4(kLight ? row[k] : a[k], kLight ? u[k] : b[k], w[k], e0 + k); }, wl, cnt, cap,
          overflow);
    });
  stg.flush(wl, cnt, cap, overflow);
  mst_overflow(overflow, status);
}

// A block's table of component roots (open addressing, kRootProbes probes)
// with the smallest key the block has for each.  Once a few hundred large
// components hold most of the edges, every thread of the grid publishes to
// the same few hundred key words, and a first touch of such a word by all of
// them queues at its L2 slice.  The table lowers a root's key in shared
// memory and publishes it with one atomic per block and round; a root whose
// probes meet only other roots goes to global memory directly, and so do all
// roots of a block whose first step finds few roots twice (most components
// still small: a table entry would then serve one edge).
constexpr int kBorTPB = 1024;    // one block a SM: 148 tables to publish, and 148 arrivals a barrier
constexpr int kBorBatch = 4;     // entries a thread keeps in flight
constexpr int kRootSlots = 2048;
constexpr int kRootProbes = 2;
constexpr size_t kBorSmem =
    sizeof(int4) * (kBorTPB / 32) * kStage + kRootSlots * (sizeof(u64) + sizeof(int)) + (kBorTPB / 32) * kStage * sizeof(int);

template <typename T>
using bref = cuda::atomic_ref<T, cuda::thread_scope_block>;

struct RootTable {
  int* root;  // kRootSlots entries, -1 = empty
  u64* key;

  // All threads of the block call, between block barriers.
  __device__ void reset() {
    for (int i = threadIdx.x; i < kRootSlots; i += blockDim.x) {
      root[i] = -1;  // race-free: block-owned, barrier-separated from every reader
      key[i] = ~0ull;
    }
  }
  // Lowers r's key in the table; false when r has no slot (the caller then
  // publishes it).  *seen: r had a slot already.
  __device__ bool lower(int r, u64 k, bool* seen) {
    int h = (int)(((unsigned)r * 2654435761u) >> 21);
    static_assert(kRootSlots == 1 << (32 - 21), "the slot is the hash's top bits");
    for (int p = 0; p < kRootProbes; p++, h = (h + 1) & (kRootSlots - 1)) {
      int c = bref<int>(root[h]).load(cuda::memory_order_relaxed);
      const bool mine = c == -1 && bref<int>(root[h]).compare_exchange_strong(c, r, cuda::memory_order_relaxed);
      if (mine || c == r) {
        *seen = !mine;
        if (bref<u64>(key[h]).load(cuda::memory_order_relaxed) > k)
          bref<u64>(key[h]).fetch_min(k, cuda::memory_order_relaxed);
        return true;
      }
    }
    return false;
  }
};

// Phase B for one entry: the root whose smallest key it is hooks to the other;
// of two that both chose it the smaller id stays a root.
__device__ __forceinline__ void mst_hook(const int4& e, u64 ka, u64 kb, int* parent, unsigned char* in_mst, u64& local) {
  const u64 key = ((u64)(unsigned)e.z << 32) | (unsigned)e.w;
  const bool ha = ka == key, hb = kb == key;
  if (!ha && !hb) return;
  if (ha && !(hb && e.x < e.y)) st(&parent[e.x], e.y);
  if (hb && !(ha && e.y < e.x)) st(&parent[e.y], e.x);
  in_mst[e.w] = 1;  // race-free: one entry j stands once in the list, and the flags are never read here
  local += (u64)(unsigned)e.z;
}

// The remaining rounds of a list of at most kSolo entries, by the first block
// alone: the same three phases with block barriers between them, the entries
// relabelled in place and the key words cleared by the entries that lowered
// them.  A short round is all latency, and the block's own rounds have no grid
// barriers, no list to write and no roots to list: 5 us each against 14 for the
// general form on one block.  Measured, the light pass's rounds, general form /
// kSolo = 512 / 2048 / 8192: R-MAT with 1 k vertices 64 / 24 / 25 / 24 us, with
// 2 k 57 / 57 / 49 / 47, G(5 k, 15 k) 98 / 98 / 85 / 134, G(20 k, 80 k) 124 /
// 123 / 124 / 154: one block is too narrow for longer lists.  An entry's two
// ends climbed one after another, link by link -> side by side, leaving what
// they reach to the others: a path of 2 k vertices with random weights 63 -> 55
// us, with equal ones, which all hook into one chain, 1284 -> 36.  All threads
// of the block call.
constexpr int kSolo = 2048;
constexpr int kSoloBatch = kSolo / kBorTPB;  // entries a thread keeps in flight: its share of the list

__device__ __noinline__ void mst_solo(int4* list, int sz, int& r, int* parent, u64* minv, unsigned char* in_mst,
                                      RootTable tab, u64& local) {
  bool lowered = false;
  for (; r < kMaxRounds; r++) {
    tab.reset();
    bool live = false;
    for (int i0 = threadIdx.x; i0 < sz; i0 += kBorTPB * kSoloBatch) {
      int2 e[kSoloBatch];
      int a[kSoloBatch], b[kSoloBatch];
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++) {
        const int i = i0 + k * kBorTPB;
        e[k] = i < sz ? *reinterpret_cast<const int2*>(&list[i]) : make_int2(-1, -1);
      }
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++) {
        if (e[k].x < 0) continue;
        if (lowered) {
          st(&minv[e[k].x], ~0ull);
          st(&minv[e[k].y], ~0ull);
        }
        a[k] = ld(&parent[e[k].x]);
        b[k] = ld(&parent[e[k].y]);
      }
      // All ends go up side by side, and what they reach they leave in their
      // parent words for the others: the entries can have hooked into one chain
      // as long as the list (equal weights along a path), of which every end so
      // leaves half at each step.
      unsigned go = 0;  // bits 2 k, 2 k + 1: entry k's ends are below a[k], b[k]
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++)
        if (e[k].x >= 0) go |= (a[k] != e[k].x ? 1u << (2 * k) : 0u) | (b[k] != e[k].y ? 2u << (2 * k) : 0u);
      while (go) {
        int pa[kSoloBatch], pb[kSoloBatch];
#pragma unroll
        for (int k = 0; k < kSoloBatch; k++) {
          if ((go >> (2 * k)) & 1u) pa[k] = ld(&parent[a[k]]);
          if ((go >> (2 * k)) & 2u) pb[k] = ld(&parent[b[k]]);
        }
#pragma unroll
        for (int k = 0; k < kSoloBatch; k++) {
          if ((go >> (2 * k)) & 1u) {
            if (pa[k] == a[k]) go &= ~(1u << (2 * k));
            else st(&parent[e[k].x], a[k] = pa[k]);
          }
          if ((go >> (2 * k)) & 2u) {
            if (pb[k] == b[k]) go &= ~(2u << (2 * k));
            else st(&parent[e[k].y], b[k] = pb[k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++) {
        if (e[k].x < 0) continue;
        if (a[k] == b[k]) a[k] = -1;
        live |= a[k] >= 0;
        *reinterpret_cast<int2*>(&list[i0 + k * kBorTPB]) = make_int2(a[k], b[k]);
      }
    }
    if (!__syncthreads_or(live)) break;
    for (int i = threadIdx.x; i < sz; i += kBorTPB) {
      const int4 e = list[i];  // race-free: this thread's own, relabelled before the block barrier
      if (e.x < 0) continue;
      const u64 key = ((u64)(unsigned)e.z << 32) | (unsigned)e.w;
      bool had;
      if (!tab.lower(e.x, key, &had)) fetch_min(&minv[e.x], key);
      if (!tab.lower(e.y, key, &had)) fetch_min(&minv[e.y], key);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRootSlots; i += kBorTPB) {
      const int rt = tab.root[i];  // race-free: claims ended at the barrier above
      if (rt >= 0) fetch_min(&minv[rt], tab.key[i]);
    }
    __syncthreads();
    for (int i0 = threadIdx.x; i0 < sz; i0 += kBorTPB * kSoloBatch) {
      int4 e[kSoloBatch];
      u64 ka[kSoloBatch], kb[kSoloBatch];
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++) {
        const int i = i0 + k * kBorTPB;
        e[k] = i < sz ? list[i] : make_int4(-1, -1, 0, 0);  // race-free: not written in this phase
      }
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++) {
        if (e[k].x < 0) continue;
        ka[k] = ld(&minv[e[k].x]);
        kb[k] = ld(&minv[e[k].y]);
      }
#pragma unroll
      for (int k = 0; k < kSoloBatch; k++)
        if (e[k].x >= 0) mst_hook(e[k], ka[k], kb[k], parent, in_mst, local);
    }
    lowered = true;
    __syncthreads();
  }
}

// Moves parent[v] (p as loaded) up v's tree by at most kJumps steps; true when
// it is the root.  The tree is fixed; every parent on it moves up meanwhile.
constexpr int kJumps = 32;

__device__ __forceinline__ bool mst_jump(int v, int p, int* parent) {
  for (int k = 0; k < kJumps; k++) {
    const int pp = ld(&parent[p]);
    if (pp == p) return true;
    st(&parent[v], pp);
    p = pp;
  }
  return false;
}

// All Boruvka rounds of one pass.  wlA holds the pass's initial worklist
// (size wlcount[pass][0]), whose entries join two distinct roots; later rounds
// alternate wlA / wlB.  A round has three phases, a grid barrier after each:
//   A  relabels each entry's ends with one load each (the roots are flat),
//      drops the entries inside one component, and lowers minv[root] of both
//      ends to the entry's key.  Round 0 takes the list as it stands.
//   B  hooks: the one entry that holds minv[a] sets parent[a] = b.  Keys are
//      unique, so each root is written by one entry, and the only cycles are
//      two roots that chose the same entry; the smaller of the two stays a root.
//   C  flattens: every root that took part jumps to its component's new root
//      and has its key word cleared; the new roots are listed for the next
//      round (round 0 looks at all vertices instead of a list).  A vertex goes
//      up kJumps steps and then waits until its thread has been through all of
//      its own: a tree can be as deep as the round has roots (a path whose
//      weights fall along it), and a thread that climbs on alone meets parents
//      that nobody has moved yet, one by one (1 M vertices: 464 ms; so, 0.17).
// Only phase B writes what phase A reads and the other way round, so the loads
// of parent[] in A and of minv[] in B are plain loads that the SM's L1 serves:
// with a union-find walked by relaxed atomic loads, every entry of a middle
// round ended its walk on the words of a few large components, and those L2
// slices were the bound.  Bound now by the random loads and atomics of phase A
// on the first two lists, and by three barriers a round on the short ones.
// Measured, light + heavy pass: R-MAT-22 1.52 -> 0.78 ms, G(150 k, 600 k)
// 0.89 -> 0.31 ms (its heavy pass 0.78 -> 0.22), 701 x 1031 grid 0.64 -> 0.34.
__global__ void __launch_bounds__(kBorTPB, 1) mst_boruvka(int n, int pass, int4* __restrict__ wlA, int4* __restrict__ wlB,
                                                          int cap, int* __restrict__ parent, u64* __restrict__ minv,
                                                          int* __restrict__ rootsA, int* __restrict__ rootsB,
                                                          unsigned char* __restrict__ in_mst, MSTCtl* __restrict__ ctl,
                                                          Status* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char s_bor[];
  __shared__ int s_seen;
  const int tid = blockIdx.x * kBorTPB + threadIdx.x;
  const int nthreads = gridDim.x * kBorTPB;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int* cnt = ctl->wlcount[pass];
  int* rcnt = ctl->rootcount[pass];
  int4* stage_buf = reinterpret_cast<int4*>(s_bor);
  u64* s_key = reinterpret_cast<u64*>(stage_buf + (kBorTPB / 32) * kStage);
  int* s_root = reinterpret_cast<int*>(s_key + kRootSlots);
  int* root_buf = s_root + kRootSlots;
  Stage stg{stage_buf + wid * kStage};
  WarpStage<int, kStage> rstg{root_buf + wid * kStage};
  RootTable tab{s_root, s_key};
  bool overflow = false;
  u64 local = 0;
  int r = 0;
  if (tid == 0) ctl->stamp[pass][0] = mst_now();
  for (; r < kMaxRounds; r++) {
    int4* in = (r == 0 || (r & 1)) ? wlA : wlB;
    int4* out = r == 0 ? wlA : ((r & 1) ? wlB : wlA);
    // a scan that overflowed (reported as BAD_GRAPH) counted more entries
    // than the list holds
    const int sz = min(ld(&cnt[r]), cap);
    if (sz == 0) break;  // the same for every thread: no phase writes cnt[r] any more
    if (sz <= kSolo) {
      if (blockIdx.x == 0) mst_solo(in, sz, r, parent, minv, in_mst, tab, local);
      break;
    }
    // ---- A
    tab.reset();
    if (threadIdx.x == 0) s_seen = 0;
    __syncthreads();
    bool use_tab = true;
    const int step = nthreads * kBorBatch;
    const int steps = (sz - 1) / step + 1;  // uniform over the grid: whole warps append together
    for (int s = 0; s < steps; s++) {
      // a warp's step takes kBorBatch slices of 32 consecutive entries
      const long long i0 = (long long)s * step + (long long)(tid - lane) * kBorBatch + lane;
      int4 e[kBorBatch];
#pragma unroll
      for (int k = 0; k < kBorBatch; k++) e[k] = i0 + 32 * k < sz ? __ldcs(&in[i0 + 32 * k]) : make_int4(-1, -1, 0, 0);
      if (r > 0) {
        int a[kBorBatch], b[kBorBatch];
#pragma unroll
        for (int k = 0; k < kBorBatch; k++) {
          a[k] = e[k].x >= 0 ? parent[e[k].x] : -1;  // race-free: parent[] is not written in phase A
          b[k] = e[k].x >= 0 ? parent[e[k].y] : -1;  // race-free: as above
        }
#pragma unroll
        for (int k = 0; k < kBorBatch; k++) {
          e[k].x = a[k] != b[k] ? a[k] : -1;
          e[k].y = b[k];
          stg.push(e[k].x >= 0, e[k], out, &cnt[r + 1], cap, overflow);
        }
      }
      int seen = 0;
      unsigned direct = 0;
#pragma unroll
      for (int k = 0; k < 2 * kBorBatch; k++) {
        const int4& x = e[k >> 1];
        if (x.x < 0) continue;
        bool had = false;
        const u64 key = ((u64)(unsigned)x.z << 32) | (unsigned)x.w;
        if (!use_tab || !tab.lower((k & 1) ? x.y : x.x, key, &had)) direct |= 1u << k;
        seen += had;
      }
      u64 cur[2 * kBorBatch];
#pragma unroll
      for (int k = 0; k < 2 * kBorBatch; k++)
        cur[k] = (direct >> k) & 1u ? ld(&minv[(k & 1) ? e[k >> 1].y : e[k >> 1].x]) : 0ull;
#pragma unroll
      for (int k = 0; k < 2 * kBorBatch; k++) {
        const int4& x = e[k >> 1];
        const u64 key = ((u64)(unsigned)x.z << 32) | (unsigned)x.w;
        if (cur[k] > key) fetch_min(&minv[(k & 1) ? x.y : x.x], key);
      }
      if (s == 0 && steps > 1) {
        seen = __reduce_add_sync(kFull, seen);
        if (lane == 0) atomicAdd(&s_seen, seen);  // shared memory
        __syncthreads();
        use_tab = s_seen >= kBorTPB * kBorBatch / 2;  // a quarter of the ends or more had a slot
      }
    }
    if (r > 0)
      stg.flush(out, &cnt[r + 1], cap, overflow);
    else if (tid == 0)
      st(&cnt[1], sz);  // round 1 reads round 0's list, whole
    // publish the block's table: one load (and at most one atomic) per root
    __syncthreads();
    for (int i = threadIdx.x; i < kRootSlots; i += kBorTPB) {
      const int rt = s_root[i];  // race-free: claims ended at the barrier above
      if (rt >= 0 && ld(&minv[rt]) > s_key[i]) fetch_min(&minv[rt], s_key[i]);
    }
    if (!grid_sync(&ctl->bar, status)) return;
    if (tid == 0) ctl->stamp[pass][3 * r + 1] = mst_now();
    const int nsz = ld(&cnt[r + 1]);
    if (nsz == 0) break;
    // ---- B
    for (long long i0 = tid; i0 < nsz; i0 += step) {
      int4 e[kBorBatch];
#pragma unroll
      for (int k = 0; k < kBorBatch; k++) {
        const long long i = i0 + (long long)k * nthreads;
        e[k] = i < nsz ? __ldcs(&out[i]) : make_int4(-1, -1, 0, 0);
      }
      u64 ka[kBorBatch], kb[kBorBatch];
#pragma unroll
      for (int k = 0; k < kBorBatch; k++) {
        ka[k] = e[k].x >= 0 ? minv[e[k].x] : 0ull;  // race-free: minv[] is not written in phase B
        kb[k] = e[k].x >= 0 ? minv[e[k].y] : 0ull;  // race-free: as above
      }
#pragma unroll
      for (int k = 0; k < kBorBatch; k++) {
        if (e[k].x >= 0) mst_hook(e[k], ka[k], kb[k], parent, in_mst, local);
      }
    }
    if (!grid_sync(&ctl->bar, status)) return;
    if (tid == 0) ctl->stamp[pass][3 * r + 2] = mst_now();
    // ---- C
    const int* rin = (r & 1) ? rootsA : rootsB;
    int* rout = (r & 1) ? rootsB : rootsA;
    const int nr = r == 0 ? n : ld(&rcnt[r]);
    bool left = false;  // one of this thread's vertices has not reached its root
    for (long long i0 = tid - lane; i0 < nr; i0 += nthreads) {  // whole warps: they append together
      const long long i = i0 + lane;
      int v = -1;
      if (i < nr) v = r == 0 ? (int)i : rin[i];  // race-free: written before the grid barrier
      bool root = false;
      if (v >= 0 && ld(&minv[v]) != ~0ull) {  // took part in this round
        st(&minv[v], ~0ull);
        const int p = ld(&parent[v]);
        root = p == v;
        left |= !root && !mst_jump(v, p, parent);
      }
      rstg.push(root, v, rout, &rcnt[r + 1], n, overflow);
    }
    rstg.flush(rout, &rcnt[r + 1], n, overflow);
    while (left) {
      left = false;
      for (long long i = tid; i < nr; i += nthreads) {
        const int v = r == 0 ? (int)i : rin[i];  // race-free: as above
        const int p = ld(&parent[v]);
        left |= p != v && !mst_jump(v, p, parent);
      }
    }
    if (!grid_sync(&ctl->bar, status)) return;
    if (tid == 0) ctl->stamp[pass][3 * r + 3] = mst_now();
  }
  if (r == kMaxRounds) raise(status, ECL_ERR_NO_CONVERGENCE, pass);
  // per-warp sum of the joined weights
  for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(kFull, local, o);
  if (lane == 0 && local) fetch_add(&ctl->total, local);
  if (threadIdx.x == 0) fetch_max(&status->rounds, r + 1);
}

struct MSTBufs {
  MSTCtl* ctl;
  int* parent;
  u64* minv;
  int* rootsA;
  int* rootsB;
  int* tilerow;
  int4* wlA;
  int4* wlB;
  int cap;
};

void mst_layout(Carve& c, int n, int m, bool symmetric, MSTBufs* b) {
  b->ctl = c.take<MSTCtl>(1);
  b->parent = c.take<int>((size_t)n);
  b->minv = c.take<u64>((size_t)n);
  b->rootsA = c.take<int>((size_t)n);
  b->rootsB = c.take<int>((size_t)n);
  b->tilerow = c.take<int>((size_t)flat_tiles(m) + 1);
  // v<n entries: at most m/2 in a symmetric, self-loop-free graph, else m.
  b->cap = symmetric ? m / 2 + 1 : (m > 0 ? m : 1);
  b->wlA = c.take<int4>((size_t)b->cap);
  b->wlB = c.take<int4>((size_t)b->cap);
}

}  // namespace

float mst_default_light(int n, int m) { return m / n >= kDenseDegree ? 0.75f : 1.5f; }

size_t mst_workspace_bytes(int n, int m) {
  Carve c;
  MSTBufs b;
  mst_layout(c, n, m, false, &b);
  return c.bytes();
}

ecl_status mst_enqueue(const GraphDev& g, unsigned char* in_mst, char* ws, Status* status, const DeviceInfo& dev,
                       cudaStream_t stream, unsigned long long** total_dev, Marker mark) {
  const bool sym = (g.flags & ECL_GRAPH_SYMMETRIC) != 0;
  Carve c{ws};
  MSTBufs b;
  mst_layout(c, g.n, g.m, sym, &b);
  // One block of 1024 threads per SM, fewer for a graph that gives each less
  // than 8 k vertices or entries: a barrier of few blocks is cheaper than the
  // work it would spread (R-MAT with 1000 vertices and 12 k entries).
  const int coop_grid = std::max(1, std::min(dev.sms, std::max(g.n, g.m) / 8192));
  ECL_CUDA_TRY(cudaFuncSetAttribute(mst_boruvka, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBorSmem));
  const int grid = dev.grid_blocks(kTPB, g.n, g.m);
  // 16-byte loads need 16-byte-aligned arrays (a lane's entries start at a multiple of 8)
  const bool vec = ((reinterpret_cast<uintptr_t>(g.nlist) | reinterpret_cast<uintptr_t>(g.eweight)) & 15) == 0;
  const int scan_grid = dev.grid_blocks(kTPB, 0, g.m);  // a thread per lane's share of a tile
  const FlatCsr fc{g.n, g.m, g.nindex, g.nlist, b.tilerow};
  if (total_dev) *total_dev = &b.ctl->total;
  fill_ranges({{b.ctl, sizeof(MSTCtl), 0},
               {in_mst, (size_t)g.m, 0},
               {b.tilerow, sizeof(int) * ((size_t)flat_tiles(g.m) + 1), 0xff}},
              dev, stream);
  // No light pass below 4 entries a vertex: all weights pass the first scan,
  // and the second would find nothing.
  const bool filter = g.m / g.n >= 4;
  const float light = dev.mst_light_factor > 0.f ? dev.mst_light_factor : mst_default_light(g.n, g.m);
  ECL_LAUNCH_NEXT(mst_init, grid + filter, kTPB, 0, stream, g.n, g.m, g.nindex, b.parent, b.minv, b.tilerow, g.eweight,
                  b.ctl, light, filter, status);
  if (g.m > 0) {
    mark();
    for (int pass = 0; pass < 2; pass++) {
      if (pass == 1 && !filter) {
        mark();
        mark();
        break;
      }
      if (pass == 0) {
        ECL_LAUNCH_NEXT(mst_scan<true>, scan_grid, kTPB, 0, stream, fc, vec, g.eweight, b.parent, b.wlA, b.cap, filter,
                        b.ctl, status);
      } else {
        ECL_LAUNCH_NEXT(mst_flatten, grid, kTPB, 0, stream, g.n, b.parent);
        ECL_LAUNCH_NEXT(mst_scan<false>, scan_grid, kTPB, 0, stream, fc, vec, g.eweight, b.parent, b.wlA, b.cap, filter,
                        b.ctl, status);
      }
      mark();
      ECL_CUDA_TRY(launch_cooperative_smem(mst_boruvka, coop_grid, kBorTPB, kBorSmem, stream, g.n, pass, b.wlA,
                                           b.wlB, b.cap, b.parent, b.minv, b.rootsA, b.rootsB, in_mst, b.ctl, status));
      mark();
    }
  }
  return ECL_OK;
}

}  // namespace ecl

extern "C" ecl_status ecl_mst(const ecl_graph_view* g, uint8_t* in_mst_out, uint64_t* total_weight, ecl_opts* opts) {
  using namespace ecl;
  ecl_opts local{};
  if (!opts) opts = &local;
  if (!in_mst_out && g && g->edges > 0) return ECL_ERR_INVALID_ARG;
  Solve s(g, opts);
  GraphNeeds needs;
  needs.weights = true;
  const bool sym = g && (g->flags & ECL_GRAPH_SYMMETRIC);
  size_t wsb = 0;
  if (g && g->nodes >= 1 && g->edges >= 0) {
    Carve c;
    MSTBufs b;
    mst_layout(c, g->nodes, g->edges, sym, &b);
    wsb = c.bytes();
  }
  ecl_status st = s.begin(needs, wsb);
  if (st != ECL_OK) return s.finish(st);
  unsigned char* in_mst = s.output(in_mst_out, (size_t)(s.m > 0 ? s.m : 1));
  if (!in_mst) return s.finish(ECL_ERR_OOM);
  GraphDev gd;
  gd.n = s.n;
  gd.m = s.m;
  gd.nindex = s.nindex;
  gd.nlist = s.nlist;
  gd.eweight = s.eweight;
  gd.flags = g->flags;
  u64* total_dev = nullptr;
  u64 hostTotal = 0;
  s.start_timer();
  st = mst_enqueue(gd, in_mst, s.ws, s.status, s.dev, s.stream, &total_dev, Marker{&s});
  s.stop_timer();
  if (st == ECL_OK && total_weight && total_dev) {
    if (cudaMemcpyAsync(&hostTotal, total_dev, sizeof(u64), cudaMemcpyDeviceToHost, s.stream) != cudaSuccess)
      st = ECL_ERR_CUDA;
  }
  st = s.finish(st);
  if (total_weight) *total_weight = (st == ECL_OK) ? hostTotal : 0;
  return st;
}

extern "C" ecl_status ecl_compute_mst(int32_t nodes, int32_t edges, const int32_t* nidx, const int32_t* nlist,
                                      const int32_t* eweight, uint8_t* in_mst) {
  ecl_graph_view g{nodes, edges, nidx, nlist, eweight, ECL_HOST, 0};
  ecl_opts o{};
  return ecl_mst(&g, in_mst, nullptr, &o);
}
