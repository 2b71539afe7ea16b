// Strongly connected components (ECL-SCC contract).
//
// Result contract (src/racefree/mesh-input/ECL-SCC_10-atomic.cu): the
// reference keeps, per vertex, the largest id that reaches it (in-max) and the
// largest id it reaches (out-max) within the current edge set, propagates both
// to a fixpoint (:132-172), retires vertices whose two values agree, drops
// edges whose endpoints disagree (:175-195), resets the rest (:198-214) and
// repeats.  A vertex retires exactly when the largest id of its SCC reaches it
// and is reached by it, so the label it reports, readFirst(iomax[v]) (:318),
// is the largest vertex id of v's SCC -- schedule independent.
//
// B200 design:
//  * graphs flagged symmetric are first tried as connected components, and in
//    a large graph the component of the vertex with the most entries is found
//    by a forward and a backward search (both below); what follows is for the
//    edges that are left;
//  * scc_mark trims first: a vertex with no in-entry or no out-entry
//    (self-loops ignored) is its own SCC and contributes no edge.  The same
//    pass writes the int2 edge list in CSR positions -- slot i holds
//    (v, nlist[i]), or a dead slot for a self-loop or a bad id -- so the list
//    costs one streaming store per entry and no separate pass (on R-MAT nearly
//    every edge survives the trim, so compacting it would buy nothing).  Rows
//    are degree-binned (lane / warp / 256-entry chunk records), so hub rows
//    spread over all warps;
//  * scc_solve runs EVERY propagation sweep and every trimming round in one
//    cooperative persistent launch, separated by bounded grid barriers (the
//    reference pays a host round trip per propagation launch, :283-287).
//    In-max and out-max of a vertex share one 64-bit word (in-max high, out-
//    max low), like the reference's iomax, so an edge costs two word loads
//    plus two for the jumps io[in-max(v)] / io[out-max(w)] (both still valid
//    bounds, so values travel many hops per sweep); a raise is a 32-bit
//    atomic max on one half.  Trimmed vertices hold a DEAD word that every
//    sweep skips.  Each lane keeps kSweepBatch edges' loads in flight (a
//    launch knob: 1, 2 or 4; fewer edges a lane leave more lanes resident);
//  * rounds after the first sweep only the surviving edges (the edges whose
//    two ends share both values and are unresolved: io[v] == io[w]); every
//    sweep appends the edges it would keep, and the round's last sweep --
//    which raised nothing, so it read final words -- leaves the next round's
//    list without a separate pass;
//  * the final labels are written by the same launch (label = in-max).
#include <algorithm>
#include <type_traits>

#include "csr_bins.cuh"
#include "fill.cuh"
#include "flat_scan.cuh"
#include "grid_sync.cuh"
#include "solvers.cuh"

namespace ecl {
namespace {

using namespace dev;

constexpr int kTPB = 256;
constexpr int kMaxSweeps = 1 << 16;
constexpr int kScanBatch = 4;  // list entries per lane whose loads are issued together

constexpr int kStamps = 256;
constexpr int kGiantLevels = 40;
constexpr int kGiantRounds = 40;

struct SCCCtl {
  GridBarrier bar;        // scc_solve's
  GridBarrier giant_bar;  // scc_giant's (another grid: a barrier counts in multiples of one)
  unsigned long long asym;  // scc_symmetry's sum: 0 iff every entry has its reverse
  // scc_giant
  unsigned long long pivot;  // (out-degree << 32) | ~id of the vertex with the most entries
  int giant_ok;              // 1: the pivot's component is found
  int giant_label;           // its largest id
  int rest;                  // edges scc_mark<true> kept for scc_solve
  int level_new[kGiantLevels];     // per forward level: vertices it added to the queue
  int level_chunks[kGiantLevels];  // ... and chunk records of its long rows
  int left[kGiantRounds + 1];  // per backward round: vertices not known to reach the pivot
  int moved[kGiantRounds];     // per backward round: some vertex was found to reach it
  int back_chunks[kGiantRounds];   // ... and chunk records of its long rows
  int pad[64];
  // %globaltimer at the start and after each grid barrier (the first
  // kStamps - 1): a time profile of sweeps, compactions and retirements that
  // costs one store per barrier
  unsigned long long stamp[kStamps];
  int changed[kMaxSweeps];   // per-sweep "something moved" flags
  int raised[kMaxSweeps];    // per-sweep counts of raises
  int kept[kMaxSweeps];      // per-sweep sizes of the list of edges a round keeps
  int again[kMaxSweeps];     // per-round "vertices left" flags, indexed by the round's last sweep
};

__device__ __forceinline__ unsigned long long scc_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// In-max (high half) and out-max (low half) of one vertex.
__device__ __forceinline__ unsigned long long io_pack(int in, int out) {
  return ((unsigned long long)(unsigned)in << 32) | (unsigned)out;
}
__device__ __forceinline__ int io_in(unsigned long long x) { return (int)(x >> 32); }
__device__ __forceinline__ int io_out(unsigned long long x) { return (int)(unsigned)x; }

// Raises the in-max (kIn) or out-max half of *p to val when `old`, the word
// last read, is below it; true when it was.  The raise is a 32-bit atomic max
// on that half: a word is read whole and raised per half, the reference's own
// access pattern (readFirst / writeFirstA on iomax, ECL-SCC_10-atomic.cu:145-
// 160), and a max never lowers a value another thread raised meanwhile.
template <bool kIn>
__device__ __forceinline__ bool io_raise(unsigned long long* p, unsigned long long old, int val) {
  if ((kIn ? io_in(old) : io_out(old)) >= val) return false;
  fetch_max(reinterpret_cast<int*>(p) + (kIn ? 1 : 0), val);  // little-endian: high half at +1
  return true;
}

// ---- symmetric graphs ----
//
// In a graph whose entries all have their reverses the strongly connected
// components are the connected ones: CC labels them with their smallest ids,
// and two passes over the vertices turn those into the largest.  Otherwise
// every sweep over all edges moves the largest id a few hops on (ten sweeps
// for a 701 x 1031 grid, 97 for a union of many grids).
// The caller's ECL_GRAPH_SYMMETRIC flag says when this is worth looking for,
// but SCC has never relied on it, so it is checked: the sum over all entries
// (v, u) of +h(v, u) where v < u and -h(u, v) where v > u, modulo 2^64 with a
// 64-bit hash h of the pair, is 0 for every symmetric entry list; a list that
// is not symmetric makes it 0 once in 2^64.  Any other sum, and the launches of
// the union-find leave at once and the general path below runs.  Measured,
// general -> this: 701 x 1031 grid 0.37 -> 0.17 ms, a union of 32 grids of 1.1 M
// vertices 4.5 ms -> about 0.2.  A directed graph that carries the flag pays for
// the check and for launches with nothing to do: R-MAT-20 (16 M edges) 0.35 ->
// 0.45 ms, R-MAT-16 0.18 -> 0.22.

// Mixing function of splitmix64 (Steele, Lea and Flood, OOPSLA 2014).
__device__ __forceinline__ unsigned long long scc_mix(unsigned long long x) {
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__global__ void __launch_bounds__(kTPB) scc_rows(int n, int m, const int* __restrict__ nindex,
                                                 int* __restrict__ tilerow, Status* __restrict__ status) {
  dep_wait();
  flat_rows_range(n, m, nindex, tilerow, (blockIdx.x * kTPB + threadIdx.x) & ~31, gridDim.x * kTPB, status);
}

// Bound by the one read of the entries: the hash is about 20 instructions each.
__global__ void __launch_bounds__(kTPB) scc_symmetry(FlatCsr g, bool vec, SCCCtl* ctl,
                                                     Status* __restrict__ status) {
  dep_wait();
  __shared__ __align__(16) int s_mark[kTPB / 32][kFlatTile];
  __shared__ unsigned long long s_sum[kTPB / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int stop = min(g.m, __ldg(&g.nindex[g.n]));
  const int tiles = flat_tiles(g.m);
  unsigned long long sum = 0;
  for (int t = blockIdx.x * (kTPB / 32) + wid; t < tiles; t += gridDim.x * (kTPB / 32))
    flat_tile(g, stop, vec, t, s_mark[wid], [&](int, const int (&row)[kFlatLane], const int (&u)[kFlatLane]) {
#pragma unroll
      for (int k = 0; k < kFlatLane; k++) {
        if (row[k] < 0 || u[k] == row[k]) continue;
        if ((unsigned)u[k] >= (unsigned)g.n) {
          raise(status, ECL_ERR_BAD_GRAPH, u[k]);
          continue;
        }
        const unsigned lo = min(row[k], u[k]), hi = max(row[k], u[k]);
        const unsigned long long h = scc_mix(((unsigned long long)hi << 32 | lo) + 0x9e3779b97f4a7c15ull);
        sum += row[k] < u[k] ? h : 0ull - h;
      }
    });
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(kFull, sum, o);
  if (lane == 0) s_sum[wid] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kTPB / 32; w++) sum += s_sum[w];
    if (sum) fetch_add(&ctl->asym, sum);
  }
}

// Smallest -> largest id, first pass: top[r] (zeroed before) = the largest id
// above r of the component that CC labelled r.  Warps go through the vertices
// from the last to the first, so the first id a lane meets of a component is
// the largest it will meet, and of a warp's lanes in the highest lane's
// component only that lane counts: the giant component's word then takes one
// access per warp of the launch, not one per vertex.
__global__ void __launch_bounds__(kTPB) scc_top(int n, const int* comp, int* __restrict__ top,
                                                const SCCCtl* ctl) {
  dep_wait();
  if (ctl->asym != 0) return;  // as scc_mark
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5, nwarps = (gridDim.x * kTPB) >> 5;
  const int groups = (n - 1) / 32 + 1;
  int seen = -1;  // component that this lane or, for it, its warp's highest lane dealt with last
  for (int q = groups - 1 - warp; q >= 0; q -= nwarps) {
    const int v = 32 * q + lane;
    const int r = v < n ? comp[v] : -1;  // race-free: not written in this launch
    const unsigned in = __ballot_sync(kFull, r >= 0);
    const int top_lane = 31 - __clz(in);
    const int high = __shfl_sync(kFull, r, top_lane);
    const bool covered = r == high && lane != top_lane;
    if (r >= 0 && r != v && r != seen && !covered && ld(&top[r]) < v) fetch_max(&top[r], v);
    if (r >= 0) seen = r;
  }
}

__global__ void __launch_bounds__(kTPB) scc_relabel(int n, int* comp, const int* top,
                                                    const SCCCtl* ctl, Status* __restrict__ status) {
  dep_wait();
  if (ctl->asym != 0) return;  // as scc_mark
  if (blockIdx.x == 0 && threadIdx.x == 0) st(&status->rounds, 1);  // no sweep: one pass of hooking
  for (int v = blockIdx.x * kTPB + threadIdx.x; v < n; v += gridDim.x * kTPB) {
    const int r = comp[v];  // race-free: thread-owned
    comp[v] = max(r, top[r]);  // race-free: thread-owned; top is not written in this launch
  }
}

// ---- the giant component ----
//
// Most directed graphs that are not meshes have one component with most of the
// edges.  Before any propagation scc_giant finds the component of the vertex
// with the most out-entries: the vertices it reaches (forward search over a
// queue, every edge looked at once), and of those the ones that reach it (each
// looks for one out-neighbour known to, and stops at the first: two or three
// entries a vertex).  What is left for the propagation sweeps -- each of them
// two random words for every edge -- is the few edges between other vertices
// on the same side of the search.  The search gives up, and the sweeps run on
// all edges as before, where it would take long or find little: forward after
// kGiantLevels levels, with few vertices reached by level kGiantPatience, or
// when two levels in a row neither grow nor shrink much while most vertices are
// still unreached (meshes and layers; a random graph's levels grow until they
// hold much of it); backward when most vertices are still candidates and a round
// after the first finds hardly any, or the candidates looked through add up to
// twice n and the number found does not grow (a few vertices that reach the
// pivot one after another, above many that do not: 0.52 -> 0.44 ms of 2.2 lost).
// Bound by the latency of the two widest levels' look-ups (a third of the time
// each at R-MAT-22).  Measured, whole solve, sweeps over all edges -> this:
// directed R-MAT-22 (65 M edges) 2.47 -> 0.83 ms, 500 k vertices (5.7 M) 0.58
// -> 0.33, G(3 M, 12 M) 2.14 -> 1.45; a 701 x 1031 grid without cycles, where
// it gives up, 17.3 -> 17.4.
constexpr int kGTPB = 512;
constexpr int kGiantPatience = 16;
// Entries from which on the search is tried: kGiantEntries where the pivot is a
// hub (kGiantHub times the average degree), and from kGiantFlat on without one,
// as a graph without hubs has more levels for its size.  With hubs: R-MAT with
// 0.45 M entries 229 -> 227 us, 1.05 M 266 -> 250, 1.8 M 363 -> 261.  Without:
// G(300 k, 1.2 M) 441 -> 528, G(600 k, 2.4 M) 659 -> 595, G(1 M, 4 M) 1078 -> 711.
// What is lost where it finds nothing, or half of what there is: an acyclic graph
// of 300 k vertices and 3 M random edges 907 -> 1002, two random graphs of 300 k
// vertices side by side 655 -> 849, 3 M edges from power-law ends 562 -> 643.
constexpr int kGiantEntries = 1 << 20;
constexpr int kGiantFlat = 1 << 21;
constexpr int kGiantHub = 32;
constexpr int kGiantLong = 256;   // longer rows are cut into chunk records of this many entries
constexpr int kBackLong = 1024;   // ... backward, where most rows are left after a few entries, only rows longer than this

struct Giant {
  unsigned* fwd;  // bit per vertex: reached from the pivot
  unsigned* bwd;  // bit per vertex: reaches the pivot (complete inside fwd)
  // race-free: not written where this is called
  __device__ __forceinline__ bool has(const unsigned* bits, int v) const { return (bits[v >> 5] >> (v & 31)) & 1u; }
  // After scc_giant's launch.
  __device__ __forceinline__ bool in(int v) const { return has(fwd, v) && has(bwd, v); }
};

// Visits the entries of 32 rows, one per lane ([beg, beg + deg)), spread evenly
// over the warp: f(owner, j, valid) for entry j of lane `owner`'s row, four
// steps of 32 consecutive entries per call round.  All lanes call f together.
template <class F>
__device__ __forceinline__ void warp_rows(int beg, int deg, F&& f) {
  const int lane = threadIdx.x & 31;
  int incl = deg;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += x;
  }
  const int excl = incl - deg, total = __shfl_sync(kFull, incl, 31);
  for (int base = 0; base < total; base += 128) {
    int owner[4], j[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int e = base + 32 * k + lane;
      int lo = 0;  // the last lane whose row starts at or before e
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(kFull, excl, lo + o) <= e) lo += o;
      owner[k] = lo;
      j[k] = __shfl_sync(kFull, beg, lo) + e - __shfl_sync(kFull, excl, lo);
      if (e >= total) j[k] = -1;
    }
    f(owner, j);
  }
}

// bits |= next, next = 0, for all words; the caller's barriers are around it.
__device__ __forceinline__ void merge_bits(unsigned* bits, unsigned* next, int words, int tid, int nthreads) {
  for (int i = tid; i < words; i += nthreads) {
    const unsigned x = ld(&next[i]);
    if (x == 0) continue;
    bits[i] |= x;  // race-free: word i is this thread's between the barriers
    st(&next[i], 0u);
  }
}

// The bits that a level (round) finds go to `next`, and fwd (bwd) is not
// written before its end: looking a vertex up first there is a plain load that
// L1 serves.  The hubs that most edges lead to are found in the first levels;
// looked up by relaxed loads, the few words that hold their bits were the
// bound (R-MAT-22: 1.18 ms for the whole search against 0.6).
__global__ void __launch_bounds__(kGTPB, 3) scc_giant(int n, int m, const int* __restrict__ nindex,
                                                      const int* __restrict__ nlist, unsigned* fwd, unsigned* bwd,
                                                      unsigned* next, int* queue, int* candA, int* candB, int2* chunks,
                                                      int chunk_cap, SCCCtl* ctl, bool checked,
                                                      Status* __restrict__ status) {
  if (checked && ctl->asym == 0) return;  // as scc_mark
  __shared__ int s_stage[kGTPB / 32][128];
  __shared__ int s_moved;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int tid = blockIdx.x * kGTPB + threadIdx.x, nthreads = gridDim.x * kGTPB;
  const int warp = tid >> 5, nwarps = nthreads >> 5;
  const int words = (n + 31) / 32;
  WarpStage<int, 128> stg{s_stage[wid]};
  bool overflow = false;
  // row of v; a malformed one (reported by scc_mark) is empty
  auto row_of = [&](int v, int& beg, int& deg) {
    beg = __ldg(&nindex[v]);
    const int end = __ldg(&nindex[v + 1]);
    deg = end - beg;
    if (beg < 0 || end < beg || end > m) beg = deg = 0;
  };
  // no bit set yet
  for (int i = tid; i < words; i += nthreads) fwd[i] = bwd[i] = next[i] = 0;  // race-free: thread-owned, barrier next
  // the pivot
  unsigned long long key = 0;
  for (int v = tid; v < n; v += nthreads) {
    int beg, deg;
    row_of(v, beg, deg);
    key = max(key, ((unsigned long long)deg << 32) | (0xffffffffu - (unsigned)v));
  }
  for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(kFull, key, o));
  if (lane == 0 && key > ld(&ctl->pivot)) fetch_max(&ctl->pivot, key);
  if (!grid_sync(&ctl->giant_bar, status)) return;
  key = ld(&ctl->pivot);
  if ((key >> 32) == 0) return;  // no entries at all
  if (m < kGiantFlat && (long long)(key >> 32) < (long long)kGiantHub * (m / n + 1)) return;
  const int pivot = (int)(0xffffffffu - (unsigned)key);
  if (tid == 0) {
    fetch_or(&fwd[pivot >> 5], 1u << (pivot & 31));
    fetch_or(&bwd[pivot >> 5], 1u << (pivot & 31));
    queue[0] = pivot;  // race-free: one thread, read behind the next grid barrier
  }
  if (!grid_sync(&ctl->giant_bar, status)) return;
  int qs = 0, qe = 1, level = 0;
  int flat = 0;  // levels in a row that neither grew nor shrank much
  // chunk records of the frontier's long rows
  auto cut_long_rows = [&]() {
    const RowChunks rc{chunks, &ctl->level_chunks[level], chunk_cap};
    for (int i0 = qs + warp * 32; i0 < qe; i0 += nwarps * 32) {
      const int i = i0 + lane;
      const int v = i < qe ? queue[i] : 0;  // race-free: written before the last grid barrier
      int beg = 0, deg = 0;
      if (i < qe) row_of(v, beg, deg);
      push_chunks_warp(rc, kGiantLong, deg > kGiantLong, v, beg, beg + deg, status);
    }
  };
  // the entries j[k] of the rows of v[k]: newly reached vertices join the queue
  // behind its present end (counted per level: a block may still be reading the
  // last level's count when another one is adding to the next), and an entry
  // that is the pivot says that v[k] reaches it
  auto reach = [&](auto count, const int* v, const int* j) {
    constexpr int K = decltype(count)::value;
    int w[K];
    unsigned have[K];
#pragma unroll
    for (int k = 0; k < K; k++) w[k] = j[k] >= 0 ? __ldg(&nlist[j[k]]) : -1;
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (j[k] >= 0 && (unsigned)w[k] >= (unsigned)n) {
        raise(status, ECL_ERR_BAD_GRAPH, w[k]);
        w[k] = -1;
      }
      have[k] = w[k] >= 0 ? fwd[w[k] >> 5] : ~0u;  // race-free: not written during a level
    }
#pragma unroll
    for (int k = 0; k < K; k++)
      if (!((have[k] >> (w[k] & 31)) & 1u)) have[k] = ld(&next[w[k] >> 5]);
#pragma unroll
    for (int k = 0; k < K; k++) {
      const unsigned bit = 1u << (w[k] & 31);
      const bool found = !(have[k] & bit) && !(fetch_or(&next[w[k] >> 5], bit) & bit);
      if (w[k] == pivot) fetch_or(&bwd[v[k] >> 5], 1u << (v[k] & 31));
      if (__any_sync(kFull, found)) stg.push(found, w[k], queue + qe, &ctl->level_new[level], n - qe, overflow);
    }
  };
  cut_long_rows();
  if (!grid_sync(&ctl->giant_bar, status)) return;
  for (; qs < qe; level++) {
    if (level + 1 == kGiantLevels || (level == kGiantPatience && qe < n / 64)) return;  // long distances: not this way
    const int nch = chunk_total(RowChunks{chunks, &ctl->level_chunks[level], chunk_cap});
    for (int c = warp; c < nch; c += nwarps) {
      const int2 r = chunks[c];  // race-free: written before the last grid barrier
      const int end = min(r.y + kGiantLong, __ldg(&nindex[r.x + 1]));
      constexpr int K = kGiantLong / 32;
      int vv[K], j[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        vv[k] = r.x;
        j[k] = r.y + 32 * k + lane < end ? r.y + 32 * k + lane : -1;
      }
      reach(std::integral_constant<int, K>{}, vv, j);
    }
    // a warp takes up to 32 rows at a time, fewer while there are not enough
    // for all warps (the hubs stand side by side in the queue)
    const int per = min(32, (qe - qs - 1) / nwarps + 1);
    for (int i0 = qs + warp * per; i0 < qe; i0 += nwarps * per) {
      const int i = lane < per ? i0 + lane : qe;
      const int v = i < qe ? queue[i] : 0;  // race-free: written before the last grid barrier
      int beg = 0, deg = 0;
      if (i < qe) row_of(v, beg, deg);
      if (deg > kGiantLong) deg = 0;  // in chunk records
      warp_rows(beg, deg, [&](const int (&owner)[4], const int (&j)[4]) {
        int vv[4];
#pragma unroll
        for (int k = 0; k < 4; k++) vv[k] = __shfl_sync(kFull, v, owner[k]);
        reach(std::integral_constant<int, 4>{}, vv, j);
      });
    }
    stg.flush(queue + qe, &ctl->level_new[level], n - qe, overflow);
    if (!grid_sync(&ctl->giant_bar, status)) return;
    merge_bits(fwd, next, words, tid, nthreads);
    const int last = qe - qs, fresh = ld(&ctl->level_new[level]);
    qs = qe;
    qe += fresh;
    flat = level >= 4 && qe < n / 8 && 4LL * fresh < 5LL * last && 2LL * fresh >= last ? flat + 1 : 0;
    if (flat == 2) return;
    level++;
    cut_long_rows();
    level--;
    if (!grid_sync(&ctl->giant_bar, status)) return;
  }
  // backward, inside the vertices reached
  int cnt = qe, cnt1 = 0, found0 = 0;  // candidates, those after the first round, the round before's finds
  long long looked = 0;
  for (int round = 0;; round++) {
    if (round == kGiantRounds) return;
    const int* in = round == 0 ? queue : ((round & 1) ? candA : candB);
    int* out = (round & 1) ? candB : candA;
    bool moved = false;
    if (threadIdx.x == 0) s_moved = 0;
    __syncthreads();
    auto reaches = [&](int w) {
      return (unsigned)w < (unsigned)n && ((bwd[w >> 5] >> (w & 31)) & 1u);  // race-free: not written during a round
    };
    auto reaches_now = [&](int w) {  // found in this round
      return (unsigned)w < (unsigned)n && ((ld(&next[w >> 5]) >> (w & 31)) & 1u);
    };
    const int per = min(32, (cnt - 1) / nwarps + 1);
    for (int i0 = warp * per; i0 < cnt; i0 += nwarps * per) {
      const int i = lane < per ? i0 + lane : cnt;
      const int v = i < cnt ? in[i] : 0;  // race-free: written before the last grid barrier
      int beg = 0, deg = 0;
      if (i < cnt && !reaches(v)) row_of(v, beg, deg);
      bool found = false;
      for (int k0 = 0; k0 < min(deg, 32) && !found; k0 += 4) {
        int w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = k0 + k < deg ? __ldg(&nlist[beg + k0 + k]) : -1;
#pragma unroll
        for (int k = 0; k < 4; k++) found |= reaches(w[k]);
        if (!found) {
#pragma unroll
          for (int k = 0; k < 4; k++) found |= reaches_now(w[k]);
        }
      }
      // a row that is still not decided: the rest of it by the whole warp, or,
      // of a long one, as chunk records by all warps (one warp alone with a hub
      // of 1 M entries that does not reach the pivot: 14 ms, in every round)
      push_chunks_warp(RowChunks{chunks, &ctl->back_chunks[round], chunk_cap}, kGiantLong, !found && deg > kBackLong, v,
                       beg, beg + deg, status);
      unsigned todo = __ballot_sync(kFull, !found && deg > 32 && deg <= kBackLong);
      while (todo) {
        const int who = __ffs(todo) - 1;
        todo &= todo - 1;
        const int wbeg = __shfl_sync(kFull, beg, who), wdeg = __shfl_sync(kFull, deg, who);
        bool hit = false;
        for (int k0 = 32; k0 < wdeg && !hit; k0 += 128) {
          bool mine = false;
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const int e = k0 + 32 * k + lane;
            const int w = e < wdeg ? __ldg(&nlist[wbeg + e]) : -1;
            mine = mine || reaches(w) || reaches_now(w);
          }
          hit = __any_sync(kFull, mine);
        }
        if (lane == who) found = hit;
      }
      if (found) {
        fetch_or(&next[v >> 5], 1u << (v & 31));
        moved = true;
      }
      stg.push(deg > 0 && !found, v, out, &ctl->left[round + 1], n, overflow);
    }
    stg.flush(out, &ctl->left[round + 1], n, overflow);
    auto tell = [&]() {  // the block's `moved` to the round's word
      if (moved) s_moved = 1;  // every writer stores the same value
      __syncthreads();
      if (threadIdx.x == 0 && s_moved) st(&ctl->moved[round], 1);
    };
    tell();
    if (!grid_sync(&ctl->giant_bar, status)) return;
    const int nch = chunk_total(RowChunks{chunks, &ctl->back_chunks[round], chunk_cap});
    for (int c = warp; c < nch; c += nwarps) {
      const int2 r = chunks[c];  // race-free: written before the last grid barrier
      if (reaches_now(r.x)) continue;
      const int end = min(r.y + kGiantLong, __ldg(&nindex[r.x + 1]));
      constexpr int K = kGiantLong / 32;
      int w[K];
      bool mine = false;
#pragma unroll
      for (int k = 0; k < K; k++) w[k] = r.y + 32 * k + lane < end ? __ldg(&nlist[r.y + 32 * k + lane]) : -1;
#pragma unroll
      for (int k = 0; k < K; k++) mine = mine || reaches(w[k]) || reaches_now(w[k]);
      if (!__any_sync(kFull, mine)) continue;
      if (lane == 0) fetch_or(&next[r.x >> 5], 1u << (r.x & 31));
      moved = true;
    }
    if (nch > 0) {  // the same for every block
      tell();
      if (!grid_sync(&ctl->giant_bar, status)) return;
    }
    if (!ld(&ctl->moved[round])) break;
    looked += cnt;
    const int left = ld(&ctl->left[round + 1]), found_now = cnt - left;
    if (round == 0) cnt1 = left;
    if (round > 0 && left > n / 2 && found_now < 3) return;
    if (looked > 16LL * n || (looked > 2LL * n && cnt1 - left < n / 16 && 2LL * found_now < 3LL * found0)) return;
    found0 = round == 0 ? 0 : found_now;
    cnt = left;
    merge_bits(bwd, next, words, tid, nthreads);
    if (!grid_sync(&ctl->giant_bar, status)) return;
  }
  // its largest id
  int top = -1;
  for (int i = tid; i < words; i += nthreads) {
    const unsigned x = ld(&fwd[i]) & ld(&bwd[i]);
    if (x) top = max(top, 32 * i + 31 - __clz(x));
  }
  top = __reduce_max_sync(kFull, top);
  if (lane == 0 && top > ld(&ctl->giant_label)) fetch_max(&ctl->giant_label, top);
  if (tid == 0) st(&ctl->giant_ok, 1);
}

// A vertex is live (can be in a non-trivial SCC) iff it has an in-entry and an
// out-entry other than self-loops.  Both facts share one flag word per vertex
// (kHasIn | kHasOut), so the liveness test is one load; scc_mark ORs kHasIn
// into flags[w] for every entry w != v and kHasOut into flags[v] for every v
// with such an entry; rows longer than bins.chunk go to chunk records.
constexpr int kHasIn = 1, kHasOut = 2;

// Marks kScanBatch entries w[k] (present where valid[k]) of v's list, at CSR
// positions j[k]: v has an out-entry and each w an in-entry (self-loops
// ignored), and slot j[k] of the edge list becomes (v, w) -- or a dead slot
// for a self-loop or an id out of range.  The flag words are read first and
// OR'ed only where kHasIn is still clear: R-MAT sends a large share of all
// entries to a few hub ids, whose words would otherwise take an atomic from
// every one of them.
// kRest (after scc_giant): only edges between two vertices outside the giant
// component and on the same side of its forward search count, and they are
// appended to the list (`keep`) instead of standing at their CSR positions.
template <bool kRest, class Keep>
__device__ __forceinline__ void scc_mark_batch(const bool (&valid)[kScanBatch], int v, const int (&w)[kScanBatch],
                                               const int (&j)[kScanBatch], int n, int* flags, int2* wl, const Giant& gi,
                                               Keep&& keep, bool& out, Status* status) {
  int f[kScanBatch];
#pragma unroll
  for (int k = 0; k < kScanBatch; k++)
    f[k] = (valid[k] && (unsigned)w[k] < (unsigned)n && w[k] != v) ? ld(&flags[w[k]]) : kHasIn;
  if constexpr (kRest) {
#pragma unroll
    for (int k = 0; k < kScanBatch; k++) {
      bool edge = valid[k] && (unsigned)w[k] < (unsigned)n && w[k] != v;
      if (valid[k] && (unsigned)w[k] >= (unsigned)n) raise(status, ECL_ERR_BAD_GRAPH, w[k]);
      edge = edge && !gi.in(w[k]) && gi.has(gi.fwd, w[k]) == gi.has(gi.fwd, v);
      if (edge) {
        if (!(f[k] & kHasIn)) fetch_or(&flags[w[k]], kHasIn);
        out = true;
      }
      keep(edge, make_int2(v, w[k]));
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanBatch; k++) {
      if (!valid[k]) continue;
      const bool edge = (unsigned)w[k] < (unsigned)n && w[k] != v;
      if ((unsigned)w[k] >= (unsigned)n) raise(status, ECL_ERR_BAD_GRAPH, w[k]);
      if (edge) {
        if (!(f[k] & kHasIn)) fetch_or(&flags[w[k]], kHasIn);
        out = true;
      }
      __stcs(&wl[j[k]], edge ? make_int2(v, w[k]) : make_int2(-1, -1));
    }
  }
}

template <bool kRest>
__device__ __forceinline__ void scc_mark_rows(int n, int m, const int* nindex, const int* nlist, int* flags, int2* wl,
                                              const RowChunks& rc, const Bins& bins, bool vec, const Giant& gi,
                                              SCCCtl* ctl, Status* status) {
  __shared__ int2 s_stage[kTPB / 32][kRest ? 128 : 1];
  WarpStage<int2, 128, true> stg{s_stage[threadIdx.x >> 5]};
  bool overflow = false;
  auto keep = [&](bool edge, int2 e) {
    if (__any_sync(kFull, edge)) stg.push(edge, e, wl, &ctl->rest, m, overflow);
  };
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  for (int base = warp * 32; base < n; base += nwarps * 32) {
    const int v = base + lane;
    int beg = 0, end = 0;
    if (v < n && !(kRest && gi.in(v))) csr_row(nindex, v, m, beg, end, status);
    const int deg = end - beg;
    push_chunks_warp(rc, bins.chunk, deg > bins.chunk, v, beg, end, status);
    bool out = false;
    const bool lanelvl = deg <= bins.lane;
    const int kmax = __reduce_max_sync(kFull, lanelvl ? deg : 0);
    for (int k0 = 0; k0 < kmax; k0 += kScanBatch) {
      int w[kScanBatch], j[kScanBatch];
      bool valid[kScanBatch];
#pragma unroll
      for (int k = 0; k < kScanBatch; k++) {
        valid[k] = lanelvl && k0 + k < deg;
        j[k] = beg + k0 + k;
        w[k] = valid[k] ? __ldg(&nlist[j[k]]) : 0;
      }
      scc_mark_batch<kRest>(valid, v, w, j, n, flags, wl, gi, keep, out, status);
    }
    unsigned todo = __ballot_sync(kFull, deg > bins.lane && deg <= bins.chunk);
    while (todo) {
      const int who = __ffs(todo) - 1;
      todo &= todo - 1;
      const int wv = __shfl_sync(kFull, v, who);
      const int wbeg = __shfl_sync(kFull, beg, who);
      const int wend = __shfl_sync(kFull, end, who);
      bool wout = false;
      warp_row(wbeg, wend, m, vec, nlist, [&](const int (&j)[4], const int (&w)[4], const bool (&valid)[4]) {
        scc_mark_batch<kRest>(valid, wv, w, j, n, flags, wl, gi, keep, wout, status);
      });
      if (__any_sync(kFull, wout) && lane == who) out = true;
    }
    if (v < n && deg <= bins.chunk && out) fetch_or(&flags[v], kHasOut);  // long rows: scc_mark_chunks
  }
  if (kRest) stg.flush(wl, &ctl->rest, m, overflow);
}

template <bool kRest>
__device__ __forceinline__ void scc_mark_records(int n, int m, const int* nindex, const int* nlist, int* flags, int2* wl,
                                                 const RowChunks& rc, int chunk, bool vec, const Giant& gi, SCCCtl* ctl,
                                                 Status* status) {
  __shared__ int2 s_stage[kTPB / 32][kRest ? 128 : 1];
  WarpStage<int2, 128, true> stg{s_stage[threadIdx.x >> 5]};
  bool overflow = false;
  auto keep = [&](bool edge, int2 e) {
    if (__any_sync(kFull, edge)) stg.push(edge, e, wl, &ctl->rest, m, overflow);
  };
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  const int total = chunk_total(rc);
  for (int c = warp; c < total; c += nwarps) {
    const int2 r = rc.rec[c];
    const int end = min(r.y + chunk, __ldg(&nindex[r.x + 1]));
    bool out = false;
    warp_row(r.y, end, m, vec, nlist, [&](const int (&j)[4], const int (&w)[4], const bool (&valid)[4]) {
      scc_mark_batch<kRest>(valid, r.x, w, j, n, flags, wl, gi, keep, out, status);
    });
    if (__any_sync(kFull, out) && lane == 0) fetch_or(&flags[r.x], kHasOut);
  }
  if (kRest) stg.flush(wl, &ctl->rest, m, overflow);
}

// kSearched: scc_giant ran before, and whether it found the component decides
// between the two forms.  Nothing to do for a symmetric graph (its labels are
// written).  Both words are plain loads of what nothing writes in these
// launches, so L1 serves them (as relaxed loads every warp of the grid queues at
// one L2 word: 6.4 us for 2824 blocks with nothing to do).
template <bool kSearched>
__global__ void __launch_bounds__(kTPB) scc_mark(int n, int m, const int* __restrict__ nindex,
                                                 const int* __restrict__ nlist, int* __restrict__ flags,
                                                 int2* __restrict__ wl, RowChunks rc, Bins bins, bool vec,
                                                 Giant gi, SCCCtl* ctl, bool checked, Status* __restrict__ status) {
  dep_wait();
  if (checked && ctl->asym == 0) return;
  if (kSearched && ctl->giant_ok != 0)
    scc_mark_rows<true>(n, m, nindex, nlist, flags, wl, rc, bins, vec, gi, ctl, status);
  else
    scc_mark_rows<false>(n, m, nindex, nlist, flags, wl, rc, bins, vec, gi, ctl, status);
}

template <bool kSearched>
__global__ void __launch_bounds__(kTPB) scc_mark_chunks(int n, int m, const int* __restrict__ nindex,
                                                        const int* __restrict__ nlist, int* __restrict__ flags,
                                                        int2* __restrict__ wl, RowChunks rc, int chunk, bool vec,
                                                        Giant gi, SCCCtl* ctl, bool checked,
                                                        Status* __restrict__ status) {
  dep_wait();
  if (checked && ctl->asym == 0) return;
  if (kSearched && ctl->giant_ok != 0)
    scc_mark_records<true>(n, m, nindex, nlist, flags, wl, rc, chunk, vec, gi, ctl, status);
  else
    scc_mark_records<false>(n, m, nindex, nlist, flags, wl, rc, chunk, vec, gi, ctl, status);
}

// Word of a trimmed vertex: it is its own SCC, and sweeps skip its edges.
constexpr unsigned long long kDead = ~0ull;
// Edges per lane whose loads are issued together in a sweep: a template
// argument (1, 2 or 4), with the blocks per SM the register budget allows.
constexpr int kSweepBatchDefault = 1;  // the measured best at R-MAT-22 (2.16 ms vs 2.24 / 2.40)
template <int kSweepBatch>
struct SweepOcc {
  static constexpr int blocks = kSweepBatch == 1 ? 8 : (kSweepBatch == 2 ? 6 : 4);
};

// Round 0 sweeps the CSR-position edge list of `m0` slots (dead slots have
// x < 0) or, after scc_giant, the list of the edges outside its component;
// later rounds sweep the compacted survivors.
template <int kSweepBatch>
__global__ void __launch_bounds__(kTPB, SweepOcc<kSweepBatch>::blocks) scc_solve(int n, int m0, int2* __restrict__ wlA, int2* __restrict__ wlB,
                                                  const int* __restrict__ flags, unsigned long long* __restrict__ io,
                                                  int* __restrict__ label, Giant gi, SCCCtl* ctl,
                                                  int max_rounds, bool checked,
                                                  Status* __restrict__ status) {
  if (checked && ld(&ctl->asym) == 0) return;  // as scc_mark
  const int lane = threadIdx.x & 31;
  const int tid = blockIdx.x * kTPB + threadIdx.x;
  const int nthreads = gridDim.x * kTPB;
  int nstamp = 0;  // thread 0: stamps written
  if (tid == 0) ctl->stamp[0] = scc_now();
  // 0. live vertices start at (v, v); trimmed ones are DEAD
  for (int v = tid; v < n; v += nthreads)
    io[v] = __ldg(&flags[v]) == (kHasIn | kHasOut) ? io_pack(v, v) : kDead;  // race-free: owned, barrier next
  if (!grid_sync(&ctl->bar, status)) return;
  if (tid == 0 && ++nstamp < kStamps) ctl->stamp[nstamp] = scc_now();
  const bool giant = ld(&ctl->giant_ok) != 0;
  if (giant) m0 = min(ld(&ctl->rest), m0);
  int size = m0;
  int sweep = 0;
  int round = 0;
  int2* cur = wlA;
  int2* nxt = wlB;
  for (;; round++) {
    if (round >= max_rounds) {
      raise(status, ECL_ERR_NO_CONVERGENCE, round);
      return;
    }
    // 1. propagate in-max forward and out-max backward to a fixpoint
    while (true) {
      if (sweep >= kMaxSweeps) {
        raise(status, ECL_ERR_NO_CONVERGENCE, -sweep);
        return;
      }
      int raises = 0;
      // Append the edges this round keeps during the sweep (below) once the
      // last sweep raised few words: the values are then close to final, and
      // few edges look kept.  Earlier, transient agreement makes millions of
      // edges look kept, and their appends would cost more than the
      // separate pass they save.
      const bool spec = sweep > 0 && ld(&ctl->raised[sweep - 1]) <= (m0 >> 6);
      // The jump targets converge on a few vertices (the largest SCC's
      // maximum id first of all), so every thread keeps its last jump of
      // each kind: a repeated target reuses the value instead of loading the
      // same word as every other edge.  A value read earlier is a smaller
      // but still valid bound (in-max and out-max only grow).
      int c_iv = -1, c_in = -1, c_ow = -1, c_out = -1;
      // Whole warps step together over kSweepBatch slices of 32 consecutive
      // slots; in CSR order neighbouring lanes mostly share v, so the out-max
      // raises of v are combined per slice (__match_any_sync + max) into one
      // atomic instead of up to 32 on one address.  Each lane's edge records,
      // then their io words, then the jump words are loaded before any is
      // used.
      for (int i0 = (tid - lane) * kSweepBatch; i0 < size; i0 += nthreads * kSweepBatch) {
        int2 e[kSweepBatch];
#pragma unroll
        for (int k = 0; k < kSweepBatch; k++) {
          const int i = i0 + 32 * k + lane;
          e[k] = i < size ? __ldcs(&cur[i]) : make_int2(-1, -1);
          if ((unsigned)e[k].x >= (unsigned)n || (unsigned)e[k].y >= (unsigned)n) e[k] = make_int2(-1, -1);
        }
        unsigned long long A[kSweepBatch], B[kSweepBatch];
#pragma unroll
        for (int k = 0; k < kSweepBatch; k++) {
          A[k] = e[k].x >= 0 ? ld(&io[e[k].x]) : kDead;
          B[k] = e[k].x >= 0 ? ld(&io[e[k].y]) : kDead;
        }
        // jumps not covered by the memo load only the half they need (in-max
        // is the high word); -1 = not loaded (live values are >= 0)
        int iv[kSweepBatch], ow[kSweepBatch], ji[kSweepBatch], jo[kSweepBatch];
#pragma unroll
        for (int k = 0; k < kSweepBatch; k++) {
          const bool live = A[k] != kDead && B[k] != kDead;
          iv[k] = live ? io_in(A[k]) : -1;
          ow[k] = live ? io_out(B[k]) : -1;
          ji[k] = (live && iv[k] != e[k].x && iv[k] != c_iv) ? ld(reinterpret_cast<const int*>(&io[iv[k]]) + 1) : -1;
          jo[k] = (live && ow[k] != e[k].y && ow[k] != c_ow) ? ld(reinterpret_cast<const int*>(&io[ow[k]])) : -1;
        }
#pragma unroll
        for (int k = 0; k < kSweepBatch; k++) {
          if (iv[k] >= 0 && iv[k] != e[k].x) {
            if (ji[k] >= 0) {
              c_iv = iv[k];
              c_in = ji[k];
            }
            if (iv[k] == c_iv) iv[k] = max(iv[k], c_in);
          }
          if (ow[k] >= 0 && ow[k] != e[k].y) {
            if (jo[k] >= 0) {
              c_ow = ow[k];
              c_out = jo[k];
            }
            if (ow[k] == c_ow) ow[k] = max(ow[k], c_out);
          }
          if (iv[k] >= 0 && io_raise<true>(&io[e[k].y], B[k], iv[k])) raises++;
          const int v = iv[k] >= 0 ? e[k].x : -1;
          const unsigned grp = __match_any_sync(kFull, v);
          const int gow = __reduce_max_sync(grp, ow[k]);
          if (v >= 0 && lane == __ffs(grp) - 1 && io_raise<false>(&io[v], A[k], gow)) raises++;
        }
        // The edges the round keeps (endpoints unresolved and in full
        // agreement), judged by the words this sweep loaded: only the last
        // sweep's list is used, and that sweep raised nothing, so its words
        // were final.  This saves a separate pass over the list and its words.
        if (spec) {
#pragma unroll
          for (int k = 0; k < kSweepBatch; k++) {
            const bool keep = A[k] != kDead && io_in(A[k]) != io_out(A[k]) && A[k] == B[k];
            const int at = warp_append(&ctl->kept[sweep], keep);
            if (keep && at < m0) nxt[at] = e[k];  // race-free: the place is this reservation's, read behind a grid barrier
          }
        }
      }
      // one count per block (a flag per warp would queue at one word)
      __shared__ int s_raises;
      if (threadIdx.x == 0) s_raises = 0;
      __syncthreads();
      const int wr = __reduce_add_sync(kFull, raises);
      if (lane == 0 && wr) atomicAdd(&s_raises, wr);  // shared memory
      __syncthreads();
      if (threadIdx.x == 0 && s_raises) {
        fetch_add(&ctl->raised[sweep], s_raises);
        st(&ctl->changed[sweep], 1);
      }
      if (!grid_sync(&ctl->bar, status)) return;
      if (tid == 0 && ++nstamp < kStamps) ctl->stamp[nstamp] = scc_now();
      const bool again = ld(&ctl->changed[sweep]) != 0;
      sweep++;
      if (!again) {
        if (spec) break;
        // 1b. the last sweep kept no list: keep the edges whose endpoints are
        // unresolved and agree, in a pass of its own
        for (int i0 = tid - lane; i0 < size; i0 += nthreads) {
          const int i = i0 + lane;
          bool keep = false;
          int2 e = make_int2(0, 0);
          if (i < size) {
            e = cur[i];  // race-free: not written in this round
            if ((unsigned)e.x < (unsigned)n && (unsigned)e.y < (unsigned)n) {
              const unsigned long long A = ld(&io[e.x]);
              keep = A != kDead && io_in(A) != io_out(A) && A == ld(&io[e.y]);
            }
          }
          const int at = warp_append(&ctl->kept[sweep - 1], keep);
          if (keep && at < m0) nxt[at] = e;  // race-free: the place is this reservation's, read behind a grid barrier
        }
        if (!grid_sync(&ctl->bar, status)) return;
        break;
      }
    }
    // 2. retire resolved (and trimmed) vertices, reset the rest to their own id
    bool again = false;
    for (int v = tid; v < n; v += nthreads) {
      const unsigned long long A = ld(&io[v]);
      if (A == kDead) {
        label[v] = giant && gi.in(v) ? ld(&ctl->giant_label) : v;  // race-free: the output, thread-owned and never read here
      } else if (io_in(A) == io_out(A)) {
        label[v] = io_in(A);  // race-free: as above
      } else {
        st(&io[v], io_pack(v, v));
        again = true;
      }
    }
    if (__any_sync(kFull, again) && lane == 0) st(&ctl->again[sweep - 1], 1);
    if (!grid_sync(&ctl->bar, status)) return;
    if (tid == 0 && ++nstamp < kStamps) ctl->stamp[nstamp] = scc_now();
    if (!ld(&ctl->again[sweep - 1])) break;
    size = min(ld(&ctl->kept[sweep - 1]), m0);
    int2* t = cur;
    cur = nxt;
    nxt = t;
  }
  if (tid == 0) st(&status->rounds, sweep);
}

struct SCCBufs {
  SCCCtl* ctl;
  int* flags;
  int* nchunks;
  int2* chunks;
  unsigned long long* io;
  int2* wlA;
  int2* wlB;
  int* tilerow;
  unsigned* bits;  // Giant's two bit arrays
  unsigned* next;
  int* queue;
  int* candA;
  int* candB;
  char* cc_ws;
  int max_rounds;
};

// Sizes at which a graph flagged symmetric is tried as connected components (not
// with hardly any entries, where the general path trims nearly all vertices at
// once and CC's passes over them cost more: 4 M vertices with 6 entries 90 us
// against 136, 1 M with pairs among an eighth of them 71 against 77, among a
// quarter 79 against 80, among half 93 against 82), and at which the search for
// the giant component may run (with fewer entries than vertices there is none).
constexpr bool scc_checked(int n, int m) { return m >= n / 4; }
constexpr bool scc_searched(int n, int m) { return m >= kGiantEntries && m >= n; }

void scc_layout(Carve& c, int n, int m, SCCBufs* b) {
  b->ctl = c.take<SCCCtl>(1);
  b->max_rounds = n + 1;
  b->flags = c.take<int>((size_t)n);
  b->nchunks = c.take<int>(64);
  b->chunks = c.take<int2>(row_chunk_capacity(m, kMinChunk));
  b->io = c.take<unsigned long long>((size_t)n);
  // The check's and the search's arrays lie where the edge lists come later: the
  // union-find's scratch, and after it the search's candidates, in the first
  // one, the check's rows, and after them the search's queue, in the second
  // (the search is tried with n entries or more, so the lists are long enough),
  // and its `next` in io.  Only the two bit arrays that the later launches read
  // are its own.
  const size_t list = sizeof(int2) * (size_t)(m > 0 ? m : 1);
  b->cc_ws = c.take<char>(scc_checked(n, m) ? std::max(list, cc_workspace_bytes(n, m)) : list);
  b->wlA = reinterpret_cast<int2*>(b->cc_ws);
  b->wlB = c.take<int2>((size_t)(m > 0 ? m : 1));
  b->tilerow = reinterpret_cast<int*>(b->wlB);
  b->queue = reinterpret_cast<int*>(b->wlB);
  b->candA = reinterpret_cast<int*>(b->wlA);
  b->candB = b->candA + n;
  b->bits = c.take<unsigned>(scc_searched(n, m) ? 2 * (((size_t)n + 31) / 32) : 0);
  b->next = reinterpret_cast<unsigned*>(b->io);
}

}  // namespace

size_t scc_workspace_bytes(int n, int m) {
  Carve c;
  SCCBufs b;
  scc_layout(c, n, m, &b);
  return c.bytes();
}

}  // namespace ecl

namespace ecl {

ecl_status scc_enqueue(const GraphDev& g, int* label, char* ws, Status* status, const DeviceInfo& dev,
                       cudaStream_t stream, int max_rounds, Marker mark, const UnionInfo* uni) {
  Carve c{ws};
  SCCBufs b;
  scc_layout(c, g.n, g.m, &b);
  const int batch = dev.scc_sweep_batch > 0 ? dev.scc_sweep_batch : kSweepBatchDefault;
  void (*solve)(int, int, int2*, int2*, const int*, unsigned long long*, int*, Giant, SCCCtl*, int, bool,
                Status*) =
      batch == 1 ? scc_solve<1> : (batch == 4 ? scc_solve<4> : scc_solve<2>);
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, solve, kTPB, 0) != cudaSuccess || occ < 1)
    return ECL_ERR_CUDA;
  const int coop_grid = dev.sms * occ;
  const int grid = dev.grid_blocks(kTPB, g.n, g.m);
  // a graph flagged symmetric may be solved as connected components (not when
  // the caller limits the rounds: that limit is the general path's)
  const bool check = (g.flags & ECL_GRAPH_SYMMETRIC) != 0 && max_rounds <= 0 && scc_checked(g.n, g.m);
  // (the same limit; a flagged graph that is what its flag says leaves the search at once)
  const bool giant = max_rounds <= 0 && scc_searched(g.n, g.m);
  if (max_rounds <= 0 || max_rounds > b.max_rounds) max_rounds = b.max_rounds;

  fill_ranges({{b.ctl, sizeof(SCCCtl), 0},
               {b.flags, sizeof(int) * (size_t)g.n, 0},
               {b.nchunks, sizeof(int), 0},
               {b.tilerow, check ? sizeof(int) * ((size_t)flat_tiles(g.m) + 1) : 0, 0xff}},
              dev, stream);
  const RowChunks rc{b.chunks, b.nchunks, (int)row_chunk_capacity(g.m, kMinChunk)};
  // chunk records of 128 entries by default: the mark pass measured faster
  // with them than with 256 (R-MAT-22: 0.65 vs 0.72 ms)
  const Bins bins = bins_of(dev, Bins{kBinLane, kMinChunk});
  const bool vec = (reinterpret_cast<uintptr_t>(g.nlist) & 15) == 0 && dev.row_vec;  // 16-byte row loads
  if (check) {
    ECL_LAUNCH_NEXT(scc_rows, dev.grid_blocks(kTPB, g.n, 0), kTPB, 0, stream, g.n, g.m, g.nindex, b.tilerow, status);
    if (g.m > 0)
      ECL_LAUNCH_NEXT(scc_symmetry, dev.grid_blocks(kTPB, 0, g.m), kTPB, 0, stream,
                 FlatCsr{g.n, g.m, g.nindex, g.nlist, b.tilerow}, (reinterpret_cast<uintptr_t>(g.nlist) & 15) == 0, b.ctl,
                 status);
    const ecl_status st = cc_enqueue(g, label, b.cc_ws, status, dev, stream, {}, uni, &b.ctl->asym);
    if (st != ECL_OK) return st;
    // (the general path's flags stay zero when the graph is not symmetric)
    ECL_LAUNCH_NEXT(scc_top, dev.sms * 4, kTPB, 0, stream, g.n, label, b.flags, b.ctl);
    ECL_LAUNCH_NEXT(scc_relabel, dev.grid_blocks(kTPB, g.n, 0), kTPB, 0, stream, g.n, label, b.flags, b.ctl,
                    status);
  }
  const size_t words = ((size_t)g.n + 31) / 32;
  const Giant gi{b.bits, b.bits + words};
  if (giant) {
    int gocc = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&gocc, scc_giant, kGTPB, 0) != cudaSuccess || gocc < 1)
      return ECL_ERR_CUDA;
    const int blocks = std::max(1, std::min(dev.sms * gocc, (int)(std::max((long long)g.n, (long long)g.m / 4) / kGTPB)));
    ECL_CUDA_TRY(launch_cooperative(scc_giant, blocks, kGTPB, stream, g.n, g.m, g.nindex, g.nlist, gi.fwd, gi.bwd,
                                    b.next, b.queue, b.candA, b.candB, b.chunks, (int)row_chunk_capacity(g.m, kMinChunk), b.ctl,
                                    check, status));
  }
  ECL_LAUNCH_NEXT(giant ? scc_mark<true> : scc_mark<false>, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, b.flags,
                  b.wlA, rc, bins, vec, gi, b.ctl, check, status);
  ECL_LAUNCH_NEXT(giant ? scc_mark_chunks<true> : scc_mark_chunks<false>, grid, kTPB, 0, stream, g.n, g.m, g.nindex,
                  g.nlist, b.flags, b.wlA, rc, bins.chunk, vec, gi, b.ctl, check, status);
  mark();
  ECL_CUDA_TRY(launch_cooperative(solve, coop_grid, kTPB, stream, g.n, g.m, b.wlA, b.wlB, b.flags, b.io, label, gi,
                                  b.ctl, max_rounds, check, status));
  mark();
  return ECL_OK;
}

}  // namespace ecl

extern "C" ecl_status ecl_scc(const ecl_graph_view* g, int32_t* label_out, ecl_opts* opts) {
  using namespace ecl;
  ecl_opts local{};
  if (!opts) opts = &local;
  if (!label_out) return ECL_ERR_INVALID_ARG;
  Solve s(g, opts);
  ecl_status st = s.begin(GraphNeeds{}, g ? scc_workspace_bytes(g->nodes, g->edges) : 0);
  if (st != ECL_OK) return s.finish(st);
  int* label = s.output(label_out, (size_t)s.n);
  if (!label) return s.finish(ECL_ERR_OOM);
  GraphDev gd;
  gd.n = s.n;
  gd.m = s.m;
  gd.nindex = s.nindex;
  gd.nlist = s.nlist;
  gd.flags = g->flags;
  s.start_timer();
  st = scc_enqueue(gd, label, s.ws, s.status, s.dev, s.stream, opts->max_rounds, Marker{&s});
  s.stop_timer();
  return s.finish(st);
}

extern "C" ecl_status ecl_compute_scc(int32_t nodes, int32_t edges, const int32_t* nidx, const int32_t* nlist,
                                      int32_t* label) {
  ecl_graph_view g{nodes, edges, nidx, nlist, nullptr, ECL_HOST, 0};
  ecl_opts o{};
  return ecl_scc(&g, label, &o);
}
