// Graph colouring (ECL-GC contract).
//
// Result contract (src/racefree/egr-input/GC/ECL-GC-atomic.cu): priorities
// are (degree, hash, id) (:102); init/runLarge/runSmall (:78-303) only fix a
// colour once it is the smallest colour not taken by a decided higher-priority
// list entry and no undecided one can still take it, i.e. the result is the
// first-fit greedy colouring in descending priority order.  Self-loops are
// never higher priority (:102 compares v with itself) and are ignored.
//
// B200 design: greedy colouring pulled in priority order.
//  * gc_keys writes every vertex's priority key (the inverted (degree, hash)
//    word) and colours the isolated vertices 0; gc_init / gc_init_chunks
//    (degree-binned: lane / warp / 256-entry chunk records) compare each
//    list entry with one 8-byte key load and compact every row's
//    higher-priority entries to the front of the row's slot in nl2[];
//    hc[v] = their number.
//  * radix_order then ranks the vertices that have entries by priority
//    (an LSD sort of their keys), which is a topological order of the
//    colouring dependencies.
//  * gc_pull is ONE cooperative persistent launch.  Ranks are dealt to the
//    warps round-robin -- one long row (> 32 entries; they form a prefix of
//    the order, priority being degree-first) or 32 short rows at a time --
//    and every warp takes its own in increasing order; each vertex waits
//    (bounded polling of exactly its own higher-priority neighbours' colour
//    words) until they are coloured and stores the smallest colour they do
//    not use.  The warp holding the lowest unfinished rank is working on it,
//    and all its dependencies have lower ranks, so the launch always makes
//    progress.  There is no push, no counter and no queue: the total work is
//    one read of every higher-priority entry, and the longest priority chain
//    (about 2700 vertices at R-MAT-22, most of it in the hub core) costs one
//    poll-and-store hop per vertex on it.
//  * A long row is scanned by a whole warp with a 2048-colour bitmap in
//    shared memory.  The first pass never blocks: colours already published
//    go into the bitmap and the undecided entries into a per-warp pending
//    list; lanes then wait on listed entries (one address per lane) and
//    re-check the rest of the list without blocking -- so a hop along the
//    chain costs one poll and a short re-check, not a rescan of the row
//    (short rows: the same with a bit mask per lane).
#include <algorithm>
#include <vector>

#include "csr_bins.cuh"
#include "fill.cuh"
#include "grid_sync.cuh"
#include "radix_sort.cuh"
#include "solvers.cuh"

namespace ecl {
namespace {

using namespace dev;

constexpr int kTPB = 256;

constexpr int kWarpRow = 32;  // rows longer than this are coloured by a whole warp

struct GCCtl {
  int nchunks;
  int nbig;        // rows longer than kWarpRow: a prefix of the priority order
  int nkeys;       // vertices with at least one entry: the ones sorted and pulled
  int maxdeg;      // largest degree: how many digits of it the sort looks at
  int sort_failed;  // the sort gave up: the order is not whole, and nothing is indexed by it
  int bad_rows;  // some row is malformed, so rows may overlap
  int nwide;     // core rows of more than two segments
  int pad2[25];
  GridBarrier sort_bar;
};

// Priority hash of vertex x: the reference hashes the vertex id; in a union
// of graphs (vhash != nullptr) it is the hash of x's LOCAL id, precomputed.
__device__ __forceinline__ unsigned gc_h(const unsigned* vhash, int x) {
  return vhash ? vhash[x] : ecl_hash((unsigned)x);  // race-free: not written in the launches that call this
}

// Entries per lane whose loads are issued together in the init scans.
constexpr int kInitBatch = 4;

// Classes of kInitBatch list entries of v -- 0: ignore (self-loop or
// invalid), 1: higher priority than v, 2: lower.  A vertex's priority is its
// sort key (gc_keys: the inverted (degree, hash) word, so a SMALLER key is a
// higher priority) with ties to the larger id; kv is v's key.  The list
// entries are loaded first, then every neighbour's key (one 8-byte load each
// instead of both row bounds and a rehash), all before any is compared.
__device__ __forceinline__ void gc_class_batch(const int (&u)[kInitBatch], const bool (&valid)[kInitBatch], int v,
                                               unsigned long long kv, int n, const unsigned long long* keys,
                                               Status* status, int (&cls)[kInitBatch]) {
  unsigned long long ku[kInitBatch];
#pragma unroll
  for (int k = 0; k < kInitBatch; k++) {
    const bool ok = valid[k] && (unsigned)u[k] < (unsigned)n && u[k] != v;
    ku[k] = ok ? keys[n - 1 - u[k]] : 0ull;  // race-free: not written in this launch
  }
#pragma unroll
  for (int k = 0; k < kInitBatch; k++) {
    cls[k] = 0;
    if (!valid[k]) continue;
    if ((unsigned)u[k] >= (unsigned)n) {
      raise(status, ECL_ERR_BAD_GRAPH, u[k]);
    } else if (u[k] != v) {
      cls[k] = (ku[k] < kv || (ku[k] == kv && u[k] > v)) ? 1 : 2;
    }
  }
}

// vhash[v] = hash of v's local id in a union of graphs.
__global__ void __launch_bounds__(kTPB) gc_union_hash(int n, const int* __restrict__ vbase, int ngraphs,
                                                      unsigned* __restrict__ vhash) {
  dep_wait();
  for (int v = blockIdx.x * kTPB + threadIdx.x; v < n; v += gridDim.x * kTPB) {
    const int base = __ldg(&vbase[union_graph_of(vbase, ngraphs, v)]);
    vhash[v] = ecl_hash((unsigned)(v - base));  // race-free: thread-owned, no reader in this launch
  }
}

constexpr int kSmallGroup = 4;

// A warp takes `group` (a power of two, at most 32) vertices at a time: 32 on
// graphs that give every warp of the device some, fewer below, because a
// group's rows of more than bins.lane entries run one after another, and the
// first groups of a power-law graph have little else.
__global__ void __launch_bounds__(kTPB) gc_init(int n, int m, const int* __restrict__ nindex,
                                                const int* __restrict__ nlist, int* __restrict__ nl2,
                                                int* __restrict__ hc, RowChunks rc, Bins bins, int group, bool vec,
                                                const unsigned long long* keys,
                                                Status* __restrict__ status) {
  dep_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  for (long long base = (long long)warp * group; base < n; base += (long long)nwarps * group) {
    const int v = lane < group ? (int)min(base + lane, (long long)n) : n;
    int beg = 0, end = 0;
    if (v < n) csr_row(nindex, v, m, beg, end, status);
    const int dv = end - beg;
    const unsigned long long kv = (v < n) ? keys[n - 1 - v] : 0ull;  // race-free: not written in this launch
    int h = 0;
    push_chunks_warp(rc, bins.chunk, dv > bins.chunk, v, beg, end, status);
    if (v < n && dv <= bins.lane) {
      for (int i0 = beg; i0 < end; i0 += kInitBatch) {
        int u[kInitBatch], cls[kInitBatch];
        bool valid[kInitBatch];
#pragma unroll
        for (int k = 0; k < kInitBatch; k++) {
          valid[k] = i0 + k < end;
          u[k] = valid[k] ? __ldg(&nlist[i0 + k]) : 0;
        }
        gc_class_batch(u, valid, v, kv, n, keys, status, cls);
#pragma unroll
        for (int k = 0; k < kInitBatch; k++)
          if (cls[k] == 1) nl2[beg + h++] = u[k];  // race-free: v's own slot, no reader in this launch
      }
    }
    unsigned todo = __ballot_sync(kFull, dv > bins.lane && dv <= bins.chunk);
    while (todo) {
      const int who = __ffs(todo) - 1;
      todo &= todo - 1;
      const int wv = __shfl_sync(kFull, v, who);
      const int wbeg = __shfl_sync(kFull, beg, who);
      const int wend = __shfl_sync(kFull, end, who);
      const unsigned long long wkv = __shfl_sync(kFull, kv, who);
      int wh = 0;
      warp_row(wbeg, wend, m, vec, nlist, [&](const int(&)[4], const int (&u)[4], const bool (&valid)[4]) {
        int cls[kInitBatch];
        gc_class_batch(u, valid, wv, wkv, n, keys, status, cls);
#pragma unroll
        for (int k = 0; k < kInitBatch; k++) {
          const unsigned bh = __ballot_sync(kFull, cls[k] == 1);
          // race-free: wv's own slot, no reader in this launch
          if (cls[k] == 1) nl2[wbeg + wh + __popc(bh & ((1u << lane) - 1))] = u[k];
          wh += __popc(bh);
        }
      });
      if (lane == who) h = wh;
    }
    // race-free: v's own count, read only by later launches; chunked rows start at 0 (gc_init_chunks adds)
    if (v < n) hc[v] = dv > bins.chunk ? 0 : h;
  }
}

__global__ void __launch_bounds__(kTPB) gc_init_chunks(int n, int m, const int* __restrict__ nindex,
                                                       const int* __restrict__ nlist, int* __restrict__ nl2,
                                                       int* __restrict__ hc, RowChunks rc, int chunk, bool vec,
                                                       const unsigned long long* keys,
                                                       Status* __restrict__ status) {
  dep_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  const int total = chunk_total(rc);
  for (int c = warp; c < total; c += nwarps) {
    const int2 r = rc.rec[c];
    const int v = r.x;
    const int beg = __ldg(&nindex[v]), end = __ldg(&nindex[v + 1]);
    const int stop = min(r.y + chunk, end);
    const unsigned long long kv = keys[n - 1 - v];  // race-free: not written in this launch
    warp_row(r.y, stop, m, vec, nlist, [&](const int(&)[4], const int (&u)[4], const bool (&valid)[4]) {
      int cls[kInitBatch];
      gc_class_batch(u, valid, v, kv, n, keys, status, cls);
      unsigned bh[kInitBatch];
      int nh = 0;
#pragma unroll
      for (int k = 0; k < kInitBatch; k++) {
        bh[k] = __ballot_sync(kFull, cls[k] == 1);
        nh += __popc(bh[k]);
      }
      int hbase = 0;
      if (lane == 0 && nh) hbase = fetch_add(&hc[v], nh);
      hbase = __shfl_sync(kFull, hbase, 0);
#pragma unroll
      for (int k = 0; k < kInitBatch; k++) {
        // race-free: the places are this reservation's
        if (cls[k] == 1) nl2[beg + hbase + __popc(bh[k] & ((1u << lane) - 1))] = u[k];
        hbase += __popc(bh[k]);
      }
    });
  }
}

// Priority keys: keys[n - 1 - v] = ~((degree << 32) | hash) for every v, the
// array gc_init compares neighbours by; ascending order of the keys is
// descending (degree, hash), the priority (within one graph the hash is a
// bijection of the id, so no two vertices tie).  The vertices with at least
// one entry are also appended to (skeys, svals), the sort's input, counted in
// ctl->nkeys.  An isolated vertex has no neighbour to wait for or to block:
// its colour is 0, written here, and it is neither sorted nor pulled
// (R-MAT-22 has 1.8 M of them among its 4.2 M vertices).  Bound by the appends'
// counter: with one vertex a thread and reservation the pass took 46 us at
// R-MAT-22 (75 MB), with four 29.
constexpr int kKeyBatch = 4;

__global__ void __launch_bounds__(kTPB) gc_keys(int n, int m, const int* __restrict__ nindex,
                                                unsigned long long* __restrict__ keys,
                                                unsigned long long* __restrict__ skeys, int* __restrict__ svals,
                                                const unsigned* vhash, int* __restrict__ color,
                                                GCCtl* __restrict__ ctl) {
  dep_wait();
  // rows longer than kWarpRow are counted per block and added once per block;
  // the appends reserve their room with one atomic per block and step of
  // kKeyBatch vertices a thread, as all of them meet at one word
  __shared__ int s_big, s_deg;
  __shared__ int s_woff[kKeyBatch * kTPB / 32];
  __shared__ int s_base;
  if (threadIdx.x == 0) s_big = s_deg = 0;
  __syncthreads();
  int nb = 0, dmax = 0;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int kStep = kKeyBatch * kTPB, kGroups = kKeyBatch * kTPB / 32;
  static_assert(kGroups == 32, "one warp adds the groups up");
  for (long long bbase = (long long)blockIdx.x * kStep; bbase < n; bbase += (long long)gridDim.x * kStep) {  // block-uniform
    unsigned long long key[kKeyBatch];
    unsigned deg[kKeyBatch], bal[kKeyBatch];
#pragma unroll
    for (int k = 0; k < kKeyBatch; k++) {
      const long long i = bbase + k * kTPB + threadIdx.x;
      const int v = n - 1 - (int)i;
      deg[k] = 0u;
      if (i < n) {
        const int beg = __ldg(&nindex[v]), end = __ldg(&nindex[v + 1]);
        deg[k] = (unsigned)(end - beg);
        if (beg < 0 || end < beg || end > m) st(&ctl->bad_rows, 1);  // (gc_init reports it)
      }
    }
#pragma unroll
    for (int k = 0; k < kKeyBatch; k++) {
      const long long i = bbase + k * kTPB + threadIdx.x;
      const int v = n - 1 - (int)i;
      key[k] = 0;
      if (i < n) {
        key[k] = ~(((unsigned long long)deg[k] << 32) | gc_h(vhash, v));
        keys[i] = key[k];  // race-free: thread-owned, no reader in this launch
        dmax = max(dmax, (int)min(deg[k], 0x7fffffffu));
        if (deg[k] == 0) color[v] = 0;  // race-free: the output, thread-owned; nothing reads it in this launch
      }
      nb += __popc(__ballot_sync(kFull, deg[k] > (unsigned)kWarpRow));
      bal[k] = __ballot_sync(kFull, deg[k] > 0);
      if (lane == 0) s_woff[k * (kTPB / 32) + wid] = __popc(bal[k]);
    }
    __syncthreads();
    if (wid == 0) {
      const int c = s_woff[lane];
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += x;
      }
      s_woff[lane] = incl - c;
      if (lane == 31) s_base = incl ? fetch_add(&ctl->nkeys, incl) : 0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kKeyBatch; k++) {
      if (deg[k] == 0) continue;
      const int at = s_base + s_woff[k * (kTPB / 32) + wid] + __popc(bal[k] & ((1u << lane) - 1));
      skeys[at] = key[k];  // race-free: the place is this reservation's
      svals[at] = n - 1 - (int)(bbase + k * kTPB + threadIdx.x);  // race-free: as above
    }
    __syncthreads();  // s_woff and s_base are rewritten next step
  }
  dmax = __reduce_max_sync(kFull, dmax);
  if (lane == 0) {
    if (nb) atomicAdd(&s_big, nb);
    atomicMax(&s_deg, dmax);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_big) fetch_add(&ctl->nbig, s_big);
    if (s_deg > ld(&ctl->maxdeg)) fetch_max(&ctl->maxdeg, s_deg);
  }
}

__device__ __forceinline__ unsigned long long gc_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr unsigned long long kStallNs = 2000000000ull;  // 2 s without progress -> give up
constexpr int kMexWords = 64;                           // warp bitmap: 2048 colours per window
constexpr int kPend = 1024;                             // per-warp list of undecided entries
constexpr int kBatch = 16;                              // entries per lane whose loads are in flight together

// Colour of u once it is published (bounded wait).  Returns -1 on a stall.
__device__ __forceinline__ int gc_wait_colour(const int* color, int u, Status* status, unsigned nap_cap = 512u) {
  int c = ld(&color[u]);
  if (c >= 0) return c;
  unsigned nap = 32, spins = 0;
  const unsigned long long t0 = gc_now();
  while ((c = ld(&color[u])) < 0) {
    // the stall checks every 64th poll: status->code is one word, and every
    // polling lane of the grid reading it on every poll makes its L2 slice a
    // hot spot that slows the colour polls themselves
    if ((++spins & 63u) == 0 && (spins > (1u << 24) || gc_now() - t0 > kStallNs || ld(&status->code) != 0)) {
      raise(status, ECL_ERR_NO_CONVERGENCE, u);
      return -1;
    }
    __nanosleep(nap);
    nap = min(nap * 2, nap_cap);
  }
  return c;
}

__device__ __forceinline__ void gc_mark(unsigned* bits, int c, int off) {
  const int d = c - off;
  if (d >= 0 && d < 32 * kMexWords) atomicOr(&bits[d >> 5], 1u << (d & 31));
}

// Colour of a long row: the smallest colour no entry of nl2[wb, we) uses.
// Each window of 2048 colours starts with one non-blocking pass over the row:
// colours already published go into the bitmap, still-undecided entries into
// the per-warp list `pend`.  Then every lane waits (bounded, one address per
// lane as before) for one listed entry, and the rest of the list is
// re-checked without blocking and compacted; repeat until it is empty.  Once
// the last dependency is coloured the row is one poll and one short re-check
// from its colour -- a lane no longer walks the rest of its share of the row
// after each wait.  The pass stops while the list still has room for a whole
// step of 32 entries; the listed ones are resolved and the pass resumes where
// it stopped, so every entry is read once by the pass.  `ahead` holds the
// row's first 32 * kAhead entries (entry 32 k + lane), loaded while the row
// before was being coloured.  Returns -1 on a stall.  All lanes call.
constexpr int kAhead = 4;

__device__ int gc_long_row(int wb, int we, const int (&ahead)[kAhead], const int* nl2, const int* color, unsigned* bits,
                           int* pend, int pend_cap, unsigned nap_cap, Status* status) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1;
  for (int off = 0;; off += 32 * kMexWords) {
    bits[lane] = 0;
    bits[lane + 32] = 0;
    __syncwarp();
    int cursor = wb;
    while (cursor < we) {
      int np = 0;
      int i0 = cursor;
      if (off == 0 && i0 == wb) {
        int c[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; k++) c[k] = wb + 32 * k + lane < we ? ld(&color[ahead[k]]) : 0;
#pragma unroll
        for (int k = 0; k < kAhead; k++) {
          const bool in = wb + 32 * k + lane < we, undecided = in && c[k] < 0;
          if (in && !undecided) gc_mark(bits, c[k], off);
          const unsigned ub = __ballot_sync(kFull, undecided);
          if (undecided) pend[np + __popc(ub & lt)] = ahead[k];
          np += __popc(ub);
        }
        i0 += 32 * kAhead;
      }
      // kBatch entries per lane per step: all index loads, then all colour
      // loads, are issued before any result is used (one round trip per
      // 32 * kBatch entries instead of two per 32)
      for (; i0 < we && np + 32 * kBatch <= pend_cap; i0 += 32 * kBatch) {
        int u[kBatch], c[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
          const int i = i0 + 32 * k + lane;
          u[k] = i < we ? __ldg(&nl2[i]) : -1;
        }
#pragma unroll
        for (int k = 0; k < kBatch; k++) c[k] = u[k] >= 0 ? ld(&color[u[k]]) : 0;
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
          const bool undecided = u[k] >= 0 && c[k] < 0;
          if (u[k] >= 0 && c[k] >= 0) gc_mark(bits, c[k], off);
          const unsigned ub = __ballot_sync(kFull, undecided);
          if (undecided) pend[np + __popc(ub & lt)] = u[k];
          np += __popc(ub);
        }
      }
      cursor = i0;  // the list is full or the row is done: resolve, then resume here
      int cnt = np;
      while (cnt > 0) {
        __syncwarp();
        bool stalled = false;
        if (lane < cnt) {
          const int c = gc_wait_colour(color, pend[lane], status, nap_cap);
          if (c < 0)
            stalled = true;
          else
            gc_mark(bits, c, off);
        }
        if (__any_sync(kFull, stalled)) return -1;
        int kept = 0;
        for (int j0 = 32; j0 < cnt; j0 += 32 * kBatch) {
          int u[kBatch], c[kBatch];
#pragma unroll
          for (int k = 0; k < kBatch; k++) {
            const int j = j0 + 32 * k + lane;
            u[k] = j < cnt ? pend[j] : -1;
          }
#pragma unroll
          for (int k = 0; k < kBatch; k++) c[k] = u[k] >= 0 ? ld(&color[u[k]]) : 0;
          __syncwarp();  // every lane has read its slots before any is overwritten
#pragma unroll
          for (int k = 0; k < kBatch; k++) {
            const bool still = u[k] >= 0 && c[k] < 0;
            if (u[k] >= 0 && c[k] >= 0) gc_mark(bits, c[k], off);
            const unsigned sb = __ballot_sync(kFull, still);
            if (still) pend[kept + __popc(sb & lt)] = u[k];  // index < j0: already read
            kept += __popc(sb);
          }
        }
        cnt = kept;
      }
    }
    __syncwarp();
    const unsigned w0 = bits[lane], w1 = bits[lane + 32];
    const unsigned f0 = __ballot_sync(kFull, w0 != ~0u), f1 = __ballot_sync(kFull, w1 != ~0u);
    int c = -1;
    if (f0) {
      const int wi = __ffs(f0) - 1;
      c = off + wi * 32 + __ffs(~__shfl_sync(kFull, w0, wi)) - 1;
    } else if (f1) {
      const int wi = __ffs(f1) - 1;
      c = off + (wi + 32) * 32 + __ffs(~__shfl_sync(kFull, w1, wi)) - 1;
    }
    __syncwarp();
    if (c >= 0) return c;
  }
}

// Colour of a short row (h <= 32 entries at nl2[beg]): one lane, the same
// scheme with a bit mask of the undecided entries -- wait for the first one,
// re-check the others without blocking.  -1 on a stall.
__device__ int gc_short_row(int beg, int h, const int* nl2, const int* color, Status* status) {
  // colour <= h <= 32: a neighbour's colour of 64 or more (a hub's) cannot
  // be the smallest free one and is left out of the mask
  unsigned long long used = 0;
  unsigned pendm = 0;
  for (int k0 = 0; k0 < h; k0 += kBatch) {
    int u[kBatch], c[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) u[k] = k0 + k < h ? __ldg(&nl2[beg + k0 + k]) : -1;
#pragma unroll
    for (int k = 0; k < kBatch; k++) c[k] = u[k] >= 0 ? ld(&color[u[k]]) : 0;
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      if (u[k] < 0) continue;
      if (c[k] >= 0)
        used |= c[k] < 64 ? 1ull << c[k] : 0ull;
      else
        pendm |= 1u << (k0 + k);
    }
  }
  while (pendm) {
    const int k0 = __ffs(pendm) - 1;
    const int c0 = gc_wait_colour(color, __ldg(&nl2[beg + k0]), status);
    if (c0 < 0) return -1;
    used |= c0 < 64 ? 1ull << c0 : 0ull;
    pendm &= pendm - 1;
    for (unsigned mm = pendm; mm; mm &= mm - 1) {
      const int k = __ffs(mm) - 1;
      const int c = ld(&color[__ldg(&nl2[beg + k])]);
      if (c >= 0) {
        used |= c < 64 ? 1ull << c : 0ull;
        pendm &= ~(1u << k);
      }
    }
  }
  return __ffsll((long long)~used) - 1;
}

// ---- the hub core: the first ranks of the order, coloured in shared memory ----
//
// On R-MAT the longest priority chain (about 2700 vertices at scale 22)
// runs almost entirely through the long rows at the front of the order:
// about 2200 of its hops lie in the first 16k ranks and 2470 in the first 32k.
// A hop through L2 costs a store, a poll and a wake-up (about 1.5 us as the
// pull achieves it); in shared memory it costs a few hundred cycles.  So the
// first `core` ranks (core = min(long rows, cap)) are coloured by a cluster
// of CTAs of 32 warps each (two by default) with the colours in shared
// memory, indexed by rank -- a copy in every CTA, each colour stored into its own
// CTA's directly and into the others' through distributed shared memory (its own
// that way too: 45 ns more a hop): every higher-priority entry of a
// core row is itself a core vertex (it has a smaller rank), so a core row
// never waits on global memory.  Two small launches first rewrite
// the core rows' entries in nl2 from vertex ids to ranks (rank[] is the
// inverse of the order over the core) and record each core rank's row
// (start, length, vertex).
//
// The cluster's SMs stream all core rows (5.4 M entries for the first 8192
// ranks of R-MAT-22, 660 a row), so the instructions and shared-memory cycles
// per entry bound the core as much as the chain does.  Rows hold 16-bit ranks,
// packed and 16-byte aligned by gc_core_translate, and arrive through two
// shared-memory buffers per warp with bulk asynchronous copies (cp.async.bulk,
// completion counted on an mbarrier): while a warp colours one segment of a
// row, the next segment -- of this row or of its next row -- is already on its
// way.  A lane reads eight ranks with one 16-byte load, looks each colour up
// (16-bit words, 0xffff = not yet coloured; a core colour is at most the row's
// length, below 2^15), sets a byte of the warp's mark array for it without any
// test -- undecided and far colours go to a byte that nobody reads -- and keeps
// the undecided entries in a 32-bit mask.  A byte store needs no atomic: lanes
// that mark the same colour store the same value.
//
// On the chain lies what a warp does between its last neighbour's colour and its
// own, among 31 other warps' polls.  So all of a row is scanned before any wait,
// the search for the smallest
// colour starts where it ended before the wait, and the marks are cleared and the
// next row fetched behind the publication.  Measured, core, a lane polling its
// lowest entry after each segment, 1016 colours a window and the search from 0 ->
// this: R-MAT-22 1.35 -> 1.21 ms, R-MAT-16 0.53 -> 0.49, a clique of 1000 vertices
// 0.91 -> 0.59, of 2000 12.5 -> 1.3, a complete bipartite graph of 2 x 2000 2.6 -> 1.45.
constexpr int kCoreThreads = 1024;
constexpr int kCoreWarps = kCoreThreads / 32;
// Default CTAs of the core's cluster.  A hop between CTAs, through distributed
// shared memory, costs more than one inside a CTA.  R-MAT-22, core time by
// CTAs (8192 ranks): 1: 1.50 ms, 2: 1.21, 4: 1.20; core + pull by ranks (2
// CTAs): 4096: 2.55 ms, 8192: 2.22, 16384: 2.38, 32768: 3.05.
constexpr int kCoreCtas = 2;
constexpr int kCoreDefault = 8192;      // default core size (ranks): the measured best at R-MAT-22 with 2 CTAs
constexpr int kCoreMax = 36864;         // shared memory bound
constexpr int kSegMax = 1024;           // entries per segment: a bit each of a lane's 32-bit mask
constexpr unsigned kUncoloured = 0xffffu;
constexpr int kWin = 2032;              // colours of a mark window; a byte behind it takes what is outside
constexpr int kMarkBytes = 2048;
constexpr int kCorePend = 256;          // undecided entries that a warp's list holds (rows of more than two segments)
constexpr int kFromRow = 512;           // rows from which on the search starts ahead (a shorter row's marks are one load)
constexpr size_t kCoreSmemLimit = 227 * 1024;

// Dynamic shared memory of a core CTA: colours (16-bit, per rank), then per
// warp two mbarriers, two staging buffers of `seg` entries, the mark bytes and
// the list of undecided entries.
// The buffers take what the colours leave, up to kSegMax entries.
__host__ __device__ constexpr size_t gc_core_colour_bytes(int cap) { return ((size_t)cap * 2 + 15) & ~size_t(15); }
__host__ __device__ constexpr size_t gc_core_warp_bytes(int seg) {
  return 2 * sizeof(unsigned long long) + ((size_t)seg * 2 + kCorePend) * sizeof(unsigned short) + kMarkBytes;
}
__host__ __device__ constexpr int gc_core_seg(int cap) {
  const size_t fixed = gc_core_colour_bytes(cap) + kCoreWarps * gc_core_warp_bytes(0);
  const size_t per = (kCoreSmemLimit - fixed) / kCoreWarps / (2 * sizeof(unsigned short));
  return (int)((per < (size_t)kSegMax ? per : (size_t)kSegMax) & ~size_t(7));
}
__host__ __device__ constexpr size_t gc_core_smem(int cap) {
  return gc_core_colour_bytes(cap) + kCoreWarps * gc_core_warp_bytes(gc_core_seg(cap));
}
static_assert(gc_core_seg(kCoreMax) >= 256 && gc_core_smem(kCoreMax) <= kCoreSmemLimit,
              "core shared memory over the per-block limit");

// Core size of this solve: the long rows (a prefix of the order), at most cap.
// None when the sort failed, and none when rows may overlap: the core's rows
// are packed in place, and another row in the same slot would take two of
// their 16-bit ranks for a vertex.
__device__ __forceinline__ int gc_core_size(const GCCtl* ctl, int cap) {
  return ld(&ctl->sort_failed) || ld(&ctl->bad_rows) ? 0 : min(ld(&ctl->nbig), cap);
}

// rank[order[r]] = r over the core.
__global__ void __launch_bounds__(kTPB) gc_core_rank(const int* order, int* __restrict__ rank,
                                                     const GCCtl* ctl, int cap) {
  dep_wait();
  const int core = gc_core_size(ctl, cap);
  // race-free: order is whole and has each vertex once
  for (int r = blockIdx.x * kTPB + threadIdx.x; r < core; r += gridDim.x * kTPB) rank[order[r]] = r;
}

// Rewrites the higher-priority entries of every core row from vertex ids to
// 16-bit ranks, one warp per row, packed from the first 16-byte boundary of the
// row's slot on, and records the row: rowinfo[r] = (start in 16-byte units,
// length, vertex).  Such an entry outranks its row, so its rank is below the
// row's and inside the core.  In place: a step's 32 entries are read before
// any rank of them is written, and the ranks written up to step i end below
// the first entry of step i + 1.  A core row has more than kWarpRow entries,
// so its 4-byte slot holds the packed ranks and the copies' rounding.
__global__ void __launch_bounds__(kTPB) gc_core_translate(const int* __restrict__ nindex, int* nl2,
                                                          const int* hc, const int* order,
                                                          const int* rank, int4* __restrict__ rowinfo,
                                                          GCCtl* ctl, int cap,
                                                          Status* __restrict__ status) {
  dep_wait();
  const int lane = threadIdx.x & 31;
  const int core = gc_core_size(ctl, cap);
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  for (int r = warp; r < core; r += nwarps) {
    const int v = order[r];  // race-free: not written in this launch
    const int b = __ldg(&nindex[v]), h = hc[v];  // race-free: not written in this launch
    const int first = (int)(((long long)b + 3) >> 2);  // 16-byte units
    unsigned short* out = reinterpret_cast<unsigned short*>(nl2) + (size_t)first * 8;
    for (int i0 = 0; i0 < h; i0 += 32) {
      const int i = i0 + lane;
      unsigned short q = 0;
      if (i < h) {
        const int x = rank[nl2[(size_t)b + i]];  // race-free: rank is not written, nl2 by this warp in its own row
        if ((unsigned)x < (unsigned)r)
          q = (unsigned short)x;
        else  // only where a union's entry leaves its graph for a vertex of the same key
          raise(status, ECL_ERR_BAD_GRAPH, v);
      }
      __syncwarp();
      if (i < h) out[i] = q;
      __syncwarp();
    }
    if (lane == 0) rowinfo[r] = make_int4(first, h, v, 0);  // race-free: the warp's own, no reader in this launch
    if (lane == 0 && h > 2 * gc_core_seg(cap)) fetch_add(&ctl->nwide, 1);
  }
}

// ---- shared-memory and bulk-copy primitives (CTA-local, inline PTX) ----

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// 16-bit colour words: relaxed CTA-scope atomic loads and stores.
// The core's colours live in every CTA of its cluster (one copy per CTA's
// shared memory): a colour is stored into each copy (distributed shared
// memory) and read from the local one, so both sides are cluster-scope
// relaxed accesses.
__device__ __forceinline__ unsigned col_ld(const unsigned short* p) {
  unsigned short v;
  asm volatile("ld.relaxed.cluster.shared::cta.u16 %0, [%1];" : "=h"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void col_st(unsigned short* p, unsigned v) {
  asm volatile("st.relaxed.cluster.shared::cta.u16 [%0], %1;" ::"r"(smem_u32(p)), "h"((unsigned short)v) : "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_ctas() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Every thread of every CTA of the cluster; memory before it is visible to
// the whole cluster after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Stores colour v of the rank at p (a local shared address) into this CTA's copy
// and into that of every other CTA of the cluster.
__device__ __forceinline__ void col_publish(unsigned short* p, unsigned v, int ctas) {
  col_st(p, v);
  const unsigned local = smem_u32(p), me = cluster_rank();
  for (int k = 0; k < ctas; k++) {
    if (k == (int)me) continue;
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(k));
    asm volatile("st.relaxed.cluster.shared::cluster.u16 [%0], %1;" ::"r"(remote), "h"((unsigned short)v) : "memory");
  }
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// Starts a bulk copy of `bytes` (a multiple of 16, both ends 16-byte aligned)
// from global src into shared dst, completing on bar.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier generic reads of dst come first
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase `parity` of bar (2 s); false when it ran out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = gc_now();
  for (unsigned spins = 1;; spins++) {
    if (mbar_test(bar, parity)) return true;
    if ((spins & 255u) == 0 && gc_now() - t0 > kStallNs) return false;
  }
}

// The smallest colour of the window at `off` that the warp's marks leave free,
// or -1, with all below `start` known to be taken; `end` is the last byte that
// may be set.  128 bytes a ballot, the loads of four of them in flight.  All
// lanes call, behind a __syncwarp.
__device__ __forceinline__ int gc_core_mex(const unsigned char* marks, int off, int start, int end) {
  const int lane = threadIdx.x & 31;
  for (int i0 = start & ~127; i0 <= end; i0 += 512) {
    unsigned w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = i0 + 128 * k + 4 * lane;
      w[k] = i < kWin ? *reinterpret_cast<const unsigned*>(marks + i) : ~0u;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const unsigned z = (w[k] - 0x01010101u) & ~w[k] & 0x80808080u;  // lowest set bit: the lowest zero byte
      const unsigned f = __ballot_sync(kFull, z != 0);
      if (f) {
        const int who = __ffs(f) - 1;
        return off + i0 + 128 * k + 4 * who + ((__ffs(__shfl_sync(kFull, z, who)) - 1) >> 3);
      }
    }
  }
  return -1;
}
static_assert(kWin % 4 == 0 && kWin < kMarkBytes && kMarkBytes % 512 == 0, "gc_core_mex and gc_core_clear");

// Clears the marks up to byte `end`.  All lanes call.
__device__ __forceinline__ void gc_core_clear(unsigned char* marks, int end) {
  for (int i0 = 0; i0 <= end; i0 += 512)
    reinterpret_cast<uint4*>(marks + i0)[threadIdx.x & 31] = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
}

// Colour of a core row of `h` ranks at `row` (16-byte aligned) whose first kWin
// colours are all taken by its neighbours; every neighbour is coloured by now.
// The row is read again for each window, 1024 entries in flight: this lies on
// the chain of a clique's colours (32 entries at a time, and windows of 1016: a
// clique of 5000 vertices 166 ms; so: 47).
__device__ int gc_core_far(const unsigned short* row, int h, const unsigned short* col_s, unsigned char* marks) {
  const int lane = threadIdx.x & 31;
  const uint4* rv = reinterpret_cast<const uint4*>(row);
  constexpr int kFlight = 4;
  for (int off = kWin;; off += kWin) {
    gc_core_clear(marks, kWin - 1);
    for (int i0 = 8 * lane; i0 < h; i0 += 256 * kFlight) {
      uint4 x[kFlight];
#pragma unroll
      for (int s = 0; s < kFlight; s++) {
        const int e = i0 + 256 * s;
        x[s] = e < h ? rv[e >> 3] : make_uint4(0u, 0u, 0u, 0u);  // up to 7 entries of the slot past the row
      }
#pragma unroll
      for (int s = 0; s < kFlight; s++) {
        const int e = i0 + 256 * s;
        const unsigned w[4] = {x[s].x, x[s].y, x[s].z, x[s].w};
#pragma unroll
        for (int k = 0; k < 8; k++) {
          if (e + k >= h) continue;
          const int d = (int)col_ld(&col_s[(k & 1) ? w[k >> 1] >> 16 : w[k >> 1] & 0xffffu]) - off;
          if (d >= 0 && d < kWin) marks[d] = 1;
        }
      }
    }
    __syncwarp();
    const int c = gc_core_mex(marks, off, 0, kWin - 1);
    __syncwarp();  // read before they are cleared
    if (c >= 0) return c;
  }
}

// The undecided entries of two segments (masks open0, open1 of those at sg0, sg1)
// behind the `np` ranks of the warp's list: its new length, or -1 when they do not
// fit.
__device__ __forceinline__ int gc_core_keep(unsigned open0, unsigned open1, const unsigned short* sg0,
                                         const unsigned short* sg1, unsigned short* pend, int np) {
  const int lane = threadIdx.x & 31;
  const int mine = __popc(open0) + __popc(open1);
  int at = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(kFull, at, o);
    if (lane >= o) at += x;
  }
  const int total = __shfl_sync(kFull, at, 31);
  if (np + total > kCorePend) return -1;
  at += np - mine;
  for (int part = 0; part < 2; part++) {
    const unsigned short* sg = part ? sg1 : sg0;
    for (unsigned open = part ? open1 : open0; open; open &= open - 1) {
      const int k = __ffs(open) - 1;
      pend[at++] = sg[256 * (k >> 3) + 8 * lane + (k & 7)];
    }
  }
  __syncwarp();
  return np + total;
}

// Waits for the ranks in the warp's list and marks their colours; true on a stall.
__device__ __forceinline__ bool gc_core_settle(const unsigned short* pend, int np, const unsigned short* col_s,
                                            unsigned char* marks, unsigned beyond, int r, Status* status) {
  bool lost = false;
  unsigned spins = 0;
  unsigned long long t0 = 0;
  for (int j = threadIdx.x & 31; j < np && !lost; j += 32) {
    const unsigned short* p = &col_s[pend[j]];
    unsigned c;
    while ((c = col_ld(p)) == kUncoloured) {
      if ((++spins & 1023u) != 0) continue;
      if (t0 == 0) t0 = gc_now();
      if (gc_now() - t0 > kStallNs || ld(&status->code) != 0) {
        raise(status, ECL_ERR_NO_CONVERGENCE, r);
        lost = true;
        break;
      }
    }
    if (!lost) marks[min(c, beyond)] = 1;
  }
  return __any_sync(kFull, lost);
}

// Per-warp staging of row segments: two buffers, each with its mbarrier and
// the parity of its next phase.  A segment starts at a 16-byte unit of the
// packed rows and has at most the buffer's entries; the copy is rounded up to
// 16 bytes (the row's slot has room).
struct CoreStage {
  unsigned short* base;  // the buffers, `seg` entries each; the mbarriers lie before them, the marks behind
  int seg;
  unsigned state = 0;  // bit b: parity of buffer b's next phase; bit 2 + b: a copy into it is in flight

  // (as few registers as can be, and no arrays, which would lie in local memory:
  // both cost on the chain)
  __device__ __forceinline__ unsigned short* buf(int b) const { return base + (b ? seg : 0); }
  __device__ __forceinline__ unsigned long long* bar(int b) const {
    return reinterpret_cast<unsigned long long*>(base) - 2 + b;
  }
  __device__ __forceinline__ unsigned char* marks() const { return reinterpret_cast<unsigned char*>(base + 2 * seg); }
  __device__ __forceinline__ void issue(int b, const int* nl2, int unit, int len) {
    state |= 4u << b;
    if ((threadIdx.x & 31) == 0)
      bulk_load(buf(b), reinterpret_cast<const char*>(nl2) + (size_t)unit * 16, (2u * (unsigned)len + 15u) & ~15u, bar(b));
  }
  // Waits for buffer b's copy.  False when the wait ran out.
  __device__ __forceinline__ bool wait(int b) {
    const bool ok = mbar_wait(bar(b), (state >> b) & 1u);
    if (ok) state ^= 5u << b;  // a copy that did not land stays listed for drain()
    return ok;
  }
  // Bounded wait for every copy still in flight (before leaving on an error).
  __device__ __forceinline__ void drain() {
    if (state & 4u) wait(0);
    if (state & 8u) wait(1);
  }
};

// The cluster colours the core: rank r goes to warp r mod (32 ctas), each warp
// takes its ranks in increasing order (the warp holding the lowest uncoloured
// rank can always finish it), and every colour is published to the core's
// copies and to color[] for gc_pull.  A warp's rows are a stream of segments;
// while one segment is scanned from shared memory the next is being copied.
// CAUTION for the look-ups: a malformed graph (reported by gc_init) may leave
// any 16-bit value in a row; 2 * 0xffff bytes is inside this CTA's shared
// memory for every core size, and a wait on what is read there ends on the
// status word.
// kWide: for cores with many rows of more than two segments, whose undecided
// entries go to a list.  A form of its own, as it costs each hop of any row: a
// sixteenth of the rows have to be such.  Measured, core, without / with the list:
// R-MAT-22 1.22 / 1.59 ms, a clique of 500 vertices 0.30 / 0.39, of 5000 47 / 40, a
// complete 40-partite graph of 4000 5.7 / 3.4.
template <bool kWide>
__device__ __forceinline__ void gc_core_run(const int* nl2, const int4* rowinfo, int* color, const GCCtl* ctl, int cap,
                                            Status* status) {
  extern __shared__ __align__(16) unsigned char s_core[];
  const int lane = threadIdx.x & 31;
  const int core = gc_core_size(ctl, cap);
  // rank r belongs to warp r mod (32 ctas) of the cluster, so each CTA takes
  // every ctas-th block of 32 consecutive ranks (dealing longer runs of
  // consecutive ranks to one CTA measured slower; single ranks, no faster)
  const int ctas = (int)cluster_ctas();
  const int warp = (int)cluster_rank() * kCoreWarps + (threadIdx.x >> 5);
  const int cwarps = ctas * kCoreWarps;
  unsigned short* col_s = reinterpret_cast<unsigned short*>(s_core);
  const int seg = gc_core_seg(cap);  // row entries staged at a time
  unsigned char* wbase = s_core + gc_core_colour_bytes(cap) + (size_t)(threadIdx.x >> 5) * gc_core_warp_bytes(seg);
  CoreStage stg;
  stg.base = reinterpret_cast<unsigned short*>(wbase + 2 * sizeof(unsigned long long));
  stg.seg = seg;
  unsigned char* const marks = stg.marks();
  unsigned short* pend = reinterpret_cast<unsigned short*>(marks + kMarkBytes);
  for (int r = threadIdx.x; r < core; r += kCoreThreads) col_st(&col_s[r], kUncoloured);
  gc_core_clear(marks, kMarkBytes - 1);
  if (lane == 0) {
    mbar_init(stg.bar(0));
    mbar_init(stg.bar(1));
    mbar_fence_init();
  }
  __syncthreads();
  if (ctas > 1) cluster_sync();  // every copy is initialised before any colour is stored into it

  // Row j of this warp is rank warp + cwarps j; lane L holds the row record
  // of row jb + L (records are fetched 32 rows at a time).
  int jb = -32;
  int3 rec = make_int3(0, 0, -1);
  auto row_of = [&](int j) -> int3 {  // all lanes call
    if ((j & ~31) != jb) {
      jb = j & ~31;
      const int r = warp + cwarps * (jb + lane);
      const int4 x = r < core ? rowinfo[r] : make_int4(0, 0, -1, 0);  // race-free: not written in this launch
      rec = make_int3(x.x, x.y, x.z);
    }
    const int src = j & 31;
    return make_int3(__shfl_sync(kFull, rec.x, src), __shfl_sync(kFull, rec.y, src), __shfl_sync(kFull, rec.z, src));
  };
  // Byte that takes the colours which cannot matter: h entries leave one of the
  // colours 0 .. h free.  So a row marks, searches and clears h + 2 bytes at most.
  unsigned beyond = 0;
  // looks entry e of the staged segment up; true when it is undecided
  auto look = [&](unsigned q) -> bool {
    const unsigned c = col_ld(&col_s[q]);
    marks[min(c, beyond)] = 1;
    return c == kUncoloured;
  };
  const int nrows = core > warp ? (core - warp + cwarps - 1) / cwarps : 0;
  // The first segment of the warp's next row with entries behind row j, into buffer
  // q (rows without any are skipped).
  auto next_row = [&](int j, int q) {
    for (int jn = j + 1; jn < nrows; jn++) {
      const int3 nx = row_of(jn);
      if (nx.y > 0) {
        stg.issue(q, nl2, nx.x, min(seg, nx.y));
        return;
      }
    }
  };
  int b = 0;  // buffer of the next row's first segment
  next_row(-1, b);
  for (int j = 0; j < nrows; j++) {
    const int r = warp + cwarps * j;
    const int3 row = row_of(j);
    const int unit = row.x, h = row.y, v = row.z;
    beyond = (unsigned)min(h + 1, kWin);
    bool stalled = false;
    int from = 0;  // all colours below are taken
    int np = 0;    // entries in `pend`
    // All of a row is scanned before any undecided entry is waited for: a scan
    // behind the last neighbour's colour would lie on the chain, and costs
    // microseconds among the other warps' polls.  Two segments at a time; of a
    // longer row the undecided ones so far go to a list (kWide), if it holds them.
    for (int off = 0; off < h && !stalled; off += 2 * seg) {
      const int f = unit + off / 8, second = h - off - seg;  // entries behind the first of the two
      __syncwarp();  // buffer b ^ 1 was scanned by every lane
      if (second > 0)
        stg.issue(b ^ 1, nl2, f + seg / 8, min(seg, second));
      else
        next_row(j, b ^ 1);
      unsigned open0 = 0, open1 = 0;
      for (int part = 0; part <= (second > 0); part++) {
        const int q = b ^ part, l = min(seg, h - off - part * seg);
        if (!__all_sync(kFull, stg.wait(q))) {  // every lane polls; the verdict is the warp's
          raise(status, ECL_ERR_NO_CONVERGENCE, r);
          stalled = true;
          break;
        }
        const unsigned short* sg = stg.buf(q);
        // eight entries a lane and step; bit 8 s + k of `wait`: entry k of the
        // lane's step s is undecided
        unsigned wait = 0;
        const uint4* sv = reinterpret_cast<const uint4*>(sg);
        for (int s = 0; 256 * s < l; s++) {
          const int e = 256 * s + 8 * lane;
          unsigned undecided = 0;
          if (e + 8 <= l) {
            const uint4 x = sv[32 * s + lane];
            const unsigned w[4] = {x.x, x.y, x.z, x.w};
            unsigned c[8];
#pragma unroll
            for (int k = 0; k < 8; k++) c[k] = col_ld(&col_s[(k & 1) ? w[k >> 1] >> 16 : w[k >> 1] & 0xffffu]);
#pragma unroll
            for (int k = 0; k < 8; k++) {
              marks[min(c[k], beyond)] = 1;
              undecided |= c[k] == kUncoloured ? 1u << k : 0u;
            }
          } else {
            for (int k = 0; e + k < l; k++) undecided |= look(sg[e + k]) ? 1u << k : 0u;
          }
          wait |= undecided << (8 * s);
        }
        if (part)
          open1 = wait;
        else
          open0 = wait;
      }
      if (kWide && second > seg) {
        const int kept = gc_core_keep(open0, open1, stg.buf(b), stg.buf(b ^ 1), pend, np);
        if (kept >= 0) np = kept, open0 = open1 = 0;
      }
      // Wait for the undecided ones: a lane goes round its own and takes whichever
      // is decided, so that none holds up the others.  (R-MAT-22, core: the ranks
      // in a list that the lanes share evenly, and the colours handed to registers
      // by votes and shuffles, 1.39 ms, with naps of 40 to 100 ns 1.47; this 1.21.)
      unsigned spins = 0, turn = 0;
      unsigned long long t0 = 0;
      __syncwarp();
      if (h >= kFromRow && (!kWide || second <= seg)) from = gc_core_mex(marks, 0, from, (int)beyond);
      if (from < 0) from = kWin;
      for (int part = 0; part <= (second > 0) && !stalled; part++) {
        const unsigned short* sg = stg.buf(b ^ part);
        unsigned wait = part ? open1 : open0;
        while (wait) {
          const unsigned behind = wait & ~((1u << turn) - 1u);
          const int k = __ffs(behind ? behind : wait) - 1;
          const unsigned c = col_ld(&col_s[sg[256 * (k >> 3) + 8 * lane + (k & 7)]]);
          turn = (k + 1) & 31;
          if (c != kUncoloured) {
            marks[min(c, beyond)] = 1;
            wait &= ~(1u << k);
          } else if ((++spins & 1023u) == 0) {
            if (t0 == 0) t0 = gc_now();
            if (gc_now() - t0 > kStallNs || ld(&status->code) != 0) {
              raise(status, ECL_ERR_NO_CONVERGENCE, r);
              stalled = true;
              break;
            }
          }
        }
      }
      stalled = __any_sync(kFull, stalled);
      if (second <= 0)
        b ^= 1;
      else if (second > seg && !stalled)
        stg.issue(b, nl2, f + seg / 4, min(seg, second - seg));
    }
    if (kWide && np > 0 && !stalled) stalled = gc_core_settle(pend, np, col_s, marks, beyond, r, status);
    if (stalled) {
      stg.drain();
      break;
    }
    __syncwarp();
    int c = gc_core_mex(marks, 0, from, (int)beyond);
    if (c < 0) c = gc_core_far(reinterpret_cast<const unsigned short*>(nl2) + (size_t)unit * 8, h, col_s, marks);
    if (lane == 0) {
      col_publish(&col_s[r], (unsigned)c, ctas);
      st(&color[v], c);
    }
    __syncwarp();
    // behind the publication, off the chain
    gc_core_clear(marks, (int)beyond);
    if (h > 0 && (h - 1) / seg % 2 == 1) next_row(j, b);  // both buffers were the row's own
  }
  // a CTA's shared memory must outlive every store the others make into it:
  // every warp, done or given up (each wait is bounded), meets here
  if (ctas > 1) cluster_sync();
}

__global__ void __launch_bounds__(kCoreThreads, 1) gc_core(const int* nl2, const int4* rowinfo,
                                                           int* __restrict__ color, const GCCtl* ctl,
                                                           int cap, Status* __restrict__ status) {
  dep_wait();
  if (16LL * ld(&ctl->nwide) > gc_core_size(ctl, cap))  // the same for all CTAs
    gc_core_run<true>(nl2, rowinfo, color, ctl, cap, status);
  else
    gc_core_run<false>(nl2, rowinfo, color, ctl, cap, status);
}

__global__ void __launch_bounds__(kTPB) gc_pull(int n, const int* __restrict__ nindex, const int* __restrict__ nl2,
                                                const int* __restrict__ hc, const int* __restrict__ order,
                                                int* __restrict__ color, GCCtl* __restrict__ ctl, int core_cap,
                                                unsigned long_nap, Status* __restrict__ status) {
  __shared__ unsigned s_bits[kTPB / 32][kMexWords];
  __shared__ int s_pend[kTPB / 32][kPend];
  const int lane = threadIdx.x & 31;
  unsigned* bits = s_bits[threadIdx.x >> 5];
  int* pend = s_pend[threadIdx.x >> 5];
  if (ld(&ctl->sort_failed)) return;
  const int nbig = ld(&ctl->nbig);
  const int gwarp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  // Ranks are dealt to warps round-robin and each warp takes its own in
  // increasing order -- no shared claim counter (one atomic per row on a
  // single word would serialise ~10^6 claims in L2).  Still deadlock-free:
  // the warp holding the lowest unfinished rank is working on it, and all of
  // that vertex's dependencies have lower ranks.
  // Long rows, ONE per warp at a time: every long row in flight scans its
  // higher-priority list concurrently, so the dense hub core's rows all wait
  // at the same time instead of one after another.
  // A row's vertex, its place and length, and its first entries are three
  // dependent loads, the last one from DRAM; they are made two, one and one
  // row ahead.  Bound by what is left: a round trip to L2 for the colours, and
  // the chain.  Measured, pull, nothing loaded ahead -> this: R-MAT-22 1.12 ->
  // 0.98 ms, G(3 M, 12 M) 0.246 -> 0.217.
  // ranks below the core size were coloured by gc_core
  const int r0 = gc_core_size(ctl, core_cap) + gwarp;
  auto vertex = [&](int r) { return r < nbig ? __ldg(&order[r]) : -1; };
  auto place = [&](int v, int& b, int& h) {
    b = v >= 0 ? __ldg(&nindex[v]) : 0;
    h = v >= 0 ? __ldg(&hc[v]) : 0;
  };
  int v = vertex(r0), v1 = vertex(min(r0, nbig) + nwarps);
  int b, h;
  place(v, b, h);
  int ahead[kAhead];
#pragma unroll
  for (int k = 0; k < kAhead; k++) ahead[k] = 32 * k + lane < h ? __ldg(&nl2[b + 32 * k + lane]) : 0;
  for (int r = r0; r < nbig; r += nwarps) {
    const int v2 = r < nbig - 2 * nwarps ? __ldg(&order[r + 2 * nwarps]) : -1;
    int b1, h1;
    place(v1, b1, h1);
    int next[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; k++) next[k] = 32 * k + lane < h1 ? __ldg(&nl2[b1 + 32 * k + lane]) : 0;
    const int c = gc_long_row(b, b + h, ahead, nl2, color, bits, pend, kPend, long_nap, status);
    if (c < 0) return;
    if (lane == 0) st(&color[v], c);
    __syncwarp();
    v = v1, v1 = v2, b = b1, h = h1;
#pragma unroll
    for (int k = 0; k < kAhead; k++) ahead[k] = next[k];
  }
  // Short rows: 32 consecutive ranks per warp step, every lane its own vertex
  // (the order holds the nkeys vertices with entries; the isolated ones were
  // coloured by gc_keys).  The next step's vertices and places are loaded a
  // step ahead, and the lines of its entries asked for.
  const int nk = min(ld(&ctl->nkeys), n);
  const int first = nbig + gwarp * 32 + lane;
  int sv = first < nk ? __ldg(&order[first]) : -1;
  int sb, sh;
  place(sv, sb, sh);
  for (int base = nbig + gwarp * 32; base < nk; base += nwarps * 32) {
    const int rn = base + lane + nwarps * 32;
    const int svn = rn < nk ? __ldg(&order[rn]) : -1;
    int sbn, shn;
    place(svn, sbn, shn);
    if (shn > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(nl2 + sbn));
    if (sv >= 0) {
      const int c = gc_short_row(sb, sh, nl2, color, status);
      if (c >= 0) st(&color[sv], c);
    }
    if (__any_sync(kFull, ld(&status->code) != 0)) return;
    sv = svn, sb = sbn, sh = shn;
  }
}

struct GCBufs {
  GCCtl* ctl;
  int* nl2;
  int* hc;
  unsigned long long* keys0;
  unsigned long long* keys1;
  int* vals0;
  int* vals1;
  int* order;
  unsigned* sort_temp;
  unsigned* vhash;
  int2* chunks;
  int4* rowinfo;
};

void gc_layout(Carve& c, int n, int m, bool uni, GCBufs* b) {
  b->ctl = c.take<GCCtl>(1);
  b->nl2 = c.take<int>((size_t)m + 4);  // 4 spare entries: the core's aligned bulk copies may round up into them
  b->hc = c.take<int>((size_t)n);
  b->keys0 = c.take<unsigned long long>((size_t)n);
  b->keys1 = c.take<unsigned long long>((size_t)n);
  b->vals0 = c.take<int>((size_t)n);
  b->vals1 = c.take<int>((size_t)n);
  b->order = c.take<int>((size_t)n);
  b->sort_temp = c.take<unsigned>(radix_temp_words(n));
  b->vhash = c.take<unsigned>(uni ? (size_t)n : 0);
  b->chunks = c.take<int2>(row_chunk_capacity(m, kMinChunk));
  b->rowinfo = c.take<int4>((size_t)std::min(n, kCoreMax));
}

}  // namespace

size_t gc_workspace_bytes(int n, int m, bool uni) {
  Carve c;
  GCBufs b;
  gc_layout(c, n, m, uni, &b);
  return c.bytes();
}

}  // namespace ecl

namespace ecl {

ecl_status gc_enqueue(const GraphDev& g, int* color, char* ws, Status* status, const DeviceInfo& dev,
                      cudaStream_t stream, const UnionInfo* uni, Marker mark) {
  Carve c{ws};
  GCBufs b;
  gc_layout(c, g.n, g.m, uni && uni->vbase, &b);
  // Blocks of the pull per SM: a knob, 2 by default.  Fewer warps poll
  // fewer undecided entries at a time; on R-MAT-22 two blocks per SM colour
  // faster than four (1.81 vs 2.15 ms) -- the polls of four blocks load L2
  // enough to slow the dependency chain they wait on.
  const int pull_blocks = dev.gc_pull_blocks > 0 ? dev.gc_pull_blocks : 2;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, gc_pull, kTPB, 0) != cudaSuccess || occ < 1)
    return ECL_ERR_CUDA;
  const int coop_grid = dev.sms * std::min(occ, pull_blocks);
  const int grid = dev.grid_blocks(kTPB, g.n, g.m);
  const RowChunks rc{b.chunks, &b.ctl->nchunks, (int)row_chunk_capacity(g.m, kMinChunk)};
  const Bins bins = bins_of(dev, Bins{kBinLane, kBinChunk});

  fill_ranges({{b.ctl, sizeof(GCCtl), 0}, {color, sizeof(int) * (size_t)g.n, 0xff}}, dev, stream);
  const unsigned* vhash = nullptr;
  if (uni && uni->vbase) {
    ECL_LAUNCH_NEXT(gc_union_hash, grid, kTPB, 0, stream, g.n, uni->vbase, uni->ngraphs, b.vhash);
    vhash = b.vhash;
  }
  // the priority keys first: gc_init compares neighbours by them
  ECL_LAUNCH_NEXT(gc_keys, grid, kTPB, 0, stream, g.n, g.m, g.nindex, b.keys0, b.keys1, b.vals1, vhash, color, b.ctl);
  const bool vec = (reinterpret_cast<uintptr_t>(g.nlist) & 15) == 0 && dev.row_vec;  // 16-byte row loads
  const int warps = dev.sms * (dev.max_threads_per_sm / 32);
  int group = 32;
  while (group > kSmallGroup && g.n / group < warps) group /= 2;
  const int init_grid = group == 32 ? grid : (g.n - 1) / (group * (kTPB / 32)) + 1;
  ECL_LAUNCH_NEXT(gc_init, init_grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, b.nl2, b.hc, rc, bins, group, vec,
                  b.keys0, status);
  ECL_LAUNCH_NEXT(gc_init_chunks, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, b.nl2, b.hc, rc, bins.chunk, vec, b.keys0,
             status);
  mark();
  // the nkeys appended pairs, sorted from (keys1, vals1); the per-vertex keys
  // in keys0 are dead once gc_init has run
  const ecl_status sorted = radix_order(b.keys1, b.vals1, b.keys0, b.vals0, b.order, g.n, &b.ctl->nkeys, &b.ctl->maxdeg,
                                  b.sort_temp, vhash == nullptr, &b.ctl->sort_bar, &b.ctl->sort_failed, dev, stream, status);
  if (sorted != ECL_OK) return sorted;
  const int* order = b.order;
  mark();
  // the hub core (the sort keys are dead now: their buffer holds the ranks)
  const int cap = std::min(std::min(dev.gc_core_ranks > 0 ? dev.gc_core_ranks : kCoreDefault, kCoreMax), g.n);
  int* rank = reinterpret_cast<int*>(b.keys0);
  // (no more blocks than a full core has rows for: every warp of the launch
  // asks for the core's size, and thousands of them queue at its word; a mesh
  // of 0.7 M vertices, no core at all: 11 + 12 us with one block per 256
  // vertices)
  ECL_LAUNCH_NEXT(gc_core_rank, std::min(grid, (cap - 1) / kTPB + 1), kTPB, 0, stream, order, rank, b.ctl, cap);
  ECL_LAUNCH_NEXT(gc_core_translate, std::min(grid, (cap - 1) / (kTPB / 32) + 1), kTPB, 0, stream, g.nindex, b.nl2, b.hc, order, rank, b.rowinfo, b.ctl, cap, status);
  ECL_CUDA_TRY(cudaFuncSetAttribute(gc_core, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gc_core_smem(cap)));
  // the core's cluster: as many CTAs as asked for when such a cluster fits
  // the device, else one CTA
  const int want = dev.gc_core_ctas > 0 ? dev.gc_core_ctas : kCoreCtas;
  int ctas = 1;
  if (want > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)want);
    cfg.blockDim = dim3((unsigned)kCoreThreads);
    cfg.dynamicSmemBytes = gc_core_smem(cap);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)want;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, gc_core, &cfg) == cudaSuccess && clusters >= 1)
      ctas = want;
    else
      cudaGetLastError();  // no such cluster here: one CTA
  }
  if (ctas > 1)
    ECL_CUDA_TRY(launch_cluster(gc_core, ctas, kCoreThreads, gc_core_smem(cap), stream, b.nl2, b.rowinfo, color,
                                b.ctl, cap, status));
  else
    ECL_LAUNCH_NEXT(gc_core, 1, kCoreThreads, gc_core_smem(cap), stream, b.nl2, b.rowinfo, color, b.ctl, cap, status);
  mark();
  // the long rows' polls back off to at most gc_poll_ns, 64 ns by default
  // (they carry the dependency chain; the short rows keep 512 ns)
  const unsigned long_nap = dev.gc_poll_ns > 0 ? (unsigned)dev.gc_poll_ns : 64u;
  ECL_CUDA_TRY(launch_cooperative(gc_pull, coop_grid, kTPB, stream, g.n, g.nindex, b.nl2, b.hc, order, color, b.ctl,
                                  cap, long_nap, status));
  mark();
  return ECL_OK;
}

}  // namespace ecl

extern "C" ecl_status ecl_gc(const ecl_graph_view* g, int32_t* color_out, ecl_opts* opts) {
  using namespace ecl;
  ecl_opts local{};
  if (!opts) opts = &local;
  if (!color_out) return ECL_ERR_INVALID_ARG;
  Solve s(g, opts);
  GraphNeeds needs;
  needs.symmetric = true;
  needs.no_self_loops = true;
  ecl_status st = s.begin(needs, g ? gc_workspace_bytes(g->nodes, g->edges) : 0);
  if (st != ECL_OK) return s.finish(st);
  int* color = s.output(color_out, (size_t)s.n);
  if (!color) return s.finish(ECL_ERR_OOM);
  GraphDev gd;
  gd.n = s.n;
  gd.m = s.m;
  gd.nindex = s.nindex;
  gd.nlist = s.nlist;
  gd.flags = g->flags;
  s.start_timer();
  st = gc_enqueue(gd, color, s.ws, s.status, s.dev, s.stream, nullptr, Marker{&s});
  s.stop_timer();
  return s.finish(st);
}

extern "C" ecl_status ecl_compute_gc(int32_t nodes, int32_t edges, const int32_t* nidx, const int32_t* nlist,
                                     int32_t* color) {
  ecl_graph_view g{nodes, edges, nidx, nlist, nullptr, ECL_HOST, 0};
  ecl_opts o{};
  return ecl_gc(&g, color, &o);
}

// ---- the colouring's critical path (a host-side diagnostic) --------------------
//
// The colour of a vertex is fixed only after every higher-priority neighbour
// has its own, so no schedule finishes faster than the longest chain of such
// dependencies.  This walks the priority order once on the host: hops[v] = 1 +
// the largest hops[u] over v's higher-priority entries u (0 with none), and a
// time model path[v] = the latest path[u] + the cost of one hop to v -- the
// shared-memory hop for a vertex the GPU colours in its core (the first
// min(long rows, core_ranks) ranks), the L2 hop for every other one.  The
// bench reports the resulting latency bound beside gc_pull's time.
extern "C" ecl_status ecl_gc_critical_path(const ecl_graph_view* g, int32_t core_ranks, double hop_core_ns,
                                           double hop_rest_ns, int32_t* hops, int32_t* hops_core, double* path_ns) {
  using namespace ecl;
  if (!g || g->location != ECL_HOST || g->nodes < 1 || g->edges < 0 || !g->nindex || (g->edges > 0 && !g->nlist))
    return ECL_ERR_INVALID_ARG;
  if (core_ranks < 0 || core_ranks > kCoreMax) return ECL_ERR_INVALID_ARG;
  const int n = g->nodes;
  const int* nindex = g->nindex;
  const int* nlist = g->nlist;
  for (int v = 0; v < n; v++)
    if (nindex[v] < 0 || nindex[v + 1] < nindex[v] || nindex[v + 1] > g->edges) return ECL_ERR_BAD_GRAPH;
  std::vector<unsigned long long> key((size_t)n);
  int nbig = 0;
  for (int v = 0; v < n; v++) {
    const unsigned deg = (unsigned)(nindex[v + 1] - nindex[v]);
    key[(size_t)v] = ((unsigned long long)deg << 32) | dev::ecl_hash((unsigned)v);
    nbig += deg > (unsigned)kWarpRow;
  }
  std::vector<int> by_rank((size_t)n);
  for (int v = 0; v < n; v++) by_rank[(size_t)v] = v;
  std::sort(by_rank.begin(), by_rank.end(), [&](int a, int b) {
    return key[(size_t)a] != key[(size_t)b] ? key[(size_t)a] > key[(size_t)b] : a > b;
  });
  std::vector<int> place((size_t)n);
  for (int r = 0; r < n; r++) place[(size_t)by_rank[(size_t)r]] = r;
  const int core = std::min(nbig, core_ranks > 0 ? core_ranks : kCoreDefault);
  std::vector<int> hop((size_t)n, 0);
  std::vector<double> path((size_t)n, 0.0);
  int best = 0, best_core = 0;
  double best_path = 0.0;
  for (int r = 0; r < n; r++) {
    const int v = by_rank[(size_t)r];
    int h = -1;
    double t = -1.0;
    for (int i = nindex[v]; i < nindex[v + 1]; i++) {
      const int u = nlist[i];
      if (u < 0 || u >= n) return ECL_ERR_BAD_GRAPH;
      if (u == v || place[(size_t)u] > r) continue;
      h = std::max(h, hop[(size_t)u]);
      t = std::max(t, path[(size_t)u]);
    }
    hop[(size_t)v] = h + 1;
    path[(size_t)v] = t < 0.0 ? 0.0 : t + (r < core ? hop_core_ns : hop_rest_ns);
    best = std::max(best, hop[(size_t)v]);
    if (r < core) best_core = std::max(best_core, hop[(size_t)v]);
    best_path = std::max(best_path, path[(size_t)v]);
  }
  if (hops) *hops = best;
  if (hops_core) *hops_core = best_core;
  if (path_ns) *path_ns = best_path;
  return ECL_OK;
}
