// Connected components (ECL-CC contract).
//
// Result contract (src/racefree/egr-input/CC/ECL-CC-atomic.cu): every vertex v
// hooks only along its list entries u = nlist[i] with u < v (:132, :174,
// :218), roots are always hooked larger -> smaller (:139-146) and flatten
// points each vertex at its root (:250-264).  Hence the label of v is the
// smallest vertex id of v's component in the graph whose edges are
// {(v, u) : u in list(v), u < v}.  That value does not depend on the schedule,
// so any union-find with the same hooking rule reproduces it bit for bit.
//
// B200 design (graphs flagged ECL_GRAPH_SYMMETRIC take the sampling path
// further down: link two entries of every list, find the giant component,
// then skip every list inside it):
//  * cc_init   - parent[v] = first smaller neighbour among the first
//                kInitScan entries (free hooks; the sampling path goes two
//                such steps).
//  * cc_hook   - one pass over the vertices, 32 per warp.  Lists of <= 16
//                entries are walked by their own lane; lists of up to
//                2048 entries are walked by the whole warp (ballot loop,
//                coalesced 128-byte nlist reads); longer lists are cut into
//                2048-entry chunk records for cc_chunks (both thresholds
//                are launch knobs).
//  * cc_chunks - warp per chunk record, so a 163k-entry R-MAT hub is spread
//                over ~160 warps instead of serialising one block.
//  * cc_flatten- label[v] = root(v).
// The parent array IS the output label array (no extra n-sized buffer).
// All parent accesses are device-scope relaxed atomics; links use CAS.
#include "solvers.cuh"

#include <algorithm>
#include <mutex>

namespace ecl {
namespace {

using namespace dev;

typedef unsigned long long u64;

constexpr int kTPB = 256;
// Default degree bins: lists of <= 16 entries per lane, chunk records of
// 2048 entries (a launch knob may change both).
constexpr Bins kCCBins{16, 2048};
constexpr int kInitScan = 8;   // entries cc_init looks at for a first smaller neighbour
constexpr int kInitHops = 2;   // hops of cc_init (R-MAT-22, whole solve: 1 hop 0.244 ms, 2 0.227, 4 0.217; G(3 M, 12 M): 0.354, 0.369, 0.396)
// ... and where every entry is linked afterwards, with nothing sampled first: two
// hops leave a vertex and the one between in two trees, whose link is one more
// that climbs through the hubs' words.  1 hop / 2 (median): 300 k vertices, 3 M
// entries to power-law ends 0.69 / 0.94 ms, from such 0.56 / 0.69; 10 M entries of
// 1 M vertices 0.87 / 0.81 and 0.71 / 0.68; uniform ends, 3 M entries 0.89 / 0.65, 8 M 0.36 / 0.37.
constexpr int kInitHopsAll = 1;

// Whether this solve is not wanted after all: an earlier launch has left
// something other than 0 at `off` (nullptr: it always is).
__device__ __forceinline__ bool cc_off(const u64* off) { return off && *off != 0; }

// Row [beg, end) of v, or empty when the row is malformed (cc_init reports it).
__device__ __forceinline__ void cc_row(const int* nindex, int v, int m, int& beg, int& end) {
  beg = __ldg(&nindex[v]);
  end = __ldg(&nindex[v + 1]);
  if (beg < 0 || end < beg || end > m) beg = end = 0;
}

// Entries outside [0, n) raise ECL_ERR_BAD_GRAPH and are skipped.
__device__ __forceinline__ bool cc_valid(int u, int n, Status* status) {
  if ((unsigned)u < (unsigned)n) return true;
  raise(status, ECL_ERR_BAD_GRAPH, u);
  return false;
}

struct CCCounters {
  int nchunks;
  int giant;  // root of the sampled largest component (symmetric path)
  int pad[62];
};

// Whose entries the symmetric path need not link: one tree for all vertices,
// or one for each graph of a union (no entry leaves its graph, so the trees of
// two graphs have no entry between them to be missed).
struct Giants {
  const int* root;             // the tree's root, or one a graph
  const int* vbase = nullptr;  // union: the graphs' first vertices
  int ngraphs = 0;
};

// Root of v with path splitting.  Parent pointers only ever point at
// smaller ids, so a vertex is a root iff parent[v] == v.
// (from: parent[v], as loaded).
__device__ __forceinline__ int cc_root_from(int v, int from, int* parent) {
  int cur = from;
  if (cur == v) return v;
  int prev = v;
  int next;
  while (cur > (next = ld(&parent[cur]))) {
    st(&parent[prev], next);
    prev = cur;
    cur = next;
  }
  return cur;
}

__device__ __forceinline__ int cc_root(int v, int* parent) { return cc_root_from(v, ld(&parent[v]), parent); }

// Links the trees rooted (as last seen) at a and b; returns the root that
// survived the link as last seen by this thread.
__device__ __forceinline__ int cc_link(int a, int b, int* parent) {
  while (a != b) {
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int seen = cas(&parent[a], a, b);
    if (seen == a) return b;
    // Another thread already hung a under b: the two trees are one.  On a
    // mesh every vertex of a column links the same pair of roots, and all but
    // one would otherwise walk the freshly linked chain of roots.
    if (seen == b) return b;
    a = cc_root(seen, parent);
    b = cc_root(b, parent);
  }
  return a;
}

// Joins the trees of u and v without first walking to either root (the Link
// step of Sutton, Ben-Nun and Barak, IPDPS 2018): look one level above the
// larger side; if that already is the smaller side the trees are one, if it
// is a root hang it under the smaller side, otherwise climb two levels and
// retry.  Parents only point at smaller ids, so the loop ends.  A mesh links
// the same pair of roots from every vertex of a column; a full root walk
// there follows a chain of roots that grows while it is being walked.
__device__ __forceinline__ void cc_union(int u, int v, int* parent) {
  int p1 = ld(&parent[u]);
  int p2 = ld(&parent[v]);
  while (p1 != p2) {
    const int high = max(p1, p2), low = min(p1, p2);
    const int ph = ld(&parent[high]);
    if (ph == low) return;
    if (ph == high && cas(&parent[high], high, low) == high) return;
    p1 = ld(&parent[ld(&parent[high])]);
    p2 = ld(&parent[low]);
  }
}

// First smaller neighbour of v among the first kInitScan entries of its list
// (v itself: none).  Only those are looked at: the hook is an optional head
// start (the labels do not depend on it), and scanning a whole hub row from
// one thread would serialise a 163k-entry R-MAT hub.
__device__ __forceinline__ int cc_first_smaller(int v, int beg, int end, const int* nlist) {
  const int stop = min(end, beg + kInitScan);
  for (int i = beg; i < stop; i++) {
    const int u = __ldg(&nlist[i]);
    if (u < v && u >= 0) return u;
  }
  return v;
}

// parent[v] = the vertex kHops first-smaller-neighbour hops from v.  The
// hops go through the CSR, which nothing writes, so L1 serves the rows of the
// hubs that most vertices of a power-law graph hop to; the same steps through
// parent[] afterwards queue at the hubs' words.
// Also checks the CSR rows once: a malformed row (end < beg, or outside
// [0, m]) raises ECL_ERR_BAD_GRAPH and is treated as empty by every kernel.
template <int kHops>
__global__ void __launch_bounds__(kTPB) cc_init(int n, int m, const int* __restrict__ nindex,
                                                const int* __restrict__ nlist, int* __restrict__ parent,
                                                CCCounters* ctr, const u64* off,
                                                Status* __restrict__ status) {
  dep_wait();
  if (cc_off(off)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctr->nchunks = 0;  // race-free: first used by later launches
  for (int v = blockIdx.x * kTPB + threadIdx.x; v < n; v += gridDim.x * kTPB) {
    int beg = __ldg(&nindex[v]), end = __ldg(&nindex[v + 1]);
    if (beg < 0 || end < beg || end > m) {
      raise(status, ECL_ERR_BAD_GRAPH, v);
      beg = end = 0;
    }
    int p = cc_first_smaller(v, beg, end, nlist);
    for (int h = 1; h < kHops && p != v; h++) {
      cc_row(nindex, p, m, beg, end);
      const int q = cc_first_smaller(p, beg, end, nlist);
      if (q == p) break;
      p = q;
    }
    parent[v] = p;  // race-free: thread-owned init, no reader in this launch
  }
}

// Chunk records of chunk_capacity(m, chunk) cover every long row of a CSR
// whose rows do not overlap (a row of d > chunk entries needs
// ceil(d / chunk) < 2 d / chunk records).  A malformed CSR with overlapping
// rows can ask for more: the excess raises ECL_ERR_BAD_GRAPH and is not
// written.
constexpr int chunk_capacity(int m, int chunk) { return 2 * (m / chunk) + 2; }

__device__ __forceinline__ void cc_push_chunks(int v, int beg, int deg, int chunk, int2* chunks, int cap,
                                               CCCounters* ctr, Status* status) {
  const int nc = (deg + chunk - 1) / chunk;
  const int at = fetch_add(&ctr->nchunks, nc);
  for (int c = 0; c < nc; c++) {
    if ((unsigned)(at + c) < (unsigned)cap)
      chunks[at + c] = make_int2(v, beg + c * chunk);  // race-free: the slot is this reservation's, no reader in this launch
    else
      raise(status, ECL_ERR_BAD_GRAPH, v);
  }
}

// Records the chunk kernels may read: the requested count clamped to cap.
__device__ __forceinline__ int cc_chunk_total(const CCCounters* ctr, int cap) {
  const int c = ctr->nchunks;
  return (c < 0 || c > cap) ? cap : c;
}

__global__ void __launch_bounds__(kTPB) cc_hook(int n, int m, const int* __restrict__ nindex,
                                                const int* __restrict__ nlist, int* __restrict__ parent,
                                                int2* __restrict__ chunks, int chunk_cap, Bins bins,
                                                CCCounters* ctr, Status* __restrict__ status) {
  dep_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  for (int base = warp * 32; base < n; base += nwarps * 32) {
    const int v = base + lane;
    int beg = 0, end = 0;
    if (v < n) cc_row(nindex, v, m, beg, end);
    const int deg = end - beg;
    if (deg > bins.chunk) {
      cc_push_chunks(v, beg, deg, bins.chunk, chunks, chunk_cap, ctr, status);
    } else if (deg > 0 && deg <= bins.lane) {
      int rv = -1;
      for (int i = beg; i < end; i++) {
        const int u = __ldg(&nlist[i]);
        if (u < v && cc_valid(u, n, status)) {
          if (rv < 0) rv = cc_root(v, parent);
          const int ru = cc_root(u, parent);
          if (ru != rv) rv = cc_link(rv, ru, parent);
        }
      }
    }
    // Medium lists: the whole warp walks one list at a time.
    unsigned mid = __ballot_sync(kFull, deg > bins.lane && deg <= bins.chunk);
    while (mid) {
      const int who = __ffs(mid) - 1;
      mid &= mid - 1;
      const int wv = __shfl_sync(kFull, v, who);
      const int wbeg = __shfl_sync(kFull, beg, who);
      const int wend = __shfl_sync(kFull, end, who);
      int rv = -1;
      for (int i = wbeg + lane; i < wend; i += 32) {
        const int u = __ldg(&nlist[i]);
        if (u < wv && cc_valid(u, n, status)) {
          if (rv < 0) rv = cc_root(wv, parent);
          const int ru = cc_root(u, parent);
          if (ru != rv) rv = cc_link(rv, ru, parent);
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kTPB) cc_chunks(int n, const int* __restrict__ nindex,
                                                  const int* __restrict__ nlist, int* __restrict__ parent,
                                                  const int2* chunks, int chunk_cap, int chunk,
                                                  const CCCounters* ctr, Status* __restrict__ status) {
  dep_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  const int total = cc_chunk_total(ctr, chunk_cap);
  for (int c = warp; c < total; c += nwarps) {
    const int2 rec = chunks[c];  // race-free: not written in this launch
    const int v = rec.x;
    const int end = min(rec.y + chunk, __ldg(&nindex[v + 1]));
    int rv = -1;
    for (int i = rec.y + lane; i < end; i += 32) {
      const int u = __ldg(&nlist[i]);
      if (u < v && cc_valid(u, n, status)) {
        if (rv < 0) rv = cc_root(v, parent);
        const int ru = cc_root(u, parent);
        if (ru != rv) rv = cc_link(rv, ru, parent);
      }
    }
  }
}

// parent[v] = root(v) by pointer jumping: each thread only rewrites its own
// parent[v], once per step, and steps to the parent of its current target.
// Threads on the same chain run side by side, so every step reads a target
// that has itself jumped -- a chain of depth D is flattened in about log2(D)
// dependent loads per thread instead of D (a mesh builds chains as long as a
// grid column).  parent[v] has no other writer during the launch, so the
// array ends fully flat.
//
// A root stays one for the whole launch, so a thread does not look again at
// the root that it met last: with a giant component every vertex would
// otherwise end on the same word, and its L2 slice would be the bound.  Hence
// a grid that gives each thread several vertices of a large graph
// (flatten_blocks), kFlattenBatch of them in flight; chains that have met share
// the load.  The batch's chains walked one after another took 31 us on a
// 1024 x 1024 grid (512 deep), side by side 23.
constexpr int kFlattenBatch = 4;

// kMark, kMarkUnion: also ing[v] = whether v's root is the sampled giant
// component's (of its graph).
enum : int { kPlain = 0, kMark = 1, kMarkUnion = 2 };
template <int kWhat>
__global__ void __launch_bounds__(kTPB) cc_flatten(int n, int* __restrict__ parent, Giants gi,
                                                   unsigned char* __restrict__ ing, const u64* off) {
  dep_wait();
  if (cc_off(off)) return;
  const int stride = gridDim.x * kTPB;
  const int giant = kWhat == kMark ? gi.root[0] : -1;
  int known = -1;  // a root of this launch
  for (long long v0 = blockIdx.x * kTPB + threadIdx.x; v0 < n; v0 += (long long)stride * kFlattenBatch) {
    int q[kFlattenBatch];
    bool go[kFlattenBatch];
    bool any = false;
#pragma unroll
    for (int k = 0; k < kFlattenBatch; k++) {
      const long long v = v0 + (long long)k * stride;
      q[k] = v < n ? ld(&parent[v]) : -1;
    }
#pragma unroll
    for (int k = 0; k < kFlattenBatch; k++) {
      go[k] = q[k] >= 0 && q[k] != (int)(v0 + (long long)k * stride) && q[k] != known;
      any |= go[k];
    }
    while (any) {
      int pp[kFlattenBatch];
#pragma unroll
      for (int k = 0; k < kFlattenBatch; k++) {
        bool first = go[k];
#pragma unroll
        for (int j = 0; j < k; j++) first = first && !(go[j] && q[j] == q[k]);
        if (first) pp[k] = ld(&parent[q[k]]);
      }
#pragma unroll
      for (int k = 1; k < kFlattenBatch; k++)
#pragma unroll
        for (int j = k - 1; j >= 0; j--)  // the smallest such j is one that loaded
          if (go[k] && go[j] && q[j] == q[k]) pp[k] = pp[j];
#pragma unroll
      for (int k = 0; k < kFlattenBatch; k++) {
        if (!go[k]) continue;
        if (pp[k] < q[k]) {
          st(&parent[(int)(v0 + (long long)k * stride)], pp[k]);
          q[k] = pp[k];
        } else {
          known = q[k];
          go[k] = false;
        }
      }
      any = false;
#pragma unroll
      for (int k = 0; k < kFlattenBatch; k++) {
        go[k] = go[k] && q[k] != known;
        any |= go[k];
      }
    }
    if (kWhat != kPlain) {
#pragma unroll
      for (int k = 0; k < kFlattenBatch; k++)
        if (q[k] >= 0) {
          const long long v = v0 + (long long)k * stride;
          // race-free: thread-owned, no reader in this launch
          ing[v] = q[k] == (kWhat == kMarkUnion ? gi.root[union_graph_of(gi.vbase, gi.ngraphs, (int)v)] : giant);
        }
    }
  }
}

int flatten_blocks(const DeviceInfo& dev, int n) {
  return std::min(dev.grid_blocks(kTPB, n, 0), dev.sms * 8);
}

// ---- symmetric graphs: sampling + giant-component skip ----------------------
//
// For a symmetric graph the components over the entries u < v are the plain
// connected components, so every entry may be used in either direction
// (Sutton, Ben-Nun and Barak, "Optimizing parallel graph connectivity
// computation via subgraph sampling", IPDPS 2018).  Links still hook the
// larger root under the smaller one, so the labels stay the minimum ids.

// Sampling: cc_init hooks every vertex to its first smaller neighbour -- one
// store, no atomics -- and after a full compression cc_sample links one more
// entry of every list: the first where the list starts with a larger id (that
// vertex was left a root, most likely), the second of the others.  A full
// compression comes between any two steps, so every find starts one step from
// its root: on a mesh, linking both samples at once builds chains as long as a
// grid column.
//
// The links run in two launches, an eighth of the vertices first.  While the
// giant component forms, every link climbs through the same few words, and
// their L2 slices serialise it; once an eighth of the links is made and
// flattened, the others mostly find their two ends in one tree after two loads
// of words of their own (an eighth is enough for the giant component to form:
// with a 32nd, G(3 M, 12 M) takes 1.27 ms).  Measured, whole solve, both
// entries linked by all vertices at once -> this, with cc_flatten's known
// roots: G(3 M, 12 M) 1.68 -> 0.37 ms, G(150 k, 600 k) 0.19 -> 0.09, R-MAT-22
// 0.29 -> 0.22, 1024 x 1024 grid 0.122 -> 0.120.
template <int kPart>  // 0: one vertex in kFirstOf, 1: the others, 2: all
__global__ void __launch_bounds__(kTPB) cc_sample(int n, int m, const int* __restrict__ nindex,
                                                  const int* __restrict__ nlist, int* __restrict__ parent,
                                                  const u64* off, Status* __restrict__ status) {
  dep_wait();
  if (cc_off(off)) return;
  constexpr int kFirstOf = 8;
  const int count = kPart == 0 ? (n - 1) / kFirstOf + 1 : n;
  for (int i = blockIdx.x * kTPB + threadIdx.x; i < count; i += gridDim.x * kTPB) {
    const int v = kPart == 0 ? i * kFirstOf : i;
    if (kPart == 1 && v % kFirstOf == 0) continue;
    int beg, end;
    cc_row(nindex, v, m, beg, end);
    if (beg >= end) continue;
    int u = __ldg(&nlist[beg]);
    if (u < v && beg + 1 < end) u = __ldg(&nlist[beg + 1]);
    if (u == v || !cc_valid(u, n, status)) continue;
    cc_union(v, u, parent);
  }
}

// From this many vertices on the sample is split: below, the two more launches
// cost more than the contention they avoid.
constexpr int kSplitSample = 1 << 13;

// One block (a graph): the most frequent root among 1024 sampled vertices, counted in a
// hash table in shared memory (a sort of the samples took 9 us, this 3).  The
// links are done when it runs, so the roots it walks to are the final ones.
constexpr int kGiantSlots = 2048;

__global__ void __launch_bounds__(1024) cc_giant(int n, const int* parent, const int* __restrict__ vbase,
                                                 int* __restrict__ root, const u64* off) {
  dep_wait();
  if (cc_off(off)) return;
  const int base = vbase ? __ldg(&vbase[blockIdx.x]) : 0;
  const int size = vbase ? __ldg(&vbase[blockIdx.x + 1]) - base : n;
  __shared__ int s_root[kGiantSlots], s_count[kGiantSlots];
  __shared__ unsigned long long s_best[32];
  const int t = threadIdx.x;
  for (int i = t; i < kGiantSlots; i += 1024) s_root[i] = -1, s_count[i] = 0;
  __syncthreads();
  int r = base + (int)(ecl_hash((unsigned)t * 2654435761u + 97u) % (unsigned)size), p;
  while ((p = ld(&parent[r])) != r) r = p;
  const unsigned same = __match_any_sync(kFull, r);
  if ((t & 31) == __ffs(same) - 1) {
    // at most 1024 roots in 2048 slots: the probe ends
    int h = (int)(((unsigned)r * 2654435761u) >> 21);
    for (;; h = (h + 1) & (kGiantSlots - 1)) {
      const int c = atomicCAS(&s_root[h], -1, r);
      if (c == -1 || c == r) break;
    }
    atomicAdd(&s_count[h], __popc(same));
  }
  __syncthreads();
  unsigned long long key = 0;  // largest count, ties to the smallest root
  for (int i = t; i < kGiantSlots; i += 1024)
    if (s_root[i] >= 0) key = max(key, ((unsigned long long)s_count[i] << 32) | (0xffffffffu - (unsigned)s_root[i]));
  for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(kFull, key, o));
  if ((t & 31) == 0) s_best[t >> 5] = key;
  __syncthreads();
  if (t < 32) {
    key = s_best[t];
    for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(kFull, key, o));
    if (t == 0) root[blockIdx.x] = (int)(0xffffffffu - (unsigned)key);
  }
}

// Remaining entries of vertices outside the giant component.  An entry is
// linked when u < v (the other direction is handled from u) or when u is in
// the giant component (u skips its list entirely).
__device__ __forceinline__ bool cc_rest_wanted(int u, int v, const unsigned char* ing) {
  return u != v && (u < v || ing[u]);  // race-free: not written in this launch
}

// A warp of cc_rest takes `group` (a power of two, at most 32) vertices at a time:
// 32, and down to this many where the lists are longer than a lane's on average
// and groups of 32 would leave warps of the device without any, as a group's
// lists run one after another.  32 -> this, whole solve: 30 cliques of 300 vertices
// 208 -> 84 us, 2000 of 40 109 -> 84; SCC of the former 239 -> 110.
constexpr int kSmallGroup = 4;

__global__ void __launch_bounds__(kTPB) cc_rest(int n, int m, const int* __restrict__ nindex,
                                                const int* __restrict__ nlist, int* __restrict__ parent,
                                                const unsigned char* ing, int2* __restrict__ chunks,
                                                int chunk_cap, Bins bins, int group, CCCounters* ctr,
                                                const u64* off, Status* __restrict__ status) {
  dep_wait();
  if (cc_off(off)) return;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  for (unsigned base = warp * group; base < (unsigned)n; base += nwarps * group) {
    const int v = lane < group ? (int)min(base + lane, (unsigned)n) : n;
    int beg = 0, end = 0;
    if (v < n && !ing[v]) cc_row(nindex, v, m, beg, end);  // race-free: not written in this launch
    const int deg = end - beg;
    if (deg > bins.chunk) {
      cc_push_chunks(v, beg, deg, bins.chunk, chunks, chunk_cap, ctr, status);
    } else if (deg > 0 && deg <= bins.lane) {
      int rv = -1;
      for (int i = beg; i < end; i++) {
        const int u = __ldg(&nlist[i]);
        if (cc_valid(u, n, status) && cc_rest_wanted(u, v, ing)) {
          if (rv < 0) rv = cc_root(v, parent);
          const int pu = ld(&parent[u]);
          if (pu == rv) continue;  // linked, and no look at the root's word, which all its tree's entries share
          const int ru = cc_root_from(u, pu, parent);
          if (ru != rv) rv = cc_link(rv, ru, parent);
        }
      }
    }
    unsigned mid = __ballot_sync(kFull, deg > bins.lane && deg <= bins.chunk);
    while (mid) {
      const int who = __ffs(mid) - 1;
      mid &= mid - 1;
      const int wv = __shfl_sync(kFull, v, who);
      const int wbeg = __shfl_sync(kFull, beg, who);
      const int wend = __shfl_sync(kFull, end, who);
      int rv = -1;
      for (int i = wbeg + lane; i < wend; i += 32) {
        const int u = __ldg(&nlist[i]);
        if (cc_valid(u, n, status) && cc_rest_wanted(u, wv, ing)) {
          if (rv < 0) rv = cc_root(wv, parent);
          const int pu = ld(&parent[u]);
          if (pu == rv) continue;  // linked, and no look at the root's word, which all its tree's entries share
          const int ru = cc_root_from(u, pu, parent);
          if (ru != rv) rv = cc_link(rv, ru, parent);
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kTPB) cc_rest_chunks(int n, const int* __restrict__ nindex,
                                                       const int* __restrict__ nlist, int* __restrict__ parent,
                                                       const unsigned char* ing,
                                                       const int2* chunks, int chunk_cap, int chunk,
                                                       const CCCounters* ctr, const u64* off,
                                                       Status* __restrict__ status) {
  dep_wait();
  if (cc_off(off)) return;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  const int total = cc_chunk_total(ctr, chunk_cap);
  for (int c = warp; c < total; c += nwarps) {
    const int2 rec = chunks[c];  // race-free: not written in this launch
    const int v = rec.x;
    const int end = min(rec.y + chunk, __ldg(&nindex[v + 1]));
    int rv = -1;
    for (int i = rec.y + lane; i < end; i += 32) {
      const int u = __ldg(&nlist[i]);
      if (cc_valid(u, n, status) && cc_rest_wanted(u, v, ing)) {
        if (rv < 0) rv = cc_root(v, parent);
        const int pu = ld(&parent[u]);
        if (pu == rv) continue;  // as cc_rest
        const int ru = cc_root_from(u, pu, parent);
        if (ru != rv) rv = cc_link(rv, ru, parent);
      }
    }
  }
}

void cc_layout(Carve& c, int n, int m, CCCounters** ctr, int2** chunks, unsigned char** ing = nullptr) {
  *ctr = c.take<CCCounters>(1);
  *chunks = c.take<int2>((size_t)chunk_capacity(m, kMinChunk));
  unsigned char* g = c.take<unsigned char>((size_t)n);
  if (ing) *ing = g;
}

}  // namespace

size_t cc_workspace_bytes(int n, int m) {
  Carve c;
  CCCounters* ctr;
  int2* chunks;
  cc_layout(c, n, m, &ctr, &chunks);
  return c.bytes();
}

}  // namespace ecl

namespace ecl {

ecl_status cc_enqueue(const GraphDev& g, int* parent, char* ws, Status* status, const DeviceInfo& dev,
                      cudaStream_t stream, Marker mark, const UnionInfo* uni, const u64* off) {
  Carve c{ws};
  CCCounters* ctr;
  int2* chunks;
  unsigned char* ing;
  cc_layout(c, g.n, g.m, &ctr, &chunks, &ing);
  const int grid = dev.grid_blocks(kTPB, g.n, g.m);
  const Bins bins = bins_of(dev, kCCBins);
  const int cap = chunk_capacity(g.m, kMinChunk);  // cc_layout sized the records for the smallest chunk
  if (g.flags & ECL_GRAPH_SYMMETRIC) {
    ECL_LAUNCH_NEXT(cc_init<kInitHops>, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent, ctr, off, status);
    ECL_LAUNCH_NEXT(cc_flatten<kPlain>, flatten_blocks(dev, g.n), kTPB, 0, stream, g.n, parent, Giants{}, nullptr, off);
    if (g.n >= kSplitSample) {
      ECL_LAUNCH_NEXT(cc_sample<0>, dev.grid_blocks(kTPB, g.n / 8, 0), kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent,
                 off, status);
      ECL_LAUNCH_NEXT(cc_flatten<kPlain>, flatten_blocks(dev, g.n), kTPB, 0, stream, g.n, parent, Giants{}, nullptr, off);
      ECL_LAUNCH_NEXT(cc_sample<1>, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent, off, status);
    } else {
      ECL_LAUNCH_NEXT(cc_sample<2>, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent, off, status);
    }
    // A union has a large component in every graph.  With one tree for all of
    // it, cc_rest had the entries of 95 of 96 graphs to look at (28 M in all):
    // 540 us, and 79 in cc_rest_chunks.
    const bool per_graph = uni && uni->vbase && uni->giants;
    const Giants gi = per_graph ? Giants{uni->giants, uni->vbase, uni->ngraphs} : Giants{&ctr->giant};
    ECL_LAUNCH_NEXT(cc_giant, per_graph ? uni->ngraphs : 1, 1024, 0, stream, g.n, parent, gi.vbase,
                    per_graph ? uni->giants : &ctr->giant, off);
    ECL_LAUNCH_NEXT(per_graph ? cc_flatten<kMarkUnion> : cc_flatten<kMark>, flatten_blocks(dev, g.n), kTPB, 0, stream, g.n, parent, gi, ing, off);
    mark();
    int group = 32;
    if (g.m / g.n > bins.lane)  // kSmallGroup says why
      while (group > kSmallGroup && g.n / group < dev.sms * (dev.max_threads_per_sm / 32)) group /= 2;
    ECL_LAUNCH_NEXT(cc_rest, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent, ing, chunks, cap, bins, group, ctr,
               off, status);
    mark();
    ECL_LAUNCH_NEXT(cc_rest_chunks, grid, kTPB, 0, stream, g.n, g.nindex, g.nlist, parent, ing, chunks, cap, bins.chunk,
               ctr, off, status);
    mark();
    ECL_LAUNCH_NEXT(cc_flatten<kPlain>, flatten_blocks(dev, g.n), kTPB, 0, stream, g.n, parent, Giants{}, nullptr, off);
    mark();
    return ECL_OK;
  }
  ECL_LAUNCH_NEXT(cc_init<kInitHopsAll>, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent, ctr, nullptr, status);
  mark();
  ECL_LAUNCH_NEXT(cc_hook, grid, kTPB, 0, stream, g.n, g.m, g.nindex, g.nlist, parent, chunks, cap, bins, ctr, status);
  mark();
  ECL_LAUNCH_NEXT(cc_chunks, grid, kTPB, 0, stream, g.n, g.nindex, g.nlist, parent, chunks, cap, bins.chunk, ctr, status);
  mark();
  ECL_LAUNCH_NEXT(cc_flatten<kPlain>, flatten_blocks(dev, g.n), kTPB, 0, stream, g.n, parent, Giants{}, nullptr, nullptr);
  mark();
  return ECL_OK;
}

}  // namespace ecl

extern "C" ecl_status ecl_cc(const ecl_graph_view* g, int32_t* label, ecl_opts* opts) {
  using namespace ecl;
  ecl_opts local{};
  if (!opts) opts = &local;
  if (!label) return ECL_ERR_INVALID_ARG;
  Solve s(g, opts);
  // The sampling path of a graph flagged ECL_GRAPH_SYMMETRIC uses every entry
  // in both directions, so validation (opts->validate) checks that flag: an
  // asymmetric graph carrying it would get labels other than the reference's
  // u < v hooking gives.
  GraphNeeds needs;
  needs.symmetric = g && (g->flags & ECL_GRAPH_SYMMETRIC);
  ecl_status st = s.begin(needs, g ? cc_workspace_bytes(g->nodes, g->edges) : 0);
  if (st != ECL_OK) return s.finish(st);
  int* parent = s.output(label, (size_t)s.n);
  if (!parent) return s.finish(ECL_ERR_OOM);
  GraphDev gd;
  gd.n = s.n;
  gd.m = s.m;
  gd.nindex = s.nindex;
  gd.nlist = s.nlist;
  gd.flags = g->flags;
  s.start_timer();
  st = cc_enqueue(gd, parent, s.ws, s.status, s.dev, s.stream, Marker{&s});
  s.stop_timer();
  return s.finish(st);
}

// ---- allocation-free variant --------------------------------------------------
//
// ecl_cc_noalloc runs the same four kernels with its scratch (status block,
// counters, chunk records) in a fixed array that lives in this library's
// device memory, so the call itself allocates nothing.  Every GPU that loads
// the library holds the array until the process exits.

namespace ecl {
namespace {

constexpr size_t kNoAllocBytes = ECL_CC_NOALLOC_SCRATCH_BYTES;
// The allocation-free path always uses the default bins (no knob may enlarge
// its fixed array), so its records are sized for kCCBins.chunk.
static_assert(kStatusBytes + sizeof(CCCounters) + 256 +
                      sizeof(int2) * (size_t)chunk_capacity(ECL_CC_NOALLOC_MAX_EDGES, kCCBins.chunk) <=
                  kNoAllocBytes,
              "no-alloc scratch too small for ECL_CC_NOALLOC_MAX_EDGES");

static __device__ __align__(256) unsigned char g_cc_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
struct NoAllocSlot {
  unsigned long long ctx = 0;  // id of the context the address belongs to
  void* addr = nullptr;        // device address of g_cc_noalloc_scratch in it
};
NoAllocSlot g_noalloc_slot[64];

// Device address of g_cc_noalloc_scratch on the current device (host code
// cannot use the symbol itself as a pointer).  It is looked up once per
// device and kept with the context it was found in: after cudaDeviceReset
// the device has a new primary context, the module is loaded again, and the
// address is looked up again instead of reusing a dead one.
ecl_status noalloc_scratch(int device, void** out) {
  if (device < 0 || device >= 64) return ECL_ERR_NO_DEVICE;
  const unsigned long long ctx = context_id();
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoAllocSlot& slot = g_noalloc_slot[device];
  if (ctx == 0 || slot.ctx != ctx || !slot.addr) {  // (0: no context yet; the look-up makes it)
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_cc_noalloc_scratch);
    if (e != cudaSuccess) {
      set_last_error("cudaGetSymbolAddress(g_cc_noalloc_scratch)", e);
      return ECL_ERR_CUDA;
    }
    slot.ctx = context_id();
    slot.addr = p;
  }
  *out = slot.addr;
  return ECL_OK;
}

}  // namespace
}  // namespace ecl

extern "C" ecl_status ecl_cc_noalloc(int32_t nodes, int32_t edges, const int32_t* nindex, const int32_t* nlist,
                                     int32_t* label, void* stream_ptr) {
  using namespace ecl;
  if (nodes < 1 || edges < 0) return ECL_ERR_BAD_GRAPH;
  if (!nindex || !label || (edges > 0 && !nlist)) return ECL_ERR_INVALID_ARG;
  if (edges > ECL_CC_NOALLOC_MAX_EDGES) {
    set_last_error_msg("ecl_cc_noalloc: graph has more CSR entries than ECL_CC_NOALLOC_MAX_EDGES; use ecl_cc");
    return ECL_ERR_UNSUPPORTED;
  }
  DeviceInfo dev;
  ecl_status st = current_device(&dev);
  if (st != ECL_OK) return st;
  void* base = nullptr;
  st = noalloc_scratch(dev.device, &base);
  if (st != ECL_OK) return st;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  Status* status = static_cast<Status*>(base);
  Carve c{static_cast<char*>(base) + kStatusBytes};
  CCCounters* ctr;
  int2* chunks;
  cc_layout(c, nodes, edges, &ctr, &chunks);
  // The array keeps the previous call's contents: clear the status block and
  // the counters (adjacent, at the front of the array) before every solve.
  ECL_CUDA_TRY(cudaMemsetAsync(base, 0, kStatusBytes + sizeof(CCCounters), stream));
  const int grid = dev.grid_blocks(kTPB, nodes, edges);
  ECL_LAUNCH_NEXT(cc_init<kInitHopsAll>, grid, kTPB, 0, stream, nodes, edges, nindex, nlist, label, ctr, nullptr, status);
  ECL_LAUNCH_NEXT(cc_hook, grid, kTPB, 0, stream, nodes, edges, nindex, nlist, label, chunks,
             chunk_capacity(edges, kCCBins.chunk), kCCBins, ctr, status);
  ECL_LAUNCH_NEXT(cc_chunks, grid, kTPB, 0, stream, nodes, nindex, nlist, label, chunks,
             chunk_capacity(edges, kCCBins.chunk), kCCBins.chunk, ctr, status);
  ECL_LAUNCH_NEXT(cc_flatten<kPlain>, flatten_blocks(dev, nodes), kTPB, 0, stream, nodes, label, Giants{}, nullptr, nullptr);
  Status hs{};
  ECL_CUDA_TRY(cudaMemcpyAsync(&hs, status, sizeof(hs), cudaMemcpyDeviceToHost, stream));
  ECL_CUDA_TRY(cudaStreamSynchronize(stream));
  ECL_CUDA_TRY(cudaGetLastError());
  return static_cast<ecl_status>(hs.code);
}

extern "C" ecl_status ecl_compute_cc(int32_t nodes, int32_t edges, const int32_t* nidx, const int32_t* nlist,
                                     int32_t* nstat) {
  ecl_graph_view g{nodes, edges, nidx, nlist, nullptr, ECL_HOST, 0};
  ecl_opts o{};
  return ecl_cc(&g, nstat, &o);
}
