// Maximal independent set (ECL-MIS contract).
//
// Result contract (src/racefree/egr-input/MIS/ECL-MIS-atomic.cu): every
// vertex has a fixed priority byte (:118-136); findmins (:72-104) lets an
// undecided vertex join once every undecided neighbour has a lower
// (byte, id) and none is in.  With fixed priorities the set this converges to
// is the sequential greedy MIS in descending (byte, id) order, independent of
// the schedule, so the set below is bit-identical.
//
// B200 design:
//  * status bytes packed four per 32-bit word in the workspace (4.2 MB at
//    R-MAT-22, resident in the 126 MB L2); every shared access is a
//    device-scope relaxed atomic on the word;
//  * mis_init computes the priority bytes with the reference's fp32 formula
//    using explicit round-to-nearest intrinsics (no contraction);
//  * mis_run is ONE persistent cooperative launch (all blocks co-resident).
//    A first sweep scans every vertex's list up to the first blocker (an
//    undecided neighbour that outranks it); vertices that have to wait become
//    items {vertex, blocker's place in the list, blocker, list end} in a list of
//    their warp's own, and later sweeps look at two status words per item --
//    the vertex's and its blocker's -- until one is decided, then scan on from
//    the blocker.  No entry is scanned twice: one that was passed is out, or
//    outranked and cannot join before the vertex is decided.  Lists of <= 16
//    entries are scanned by their own lane; longer ones, from the second sweep
//    on, 128 entries per step by the whole warp (up to 32 entries by their lanes
//    too, where many of the warp have as many); a joining vertex claims itself with one CAS, then clears
//    its neighbours' bytes (fetch_and);
//  * a self-loop (the reference spins forever on one: v never outranks
//    itself) raises ECL_ERR_BAD_GRAPH when it is met; a sweep cap turns any
//    other non-converging input into ECL_ERR_NO_CONVERGENCE.
#include <algorithm>

#include "solvers.cuh"

namespace ecl {
namespace {

using namespace dev;

constexpr int kTPB = 256;
// Lists of up to this many entries are scanned by their own lane, in the first
// sweep; longer ones wait for the second (a launch knob).  R-MAT-22, mis_run,
// 32 / 16 / 8: 350 / 297 / 352 us; G(3 M, 24 M): 279 / 287 / 488.
constexpr int kLaneMax = 16;
// Lanes of a warp with lists of 17 to 32 entries from which on they scan them
// themselves.  Never / 4 / 8 / always: 20 k vertices in a row with 20 leaves each
// 46 / 32 / 33 / 32 us, G(3 M, 36 M) 439 / 371 / 367 / 377, R-MAT-22 320 / 331 /
// 323 / 341.
constexpr int kManyMid = 8;
// Vertices of a warp's group: 32, and down to kSmallGroup where the lists have
// more than kDenseRow entries on average and groups of 32 would leave warps of
// the device without any, as a group's lists, a dozen steps of the whole warp
// each, run one after another.  32 -> this: a complete bipartite graph of 2 x 1500
// vertices 575 -> 119 us (whole solve), a clique of 1200 326 -> 93, 30 cliques of
// 300 135 -> 69; with lists of 100 entries, 100 k of them, 156 -> 167.
constexpr int kSmallGroup = 4;
constexpr int kDenseRow = 128;
constexpr int kBatch = 4;  // list entries per lane whose loads are issued together
constexpr unsigned kIn = 0xfe;

__device__ __forceinline__ unsigned byte_of(unsigned word, int v) { return (word >> ((v & 3) * 8)) & 0xffu; }

__device__ __forceinline__ unsigned mis_priority(int v, int degree, float avg, float scaledavg) {
  if (degree <= 0) return kIn;
  // x = degree - hash(v) * 2^-32 ; res = rint(scaledavg / (avg + x))
  const float h = __fmul_rn(__uint2float_rn(ecl_hash((unsigned)v)), 0.00000000023283064365386962890625f);
  const float x = __fsub_rn(__int2float_rn(degree), h);
  const int res = __float2int_rn(__fdiv_rn(scaledavg, __fadd_rn(avg, x)));
  return (unsigned)((res + res) | 1) & 0xffu;
}

// For a union of graphs (vbase != nullptr) every vertex uses ITS graph's
// average degree and its local id, so each graph's bytes are exactly the ones
// a solve of that graph alone computes.
__global__ void __launch_bounds__(kTPB) mis_init(int n, int m, const int* __restrict__ nindex,
                                                 unsigned* __restrict__ st4, int nwords, const int* __restrict__ vbase,
                                                 const float* __restrict__ avgs, int ngraphs,
                                                 Status* __restrict__ status) {
  dep_wait();
  const float avg1 = __fdiv_rn(__int2float_rn(m), __int2float_rn(n));
  for (int w = blockIdx.x * kTPB + threadIdx.x; w < nwords; w += gridDim.x * kTPB) {
    unsigned word = 0;
    for (int k = 0; k < 4; k++) {
      const int v = 4 * w + k;
      unsigned b = 0;  // padding vertices are OUT
      if (v < n) {
        const int beg = __ldg(&nindex[v]), end = __ldg(&nindex[v + 1]);
        if (beg < 0 || end < beg || end > m) raise(status, ECL_ERR_BAD_GRAPH, v);
        float avg = avg1;
        int local = v;
        if (vbase) {
          const int g = union_graph_of(vbase, ngraphs, v);
          avg = __ldg(&avgs[g]);
          local = v - __ldg(&vbase[g]);
        }
        b = mis_priority(local, end - beg, avg, __fmul_rn(126.0f, avg));
      }
      word |= b << (8 * k);
    }
    st4[w] = word;  // race-free: thread-owned init, no reader in this launch
  }
}

// Outcome of scanning v's list.
enum : int { kWait = 0, kJoin = 1, kOut = 2 };

// Per-neighbour verdict: IN neighbour -> v is out; undecided neighbour with
// a higher (byte, id) -> v must wait; else no constraint.
__device__ __forceinline__ int mis_verdict(unsigned sb, unsigned b, int u, int v) {
  if (sb == kIn) return kOut;
  if ((sb & 1u) && (sb > b || (sb == b && u > v))) return kWait;
  return kJoin;
}

// Claims v as IN if its byte is still the undecided value b.
__device__ __forceinline__ bool mis_claim(unsigned* st4, int v, unsigned b) {
  unsigned* word = &st4[v >> 2];
  const int sh = (v & 3) * 8;
  unsigned cur = ld(word);
  while (byte_of(cur, v) == b) {
    const unsigned want = (cur & ~(0xffu << sh)) | (kIn << sh);
    const unsigned seen = cas(word, cur, want);
    if (seen == cur) return true;
    cur = seen;
  }
  return false;
}

__device__ __forceinline__ void mis_set_out(unsigned* st4, int u) { fetch_and(&st4[u >> 2], ~(0xffu << ((u & 3) * 8))); }

// A joined vertex sets its list entries nlist[i], i = i0, i0 + step, ...
// below end, out.  Their status words are read first (kBatch at a time) and
// only the entries not out yet take the atomic: a low-degree vertex that
// joins mostly neighbours hubs, whose words would otherwise take one atomic
// per joining neighbour.
__device__ __forceinline__ void mis_clear_list(unsigned* st4, const int* nlist, int i0, int end, int step, int n) {
  for (; i0 < end; i0 += step * kBatch) {
    int u[kBatch];
    unsigned w[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      const int i = i0 + k * step;
      u[k] = i < end ? __ldg(&nlist[i]) : -1;
    }
#pragma unroll
    for (int k = 0; k < kBatch; k++) w[k] = (unsigned)u[k] < (unsigned)n ? ld(&st4[u[k] >> 2]) : 0u;
#pragma unroll
    for (int k = 0; k < kBatch; k++)
      if ((unsigned)u[k] < (unsigned)n && byte_of(w[k], u[k]) != 0) mis_set_out(st4, u[k]);
  }
}

// Scans entries [pos, end) of v (byte b) by its own lane; stops at the first
// verdict other than kJoin and leaves pos and *blocker there.
__device__ __forceinline__ int mis_scan_lane(int v, unsigned b, int& pos, int end, int n, const int* nlist,
                                             unsigned* st4, int* blocker, Status* status) {
  for (; pos < end; pos += kBatch) {
    int u[kBatch];
    unsigned w[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) u[k] = pos + k < end ? __ldg(&nlist[pos + k]) : -1;
#pragma unroll
    for (int k = 0; k < kBatch; k++) w[k] = (unsigned)u[k] < (unsigned)n ? ld(&st4[u[k] >> 2]) : 0u;
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      if (pos + k >= end) break;
      if ((unsigned)u[k] >= (unsigned)n || u[k] == v) {  // out of range, or a self-loop
        raise(status, ECL_ERR_BAD_GRAPH, u[k]);
        continue;
      }
      const int r = mis_verdict(byte_of(w[k], u[k]), b, u[k], v);
      if (r != kJoin) {
        pos += k;
        *blocker = u[k];
        return r;
      }
    }
  }
  return kJoin;
}

// The same by the whole warp, 128 entries a step; the arguments are
// warp-uniform and all lanes call.  An IN neighbour of the step decides before
// an undecided one does.
__device__ __forceinline__ int mis_scan_warp(int v, unsigned b, int& pos, int end, int n, const int* nlist,
                                             unsigned* st4, int* blocker, Status* status) {
  const int lane = threadIdx.x & 31;
  for (; pos < end; pos += 32 * kBatch) {
    int u[kBatch];
    unsigned w[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      const int i = pos + 32 * k + lane;
      u[k] = i < end ? __ldg(&nlist[i]) : -1;
    }
#pragma unroll
    for (int k = 0; k < kBatch; k++) w[k] = (unsigned)u[k] < (unsigned)n ? ld(&st4[u[k] >> 2]) : 0u;
    bool out = false;
    int who = -1;  // a blocker among this lane's entries
#pragma unroll
    for (int k = 0; k < kBatch; k++) {
      if (pos + 32 * k + lane >= end) continue;
      if ((unsigned)u[k] >= (unsigned)n || u[k] == v) {
        raise(status, ECL_ERR_BAD_GRAPH, u[k]);
        continue;
      }
      const int r = mis_verdict(byte_of(w[k], u[k]), b, u[k], v);
      out |= r == kOut;
      if (r == kWait) who = u[k];
    }
    if (__any_sync(kFull, out)) return kOut;
    const unsigned wait = __ballot_sync(kFull, who >= 0);
    if (wait) {  // pos stays: the step is looked at again once this blocker is decided
      *blocker = __shfl_sync(kFull, who, __ffs(wait) - 1);
      return kWait;
    }
  }
  return kJoin;
}

// Without items (kItems false: a workspace of one byte a vertex) every sweep
// goes through the groups again and scans from the start: R-MAT-22 330 -> 560 us.
//
// A warp's g-th group is the vertices group (g nwarps + warp) .. + group - 1 (group:
// a power of two, at most 32), and its g-th `group` items lie at the same places,
// so the warps' lists share one array of n (rounded up) items and need no
// counters.  Bound by the latency of the chains of decisions: DRAM and L2 are far
// from busy.  Measured, groups of 32 vertices swept and scanned from the start
// until decided -> items: R-MAT-22 525 -> 297 us, 500 k vertices 169 -> 80, 1000
// vertices (fewer blocks) 40 -> 16; with the long lists scanned in the first sweep
// as well, R-MAT-22 525.
template <bool kItems>
__global__ void __launch_bounds__(kTPB) mis_run(int n, int m, const int* __restrict__ nindex,
                                                const int* __restrict__ nlist, unsigned* __restrict__ st4,
                                                int4* __restrict__ items, Status* __restrict__ status, int max_sweeps,
                                                int lane_max, int group) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * kTPB + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * kTPB) >> 5;
  const int gshift = __ffs(group) - 1;
  int kept = 0;  // items of this warp's list
  auto slot = [&](int k) -> long long { return (((long long)(k >> gshift) * nwarps + warp) << gshift) + (k & (group - 1)); };
  // Scans on for the lanes with `go` (entries [pos, end) of v), carries the
  // verdicts out and keeps the waiting ones.  All lanes call.
  auto advance = [&](bool go, bool wait, int v, unsigned b, int pos, int end, int blocker) {
    int verdict = kWait;
    // a list of up to twice as many entries by the whole warp, or, where kManyMid
    // lanes of the warp have one, each by its own lane
    const bool mid = go && end - pos > lane_max && end - pos <= 2 * lane_max;
    const bool many = __popc(__ballot_sync(kFull, mid)) >= kManyMid;
    const bool big = go && end - pos > lane_max && !(mid && many);
    if (go && !big) {
      verdict = mis_scan_lane(v, b, pos, end, n, nlist, st4, &blocker, status);
    }
    unsigned todo = __ballot_sync(kFull, big);
    while (todo) {
      const int who = __ffs(todo) - 1;
      todo &= todo - 1;
      const int wv = __shfl_sync(kFull, v, who), wend = __shfl_sync(kFull, end, who);
      const unsigned wb = __shfl_sync(kFull, b, who);
      int wpos = __shfl_sync(kFull, pos, who), wblock = -1;
      const int r = mis_scan_warp(wv, wb, wpos, wend, n, nlist, st4, &wblock, status);
      if (lane == who) verdict = r, pos = wpos, blocker = wblock;
    }
    if (go && verdict == kOut) mis_set_out(st4, v);
    // joins: the claim first, then the neighbours
    bool joined = go && verdict == kJoin && mis_claim(st4, v, b);
    const int beg = joined ? __ldg(&nindex[v]) : 0;
    if (joined && end - beg <= lane_max) mis_clear_list(st4, nlist, beg, end, 1, n);
    unsigned clear = __ballot_sync(kFull, joined && end - beg > lane_max);
    while (clear) {
      const int who = __ffs(clear) - 1;
      clear &= clear - 1;
      mis_clear_list(st4, nlist, __shfl_sync(kFull, beg, who) + lane, __shfl_sync(kFull, end, who), 32, n);
    }
    const bool keep = wait || (go && verdict == kWait);
    const unsigned bal = __ballot_sync(kFull, keep);
    // race-free: the warp's own
    if (kItems && keep) items[slot(kept + __popc(bal & ((1u << lane) - 1)))] = make_int4(v, pos, blocker, end);
    kept += __popc(bal);
  };
  int sweep = 0;
  for (bool first = true;; first = false) {  // once; without items, until all are decided
    for (unsigned base = warp * group; base < (unsigned)n; base += nwarps * group) {
      const int v = lane < group ? (int)min(base + lane, (unsigned)n) : n;
      unsigned b = 0;
      if (v < n) b = byte_of(ld(&st4[v >> 2]), v);
      const bool und = (b & 1u) != 0;
      if (!__any_sync(kFull, und)) continue;
      int beg = 0, end = 0;
      if (und) {
        beg = __ldg(&nindex[v]);
        end = __ldg(&nindex[v + 1]);
        if (beg < 0 || end < beg || end > m) beg = end = 0;  // reported by mis_init
      }
      // long lists first wait for a sweep: their vertices rank low (the priority
      // falls with the degree), and most are out before they are looked at
      const bool big = (kItems || first) && end - beg > lane_max;
      advance(und && !big, und && big, v, b, beg, end, -1);
    }
    if (kItems || kept == 0) break;
    kept = 0;
    if (sweep >= max_sweeps) {
      if (lane == 0) raise(status, ECL_ERR_NO_CONVERGENCE, warp);
      break;
    }
    sweep++;
  }
  for (; kept > 0; sweep++) {
    if (sweep >= max_sweeps) {
      if (lane == 0) raise(status, ECL_ERR_NO_CONVERGENCE, warp);
      break;
    }
    const int count = kept;
    kept = 0;
    __syncwarp();
    for (int c = 0; c < count; c += 32) {
      const int4 it = c + lane < count ? items[slot(c + lane)] : make_int4(-1, 0, 0, 0);  // race-free: the warp's own
      __syncwarp();
      const unsigned sv = it.x >= 0 ? ld(&st4[it.x >> 2]) : 0u;
      const unsigned su = it.x >= 0 && it.z >= 0 ? ld(&st4[it.z >> 2]) : 0u;
      const unsigned b = it.x >= 0 ? byte_of(sv, it.x) : 0u;  // even: a neighbour joined, the vertex is out
      const unsigned bu = byte_of(su, it.z & 3);  // 0: out, or no blocker yet
      const bool und = (b & 1u) != 0, wait = und && (bu & 1u) != 0;
      advance(und && !wait, wait, it.x, b, it.y, it.w, it.z);
    }
  }
  if (lane == 0) fetch_max(&status->rounds, sweep + 1);
}

__global__ void __launch_bounds__(kTPB) mis_emit(int n, const unsigned* st4,
                                                 unsigned char* __restrict__ out) {
  dep_wait();
  for (int v = blockIdx.x * kTPB + threadIdx.x; v < n; v += gridDim.x * kTPB) {
    out[v] = (unsigned char)byte_of(st4[v >> 2], v);  // race-free: st4 is final (mis_run finished)
  }
}

void mis_layout(Carve& c, int n, unsigned** st4, int4** items) {
  *st4 = c.take<unsigned>((size_t)(n + 3) / 4);
  if (items) *items = c.take<int4>(((size_t)n + 31) / 32 * 32);
}

}  // namespace

size_t mis_workspace_bytes(int n, int m) {
  (void)m;
  Carve c;
  unsigned* st4;
  int4* items;
  mis_layout(c, n, &st4, &items);
  return c.bytes();
}

size_t mis_small_workspace_bytes(int n) {
  Carve c;
  unsigned* st4;
  mis_layout(c, n, &st4, nullptr);
  return c.bytes();
}

}  // namespace ecl

namespace ecl {

ecl_status mis_enqueue(const GraphDev& g, unsigned char* out, char* ws, size_t ws_bytes, Status* status,
                       const DeviceInfo& dev, cudaStream_t stream, int max_sweeps, const UnionInfo* uni, Marker mark) {
  Carve c{ws};
  unsigned* st4;
  int4* items = nullptr;
  mis_layout(c, g.n, &st4, ws_bytes >= mis_workspace_bytes(g.n, g.m) ? &items : nullptr);
  const int nwords = (g.n + 3) / 4;
  const int grid = dev.grid_blocks(kTPB, g.n, g.m);
  const int* vbase = uni ? uni->vbase : nullptr;
  const float* avgs = uni ? uni->avg : nullptr;
  const int ngraphs = uni ? uni->ngraphs : 0;
  ECL_LAUNCH_NEXT(mis_init, grid, kTPB, 0, stream, g.n, g.m, g.nindex, st4, nwords, vbase, avgs, ngraphs, status);
  mark();
  // Warps of mis_run wait (by sweeping) for vertices owned by other warps,
  // so all its blocks must be resident together: a cooperative launch
  // guarantees that even when other solves share the GPU (server slots).
  int occ = 0;
  auto run = items ? mis_run<true> : mis_run<false>;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, run, kTPB, 0) != cudaSuccess || occ < 1)
    return ECL_ERR_CUDA;
  const int full = dev.sms * std::min(occ, dev.max_threads_per_sm / kTPB);
  int group = 32;
  if (g.m / g.n > kDenseRow)  // kSmallGroup says why
    while (group > kSmallGroup && g.n / group < full * (kTPB / 32)) group /= 2;
  ECL_CUDA_TRY(launch_cooperative(run, std::min(full, (g.n - 1) / (group * (kTPB / 32)) + 1), kTPB, stream, g.n,
                                  g.m, g.nindex, g.nlist, st4, items, status, max_sweeps,
                                  bins_of(dev, Bins{kLaneMax, kBinChunk}).lane, group));
  mark();
  ECL_LAUNCH_NEXT(mis_emit, grid, kTPB, 0, stream, g.n, st4, out);
  mark();
  return ECL_OK;
}

}  // namespace ecl

extern "C" ecl_status ecl_mis(const ecl_graph_view* g, uint8_t* status_out, ecl_opts* opts) {
  using namespace ecl;
  ecl_opts local{};
  if (!opts) opts = &local;
  if (!status_out) return ECL_ERR_INVALID_ARG;
  Solve s(g, opts);
  GraphNeeds needs;
  needs.symmetric = true;
  needs.no_self_loops = true;
  ecl_status st = s.begin(needs, g ? mis_workspace_bytes(g->nodes, g->edges) : 0,
                          g ? mis_small_workspace_bytes(g->nodes) : 0);
  if (st != ECL_OK) return s.finish(st);
  unsigned char* out = s.output(status_out, (size_t)s.n);
  if (!out) return s.finish(ECL_ERR_OOM);
  GraphDev gd;
  gd.n = s.n;
  gd.m = s.m;
  gd.nindex = s.nindex;
  gd.nlist = s.nlist;
  gd.flags = g->flags;
  // Warps sweep asynchronously (one may sweep many times while it waits on a
  // slower warp's vertex), so the cap is a fixed backstop against inputs that
  // cannot converge, not a per-graph bound.
  const int max_sweeps = opts->max_rounds > 0 ? opts->max_rounds : (1 << 22);
  s.start_timer();
  st = mis_enqueue(gd, out, s.ws, s.ws_size - kStatusBytes, s.status, s.dev, s.stream, max_sweeps, nullptr, Marker{&s});
  s.stop_timer();
  return s.finish(st);
}

extern "C" ecl_status ecl_compute_mis(int32_t nodes, int32_t edges, const int32_t* nidx, const int32_t* nlist,
                                      uint8_t* nstat) {
  ecl_graph_view g{nodes, edges, nidx, nlist, nullptr, ECL_HOST, 0};
  ecl_opts o{};
  return ecl_mis(&g, nstat, &o);
}
