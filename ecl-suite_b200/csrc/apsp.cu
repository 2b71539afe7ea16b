// All-pairs shortest paths, blocked Floyd-Warshall (ECL-APSP contract).
//
// Result contract (src/racefree/grid-input/ECL-APSP-atomic.cu): the matrix
// starts as init1/init2 build it (:63-83) -- 0 on the diagonal of real
// vertices, INF = INT_MAX/2 elsewhere (padding included), then each list entry
// j of row i writes eweight[j] at (i, nlist[j]) in CSR order (last duplicate
// wins, a self-loop replaces the 0) -- and ends as the Floyd-Warshall closure
// FW_cpu computes (:533-570).  With non-negative weights every entry of that
// closure is min(INF, shortest-path length), which any correct blocked
// schedule reproduces exactly: int32 add+min, no rounding, and
// INF/2 + INF/2 < INT_MAX so no sum overflows.
//
// B200 design.  Min-plus is not a ring product, so the tensor cores cannot do
// it; the work is INT32-pipe bound (one DPX __viaddmin_s32 = min(a + b, c) per
// update) once enough tiles are in flight, and bound by the chain of diagonal
// closures when the matrix is small.  ONE persistent launch runs the whole
// blocked Floyd-Warshall as a list of tile items in a fixed order, claimed by
// the CTAs one after another; an item waits (bounded) on per-tile step
// counters until the tiles that it reads are ready.  Per k-block kb:
//  * panel items: the tiles of row kb and column kb, C = min(C, D (x) C) or
//    min(C, C (x) D) with D the closed diagonal tile -- the same code as
//  * update items: C(i, j) = min(C, A(i, kb) (x) A(kb, j)) for all others;
//  * the diagonal item, first in the list of updates: tile (kb+1, kb+1) is
//    updated and closed at once by one CTA, while the others work through the
//    rest of step kb, so no step of a large matrix waits for a closure.
// Every item's dependencies precede it in the list, so the CTA that holds the
// smallest unfinished item can always go on.  A tile that step kb reads as an
// operand is not rewritten by step kb + 1 before its readers are counted done.
// Large matrices use tiles of 128, an 8x8 register tile a thread, and stream
// both operands through two shared-memory stages of 32 k with cp.async (A
// rows padded by 4 words: conflict-free).  Small ones use tiles of 64, and one
// CTA (the spine) keeps the chain of diagonal tiles in its shared memory.
// Measured (compute phase; two launches per k-block and a closure in every
// panel CTA before): n = 8192 40.1 -> 36.0 ms, 84 % of the add-min rate
// ecl_minplus_peak measures; n = 1001 0.80 -> 0.29 ms.
#include <algorithm>

#include "runtime.cuh"

namespace ecl {
namespace {

using namespace dev;

constexpr int kThreads = 256;  // 16 x 16 threads, T/16 x T/16 cells each
constexpr int kKC = 32;        // k-chunk of a stage, and block of the closure
constexpr int kPadA = 4;
constexpr int kInf = 0x7fffffff / 2;

template <int T>
struct Apsp {
  static constexpr int R = T / 16;          // cells per thread and dimension
  static constexpr int kLdA = kKC + kPadA;  // A stage [T][kLdA]
  static constexpr int kStageWords = T * kLdA + kKC * T;
  static constexpr int kLdD = T + kPadA;  // closure tile [T][kLdD], over both stages
  // tiles of 64: one CTA keeps the chain of diagonal tiles in shared memory
  static constexpr bool kSpine = T == 64;
  static constexpr int kWords = kSpine && 3 * T * kLdD > 2 * kStageWords ? 3 * T * kLdD : 2 * kStageWords;
  static constexpr size_t kSmem = sizeof(int) * (size_t)kWords;
  static constexpr int kCtasPerSm = 2;
  static_assert(T * kLdD <= 2 * kStageWords, "the closure's tile lies over the stages");
};

// Row (column) of a thread's r-th cell row (column) within a tile.
template <int kHalf = 64>
__device__ __forceinline__ int cell(int t, int r) { return (r >> 2) * kHalf + t * 4 + (r & 3); }

// acc[r][c] = min(acc[r][c], min_k As[row_r][k] + Bs[k][col_c]), k in [0, K);
// kHalf is the distance of a thread's upper four rows from its lower four.
template <int R, int K, int RC = R, int kHalf = 64>
__device__ __forceinline__ void minplus_tile(const int* As, int lda, const int* Bs, int ldb, int (&acc)[R][RC], int ty,
                                             int tx) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    int a[R][4];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int4 t = *reinterpret_cast<const int4*>(&As[cell<kHalf>(ty, r) * lda + k]);
      a[r][0] = t.x, a[r][1] = t.y, a[r][2] = t.z, a[r][3] = t.w;
    }
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      int b[RC];
#pragma unroll
      for (int h = 0; h < RC; h += 4) {
        const int4 t = *reinterpret_cast<const int4*>(&Bs[(k + kk) * ldb + cell(tx, h)]);
        b[h] = t.x, b[h + 1] = t.y, b[h + 2] = t.z, b[h + 3] = t.w;
      }
#pragma unroll
      for (int r = 0; r < R; r++) {
#pragma unroll
        for (int c = 0; c < RC; c++) acc[r][c] = __viaddmin_s32(a[r][kk], b[c], acc[r][c]);
      }
    }
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Starts the copies of one stage: A[r0 .. r0+T)[k0 .. k0+32) and
// A[k0 .. k0+32)[c0 .. c0+T).
template <int T>
__device__ __forceinline__ void stage_load(const int* A, long ld, int r0, int c0, int k0, int* stage) {
  int* As = stage;
  int* Bs = stage + T * Apsp<T>::kLdA;
#pragma unroll
  for (int q = threadIdx.x; q < T * (kKC / 4); q += kThreads) {
    const int r = q / (kKC / 4), c = q % (kKC / 4) * 4;
    cp_async16(&As[r * Apsp<T>::kLdA + c], &A[(long)(r0 + r) * ld + k0 + c]);
  }
#pragma unroll
  for (int q = threadIdx.x; q < kKC * (T / 4); q += kThreads) {
    const int r = q / (T / 4), c = q % (T / 4) * 4;
    cp_async16(&Bs[r * T + c], &A[(long)(k0 + r) * ld + c0 + c]);
  }
  cp_async_commit();
}

template <int R, int RC = R, int kHalf = 64>
__device__ __forceinline__ void load_acc(const int* A, long ld, int row0, int col0, int (&acc)[R][RC], int ty, int tx) {
#pragma unroll
  for (int r = 0; r < R; r++) {
#pragma unroll
    for (int h = 0; h < RC; h += 4) {
      const int4 x = __ldcg(reinterpret_cast<const int4*>(A + (long)(row0 + cell<kHalf>(ty, r)) * ld + col0 + cell(tx, h)));
      acc[r][h] = x.x, acc[r][h + 1] = x.y, acc[r][h + 2] = x.z, acc[r][h + 3] = x.w;
    }
  }
}

// acc to the tile at (row0, col0) of a row-major matrix (global or shared).
template <int R, int RC = R, int kHalf = 64>
__device__ __forceinline__ void store_acc(int* A, long ld, int row0, int col0, const int (&acc)[R][RC], int ty, int tx) {
#pragma unroll
  for (int r = 0; r < R; r++) {
#pragma unroll
    for (int h = 0; h < RC; h += 4)
      *reinterpret_cast<int4*>(A + (long)(row0 + cell<kHalf>(ty, r)) * ld + col0 + cell(tx, h)) =
          make_int4(acc[r][h], acc[r][h + 1], acc[r][h + 2], acc[r][h + 3]);
  }
}

// Floyd-Warshall closure of the T x T tile in D (leading dimension T + 4), in
// 32-wide blocks.  All threads call; D is complete before and after a block
// barrier.  Bound by latency: the 32 steps of a diagonal block depend on each
// other.  A lane holds 8 x 4 cells of that block, so a step is 12 shuffles and
// 32 add-mins (a column a lane: 32 shuffles; a barrier per k over the whole
// tile, as first built, took 0.35 us a step).
template <int T>
__device__ __noinline__ void close_tile(int* D, int ty, int tx) {
  constexpr int ldd = Apsp<T>::kLdD, R = Apsp<T>::R, nbk = T / 32;
  constexpr int kUnits = 2 * (nbk - 1) * 4;  // quarters of the row's and the column's other blocks
  constexpr int kWarps = kThreads / 32, kPer = (kUnits + kWarps - 1) / kWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int kk = 0; kk < nbk; kk++) {
    int* Dk = D + kk * 32 * ldd + kk * 32;
    if (warp == 0) {  // lane = 8 rows (lane / 8) x 4 columns (lane % 8)
      const int ly = lane >> 3, lx = lane & 7;
      int d[8][4];
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int4 t = *reinterpret_cast<const int4*>(&Dk[(ly * 8 + r) * ldd + lx * 4]);
        d[r][0] = t.x, d[r][1] = t.y, d[r][2] = t.z, d[r][3] = t.w;
      }
#pragma unroll
      for (int k = 0; k < 32; k++) {
        int row[4], col[8];
#pragma unroll
        for (int c = 0; c < 4; c++) row[c] = __shfl_sync(kFull, d[k & 7][c], (k >> 3) * 8 + lx);
#pragma unroll
        for (int r = 0; r < 8; r++) col[r] = __shfl_sync(kFull, d[r][k & 3], ly * 8 + (k >> 2));
#pragma unroll
        for (int r = 0; r < 8; r++) {
#pragma unroll
          for (int c = 0; c < 4; c++) d[r][c] = __viaddmin_s32(col[r], row[c], d[r][c]);
        }
      }
#pragma unroll
      for (int r = 0; r < 8; r++)
        *reinterpret_cast<int4*>(&Dk[(ly * 8 + r) * ldd + lx * 4]) = make_int4(d[r][0], d[r][1], d[r][2], d[r][3]);
    }
    __syncthreads();
    // a unit: 8 of the 32 result rows (columns) of one block, a warp each;
    // all are computed before any is written back
    int y[kPer][8];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const int q = warp + u * kWarps;
      if (q >= kUnits) continue;
      const int o = q >> 3, b = o + (o >= kk), part = (q & 3) * 8;
      int x[32];
      if (q & 4) {  // column block (b, kk): lane = row, y[j] = min_k x[k] + Dk[k][j]
        const int* X = D + (b * 32 + lane) * ldd + kk * 32;
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
          const int4 t = *reinterpret_cast<const int4*>(&X[k]);
          x[k] = t.x, x[k + 1] = t.y, x[k + 2] = t.z, x[k + 3] = t.w;
        }
        {
          const int4 t0 = *reinterpret_cast<const int4*>(&X[part]), t1 = *reinterpret_cast<const int4*>(&X[part + 4]);
          y[u][0] = t0.x, y[u][1] = t0.y, y[u][2] = t0.z, y[u][3] = t0.w;
          y[u][4] = t1.x, y[u][5] = t1.y, y[u][6] = t1.z, y[u][7] = t1.w;
        }
#pragma unroll
        for (int k = 0; k < 32; k++) {
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            const int4 t = *reinterpret_cast<const int4*>(&Dk[k * ldd + part + j]);
            y[u][j] = __viaddmin_s32(x[k], t.x, y[u][j]);
            y[u][j + 1] = __viaddmin_s32(x[k], t.y, y[u][j + 1]);
            y[u][j + 2] = __viaddmin_s32(x[k], t.z, y[u][j + 2]);
            y[u][j + 3] = __viaddmin_s32(x[k], t.w, y[u][j + 3]);
          }
        }
      } else {  // row block (kk, b): lane = column, y[i] = min_k Dk[i][k] + x[k]
        const int* X = D + kk * 32 * ldd + b * 32 + lane;
#pragma unroll
        for (int k = 0; k < 32; k++) x[k] = X[k * ldd];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          int v = X[(part + i) * ldd];
#pragma unroll
          for (int k = 0; k < 32; k += 4) {
            const int4 t = *reinterpret_cast<const int4*>(&Dk[(part + i) * ldd + k]);
            v = __viaddmin_s32(t.x, x[k], v);
            v = __viaddmin_s32(t.y, x[k + 1], v);
            v = __viaddmin_s32(t.z, x[k + 2], v);
            v = __viaddmin_s32(t.w, x[k + 3], v);
          }
          y[u][i] = v;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const int q = warp + u * kWarps;
      if (q >= kUnits) continue;
      const int o = q >> 3, b = o + (o >= kk), part = (q & 3) * 8;
      if (q & 4) {
        int* X = D + (b * 32 + lane) * ldd + kk * 32 + part;
        *reinterpret_cast<int4*>(X) = make_int4(y[u][0], y[u][1], y[u][2], y[u][3]);
        *reinterpret_cast<int4*>(X + 4) = make_int4(y[u][4], y[u][5], y[u][6], y[u][7]);
      } else {
        int* X = D + (kk * 32 + part) * ldd + b * 32 + lane;
#pragma unroll
        for (int i = 0; i < 8; i++) X[i * ldd] = y[u][i];
      }
    }
    __syncthreads();
    if (T == 64) {  // the one other block: a row and four columns a thread
      const int o = 32 * (1 - kk), r = o + (threadIdx.x >> 3), c = o + (threadIdx.x & 7) * 4;
      int4 v = *reinterpret_cast<const int4*>(&D[r * ldd + c]);
#pragma unroll
      for (int k = 0; k < 32; k += 4) {
        const int4 a = *reinterpret_cast<const int4*>(&D[r * ldd + kk * 32 + k]);
        const int av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int4 t = *reinterpret_cast<const int4*>(&D[(kk * 32 + k + h) * ldd + c]);
          v.x = __viaddmin_s32(av[h], t.x, v.x);
          v.y = __viaddmin_s32(av[h], t.y, v.y);
          v.z = __viaddmin_s32(av[h], t.z, v.z);
          v.w = __viaddmin_s32(av[h], t.w, v.w);
        }
      }
      *reinterpret_cast<int4*>(&D[r * ldd + c]) = v;
    } else {
      // the other blocks: every thread its cells of the tile, those of the
      // finished row and column blocks left as they are
      int acc[R][R];
#pragma unroll
      for (int r = 0; r < R; r++) {
#pragma unroll
        for (int h = 0; h < R; h += 4) {
          const int4 t = *reinterpret_cast<const int4*>(&D[cell(ty, r) * ldd + cell(tx, h)]);
          acc[r][h] = t.x, acc[r][h + 1] = t.y, acc[r][h + 2] = t.z, acc[r][h + 3] = t.w;
        }
      }
      minplus_tile<R, 32>(D + kk * 32, ldd, D + kk * 32 * ldd, ldd, acc, ty, tx);
#pragma unroll
      for (int r = 0; r < R; r++) {
#pragma unroll
        for (int h = 0; h < R; h += 4) {
          if ((cell(ty, r) >> 5) != kk && (cell(tx, h) >> 5) != kk)
            *reinterpret_cast<int4*>(&D[cell(ty, r) * ldd + cell(tx, h)]) =
                make_int4(acc[r][h], acc[r][h + 1], acc[r][h + 2], acc[r][h + 3]);
        }
      }
    }
    __syncthreads();
  }
}

// Progress of the item list, in the workspace (zeroed before the launch).
struct ApspCtl {
  int* next;     // items claimed
  int* ver;      // [nb * nb] steps tile (i, j) has behind it
  int* rowdone;  // [step * nb + i] update items of row i finished in that step
  int* coldone;  // [step * nb + j] ... of column j
  int* panels;   // [step] panel items finished
};
__host__ __device__ inline size_t apsp_ctl_words(int nb) { return 64 + 3 * (size_t)nb * nb + nb; }

constexpr unsigned long long kWaitNs = 4000000000ull;  // a wait this long means a lost item

// Bounded wait until *p >= want; false when it gave up or an error is raised.
__device__ __forceinline__ bool apsp_wait(const int* p, int want, Status* status) {
  if (ld_acquire(p) >= want) return true;
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (unsigned spins = 1;; spins++) {
    if (ld_acquire(p) >= want) return true;
    if ((spins & 255u) == 0) {
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t - t0 > kWaitNs) {
        raise(status, ECL_ERR_NO_CONVERGENCE, want);
        return false;
      }
      if (ld(&status->code) == ECL_ERR_NO_CONVERGENCE) return false;
    }
  }
}

// One item of the list: tile (i, j) in step kb (-1: tile (0, 0), which is
// closed before any step), and whether it is a panel tile or is closed after
// its update.
struct ApspItem {
  int i, j, kb;
  bool panel, close;
};

__device__ __forceinline__ ApspItem apsp_item(int q, int nb) {
  ApspItem t{0, 0, -1, false, true};
  if (q == 0) return t;
  const int nm1 = nb - 1, per = 2 * nm1 + nm1 * nm1;
  t.kb = (q - 1) / per;
  int o = (q - 1) % per, ti, tj;
  t.panel = o < 2 * nm1;
  t.close = false;
  if (t.panel) {
    const int x = (t.kb + 1 + (o >> 1)) % nb;
    t.i = (o & 1) ? x : t.kb;
    t.j = (o & 1) ? t.kb : x;
    return t;
  }
  o -= 2 * nm1;
  t.close = o == 0 && t.kb + 1 < nb;
  if (o < nm1) {
    ti = 0, tj = o;
  } else if (o < 2 * nm1 - 1) {
    ti = o - nm1 + 1, tj = 0;
  } else {
    o -= 2 * nm1 - 1;
    ti = 1 + o / (nm1 - 1), tj = 1 + o % (nm1 - 1);
  }
  t.i = (t.kb + 1 + ti) % nb;
  t.j = (t.kb + 1 + tj) % nb;
  return t;
}

// Condition `c` (0..6, a lane each) of an item: *p >= want before it may run;
// nullptr: no such condition.
__device__ __forceinline__ const int* apsp_need(const ApspCtl& ctl, const ApspItem& t, int nb, int c, int* want) {
  const int i = t.i, j = t.j, kb = t.kb, nm1 = nb - 1;
  if (kb < 0) return nullptr;
  switch (c) {
    case 0: *want = kb; return &ctl.ver[(size_t)i * nb + j];
    case 1: *want = j == kb ? kb : kb + 1; return &ctl.ver[(size_t)i * nb + kb];  // a column panel reads itself
    case 2: *want = i == kb ? kb : kb + 1; return &ctl.ver[(size_t)kb * nb + j];  // a row panel reads itself
    case 3: *want = kb + 1; return &ctl.ver[(size_t)kb * nb + kb];
    // tiles that the last step read as operands: their readers are done
    case 4: *want = nm1; return kb > 0 && j == kb - 1 && i != kb - 1 ? &ctl.rowdone[(size_t)(kb - 1) * nb + i] : nullptr;
    case 5: *want = nm1; return kb > 0 && i == kb - 1 && j != kb - 1 ? &ctl.coldone[(size_t)(kb - 1) * nb + j] : nullptr;
    case 6: *want = 2 * nm1; return kb > 0 && i == kb - 1 && j == kb - 1 ? &ctl.panels[kb - 1] : nullptr;
  }
  return nullptr;
}

// Publishes that tile (i, j) has `steps` steps behind it, and counts it as a
// panel or update item of step kb (kb < 0: neither).  One warp calls, after a
// block barrier behind the tile's last store: one fence for all three words
// (a release store and two release adds, one after another, took 2 us).
__device__ __forceinline__ void apsp_publish(const ApspCtl& ctl, int nb, int i, int j, int steps, int kb, bool panel) {
  const int lane = threadIdx.x & 31;
  __threadfence();
  if (lane == 0) st(&ctl.ver[(size_t)i * nb + j], steps);
  if (kb < 0) return;
  if (panel) {
    if (lane == 1) fetch_add(&ctl.panels[kb], 1);
  } else {
    if (lane == 1) fetch_add(&ctl.rowdone[(size_t)kb * nb + i], 1);
    if (lane == 2) fetch_add(&ctl.coldone[(size_t)kb * nb + j], 1);
  }
}

template <int T>
__device__ __forceinline__ void tile_load(const int* A, long ld, int row0, int col0, int* S) {
#pragma unroll
  for (int q = threadIdx.x; q < T * (T / 4); q += kThreads)
    cp_async16(&S[q / (T / 4) * Apsp<T>::kLdD + q % (T / 4) * 4], &A[(long)(row0 + q / (T / 4)) * ld + col0 + q % (T / 4) * 4]);
}
template <int T>
__device__ __forceinline__ void tile_store(int* A, long ld, int row0, int col0, const int* S) {
#pragma unroll
  for (int q = threadIdx.x; q < T * (T / 4); q += kThreads)
    *reinterpret_cast<int4*>(&A[(long)(row0 + q / (T / 4)) * ld + col0 + q % (T / 4) * 4]) =
        *reinterpret_cast<const int4*>(&S[q / (T / 4) * Apsp<T>::kLdD + q % (T / 4) * 4]);
}

// Tiles of 64: the CTA's two halves (8 x 16 threads, 8 x 4 cells each) take
// half of k each of C = min(C, SA (x) SB), and the lower half merges.  Fewer
// shared-memory reads per add-min than 4 x 4 cells over all of k.  `own` holds
// C in the lower half and receives the result there; SX (a whole tile, read by
// nobody any more when merge() is called) passes the upper half's part.
template <int T>
struct SplitK {
  static_assert(T == 64, "two halves of 8 x 16 threads with 8 x 4 cells each");
  static constexpr int ldd = Apsp<T>::kLdD;
  int half = threadIdx.x >> 7, ty = (threadIdx.x & 127) >> 4, tx = threadIdx.x & 15;

  __device__ __forceinline__ void load_smem(const int* S, int (&x)[8][4]) const {
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int4 t = *reinterpret_cast<const int4*>(&S[cell<32>(ty, r) * ldd + cell(tx, 0)]);
      x[r][0] = t.x, x[r][1] = t.y, x[r][2] = t.z, x[r][3] = t.w;
    }
  }
  __device__ __forceinline__ void product(const int* SA, const int* SB, int (&own)[8][4]) const {
    if (half) {
#pragma unroll
      for (int r = 0; r < 8; r++) own[r][0] = own[r][1] = own[r][2] = own[r][3] = 0x7fffffff;
    }
    minplus_tile<8, T / 2, 4, 32>(SA + half * (T / 2), ldd, SB + half * (T / 2) * ldd, ldd, own, ty, tx);
  }
  __device__ __forceinline__ void merge(int* SX, int (&own)[8][4]) const {
    if (half) store_acc<8, 4, 32>(SX, ldd, 0, 0, own, ty, tx);
    __syncthreads();
    if (!half) {
      int x[8][4];
      load_smem(SX, x);
#pragma unroll
      for (int r = 0; r < 8; r++) {
#pragma unroll
        for (int c = 0; c < 4; c++) own[r][c] = min(own[r][c], x[r][c]);
      }
    }
  }
};

// The spine of a small matrix, run by one CTA: per step, close the diagonal
// tile, update the next step's two neighbours of it (panel tiles (kb, kb+1)
// and (kb+1, kb)) and the next diagonal tile, all from shared memory.  The
// chain of closures is what bounds a small matrix; as three items of the list,
// each hop of it cost a store, a flag and a load through L2 (n = 1001, per
// step of 64: 20 us as items, 17 us here: 6.8 the closure, 5.3 the two panel
// tiles, 3.2 the diagonal tile, 1.7 waiting for and loading the next tiles).
template <int T>
__device__ __forceinline__ void apsp_spine(int* A, long ld_a, int nb, const ApspCtl& ctl, int* smem, Status* status) {
  constexpr int ldd = Apsp<T>::kLdD;
  __shared__ int s_go;
  int* D = smem;
  int* P1 = D + T * ldd;   // tile (kb, kb + 1)
  int* P2 = P1 + T * ldd;  // tile (kb + 1, kb)
  const SplitK<T> sp;
  const int half = sp.half, ty = sp.ty, tx = sp.tx;
  tile_load<T>(A, ld_a, 0, 0, D);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  for (int kb = 0;; kb++) {
    close_tile<T>(D, threadIdx.x >> 4, tx);
    tile_store<T>(A, ld_a, kb * T, kb * T, D);
    __syncthreads();
    if (threadIdx.x < 32) apsp_publish(ctl, nb, kb, kb, kb + 1, kb - 1, false);  // as an update item of step kb - 1
    if (kb + 1 == nb) return;
    const int k1 = kb + 1;
    if (threadIdx.x >= 32 && threadIdx.x < 64) {  // another warp than the one that publishes
      const int lane = threadIdx.x & 31;
      const int* p = lane == 0 ? &ctl.ver[(size_t)kb * nb + k1]
                               : (lane == 1 ? &ctl.ver[(size_t)k1 * nb + kb] : &ctl.ver[(size_t)k1 * nb + k1]);
      const bool ok = __all_sync(kFull, lane > 2 || apsp_wait(p, kb, status));
      if (lane == 0) s_go = ok;
    }
    __syncthreads();
    if (!s_go) return;
    tile_load<T>(A, ld_a, kb * T, k1 * T, P1);
    tile_load<T>(A, ld_a, k1 * T, kb * T, P2);
    cp_async_commit();
    int acc[8][4], own[8][4];
    load_acc<8, 4, 32>(A, ld_a, k1 * T, k1 * T, own, ty, tx);
    cp_async_wait<0>();
    __syncthreads();
    int* P = half ? P2 : P1;
    sp.load_smem(P, acc);
    if (half)
      minplus_tile<8, T, 4, 32>(P2, ldd, D, ldd, acc, ty, tx);
    else
      minplus_tile<8, T, 4, 32>(D, ldd, P1, ldd, acc, ty, tx);
    __syncthreads();
    store_acc<8, 4, 32>(P, ldd, 0, 0, acc, ty, tx);
    store_acc<8, 4, 32>(A, ld_a, half ? k1 * T : kb * T, half ? kb * T : k1 * T, acc, ty, tx);
    __syncthreads();
    if (threadIdx.x < 32) apsp_publish(ctl, nb, kb, k1, kb + 1, kb, true);
    if (threadIdx.x >= 128 && threadIdx.x < 160) apsp_publish(ctl, nb, k1, kb, kb + 1, kb, true);
    // the next diagonal tile; the reads of D are behind the barriers above
    sp.product(P2, P1, own);
    sp.merge(D, own);
    if (!half) store_acc<8, 4, 32>(D, ldd, 0, 0, own, ty, tx);
    __syncthreads();
  }
}

template <int T>
__global__ void __launch_bounds__(kThreads, Apsp<T>::kCtasPerSm) apsp_run(int* __restrict__ A, long ld_a, int nb,
                                                                          ApspCtl ctl, Status* __restrict__ status) {
  constexpr int R = Apsp<T>::R;
  extern __shared__ __align__(16) int smem[];
  __shared__ int s_item[2], s_ok[2];
  if constexpr (Apsp<T>::kSpine) {
    if (blockIdx.x == 0) {
      apsp_spine<T>(A, ld_a, nb, ctl, smem, status);
      return;
    }
  }
  const int total = 1 + nb * (nb - 1) * (nb + 1);
  if (threadIdx.x == 0) s_item[0] = fetch_add(ctl.next, 1);
  __syncthreads();
  for (int turn = 0;; turn ^= 1) {
    const int q = s_item[turn];
    if (q >= total) return;
    const ApspItem it = apsp_item(q, nb);
    // the spine's own items: the diagonal tiles and their next neighbours
    const bool skip = Apsp<T>::kSpine && (it.close || (it.panel && it.kb + 1 < nb && (it.i == it.kb + 1 || it.j == it.kb + 1)));
    // claim the next item and wait for this one's tiles, a condition a lane
    if (threadIdx.x == 32) s_item[turn ^ 1] = fetch_add(ctl.next, 1);
    if (threadIdx.x < 32) {
      int want = 0;
      const int* p = skip ? nullptr : apsp_need(ctl, it, nb, threadIdx.x, &want);
      const bool all = __all_sync(kFull, p == nullptr || apsp_wait(p, want, status));
      if (threadIdx.x == 0) s_ok[turn] = all;
    }
    __syncthreads();
    if (!s_ok[turn]) return;
    if (skip) continue;
    const int r0 = it.i * T, c0 = it.j * T, k0 = it.kb * T;
    if constexpr (Apsp<T>::kSpine) {
      int* SB = smem + T * Apsp<T>::kLdD;
      const SplitK<T> sp;
      tile_load<T>(A, ld_a, r0, k0, smem);
      tile_load<T>(A, ld_a, k0, c0, SB);
      cp_async_commit();
      int own[8][4];
      if (!sp.half) load_acc<8, 4, 32>(A, ld_a, r0, c0, own, sp.ty, sp.tx);
      cp_async_wait<0>();
      __syncthreads();
      sp.product(smem, SB, own);
      __syncthreads();
      sp.merge(smem, own);
      if (!sp.half) store_acc<8, 4, 32>(A, ld_a, r0, c0, own, sp.ty, sp.tx);
    } else {
      const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
      int acc[R][R];
      if (it.kb >= 0) {
        stage_load<T>(A, ld_a, r0, c0, k0, smem);
        load_acc<R>(A, ld_a, r0, c0, acc, ty, tx);
#pragma unroll 1
        for (int kc = 0; kc < T / kKC; kc++) {
          if (kc + 1 < T / kKC) {
            stage_load<T>(A, ld_a, r0, c0, k0 + (kc + 1) * kKC, smem + ((kc + 1) & 1) * Apsp<T>::kStageWords);
            cp_async_wait<1>();
          } else {
            cp_async_wait<0>();
          }
          __syncthreads();
          const int* st = smem + (kc & 1) * Apsp<T>::kStageWords;
          minplus_tile<R, kKC>(st, Apsp<T>::kLdA, st + T * Apsp<T>::kLdA, T, acc, ty, tx);
          __syncthreads();
        }
      } else {
        load_acc<R>(A, ld_a, r0, c0, acc, ty, tx);
      }
      if (it.close) {
        store_acc<R>(smem, Apsp<T>::kLdD, 0, 0, acc, ty, tx);
        __syncthreads();
        close_tile<T>(smem, ty, tx);
        tile_store<T>(A, ld_a, r0, c0, smem);
      } else {
        store_acc<R>(A, ld_a, r0, c0, acc, ty, tx);
      }
    }
    __syncthreads();
    // the last warp publishes while the first goes on to the next item's wait;
    // a closed tile has step kb and its own step behind it
    if (threadIdx.x >= kThreads - 32) apsp_publish(ctl, nb, it.i, it.j, it.close ? it.kb + 2 : it.kb + 1, it.kb, it.panel);
  }
}

__global__ void apsp_fill(int* __restrict__ A, long ld, int N, int n) {
  dep_wait();
  const long total4 = (long)N * N / 4;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < total4; q += (long)gridDim.x * blockDim.x) {
    const long idx = q * 4;
    const int i = (int)(idx / N), j = (int)(idx % N);
    int4 v = make_int4(kInf, kInf, kInf, kInf);
    if (i < n && i >= j && i < j + 4) (&v.x)[i - j] = 0;
    *reinterpret_cast<int4*>(&A[(long)i * ld + j]) = v;
  }
}

// One thread per row writes the row's entries in CSR order, so the last
// duplicate wins exactly as in init2 (ECL-APSP-atomic.cu:74-83).
__global__ void apsp_edges(int* __restrict__ A, long ld, int n, int m, const int* __restrict__ nindex,
                           const int* __restrict__ nlist, const int* __restrict__ eweight, Status* __restrict__ status) {
  dep_wait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int beg = __ldg(&nindex[i]), end = __ldg(&nindex[i + 1]);
    if (beg < 0 || end < beg || end > m) {
      raise(status, ECL_ERR_BAD_GRAPH, i);
      continue;
    }
    for (int j = beg; j < end; j++) {
      const int u = __ldg(&nlist[j]);
      const int w = __ldg(&eweight[j]);
      if ((unsigned)u >= (unsigned)n || w < 0) {
        raise(status, ECL_ERR_BAD_GRAPH, j);
        continue;
      }
      A[(long)i * ld + u] = w;  // race-free: one thread writes a row, no reader in this launch
    }
  }
}

// Tile edge: 64 below kSmallN vertices, 128 from there on.  A small matrix is
// bound by its chain (close, panel, update per k-block), which smaller tiles
// shorten; a large one by the INT32 pipe, which the 8x8 register tiles of 128
// keep busier.  Measured, 64 against 128: n = 1001 0.29 / 0.67 ms, 2500 1.57 /
// 1.70, 3000 2.50 / 2.27, 8192 48.6 / 36.0.
constexpr int kSmallN = 2688;
// CTAs per SM: one while the chain bounds the solve -- a second one on the SM
// of the chain's CTA halves its speed -- else two, which hide each other's
// loads.  Measured, one against two: n = 1001 0.287 / 0.295 ms, 1500 0.53 /
// 0.46 (tiles of 64); n = 3000 2.27 / 2.87, 3300 2.98 / 3.05, 8192 40.6 / 36.0
// (tiles of 128; 4096, before the last changes: 5.48 / 5.05).
constexpr int kChainBlocks64 = 20, kChainBlocks128 = 26;

int apsp_tile(int n) { return n < kSmallN ? 64 : 128; }
int apsp_padded(int n) { return (n + apsp_tile(n) - 1) / apsp_tile(n) * apsp_tile(n); }

size_t apsp_ctl_bytes(int n) { return (apsp_ctl_words(apsp_padded(n) / apsp_tile(n)) * sizeof(int) + 255) / 256 * 256; }

template <int T>
ecl_status apsp_launch(int* A, int N, int* ctl_words, const DeviceInfo& dev, cudaStream_t stream, Status* status) {
  const int nb = N / T;
  ApspCtl ctl;
  ctl.next = ctl_words;
  ctl.ver = ctl_words + 64;
  ctl.rowdone = ctl.ver + (size_t)nb * nb;
  ctl.coldone = ctl.rowdone + (size_t)nb * nb;
  ctl.panels = ctl.coldone + (size_t)nb * nb;
  ECL_CUDA_TRY(cudaMemsetAsync(ctl_words, 0, apsp_ctl_words(nb) * sizeof(int), stream));
  ECL_CUDA_TRY(cudaFuncSetAttribute(apsp_run<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Apsp<T>::kSmem));
  const long long items = 1 + (long long)nb * (nb - 1) * (nb + 1);
  const int per = nb <= (T == 64 ? kChainBlocks64 : kChainBlocks128) ? 1 : Apsp<T>::kCtasPerSm;
  const int grid = (int)std::min<long long>(items, (long long)dev.sms * per);
  if (Apsp<T>::kSpine) {  // the spine waits for CTAs that the list's order does not put before it: all are resident
    ECL_CUDA_TRY(launch_cooperative_smem(apsp_run<T>, grid, kThreads, Apsp<T>::kSmem, stream, A, (long)N, nb, ctl, status));
  } else {
    ECL_LAUNCH(apsp_run<T>, grid, kThreads, Apsp<T>::kSmem, stream, A, (long)N, nb, ctl, status);
  }
  return ECL_OK;
}

}  // namespace

size_t apsp_workspace_bytes(int n, int m) {
  (void)m;
  const size_t N = (size_t)apsp_padded(n);
  return N * N * sizeof(int) + apsp_ctl_bytes(n);
}

}  // namespace ecl

extern "C" ecl_status ecl_apsp(const ecl_graph_view* g, int32_t* dist, int64_t ld, ecl_opts* opts) {
  using namespace ecl;
  ecl_opts local{};
  if (!opts) opts = &local;
  if (!dist || !g || ld < g->nodes) return ECL_ERR_INVALID_ARG;
  if (g->nodes > 46340 * 2) return ECL_ERR_UNSUPPORTED;  // N^2 int32 must stay addressable and < HBM
  Solve s(g, opts);
  GraphNeeds needs;
  needs.weights = true;
  const int N = apsp_padded(std::max(g->nodes, 1));
  // Work in place when the caller's device matrix already has the padded
  // shape (and its rows start on 16-byte boundaries, as the tiles' loads need).
  const bool inplace = g->location == ECL_DEVICE && N == g->nodes && ld == N && (reinterpret_cast<uintptr_t>(dist) & 15) == 0;
  const size_t cbytes = apsp_ctl_bytes(std::max(g->nodes, 1));
  ecl_status st = s.begin(needs, inplace ? cbytes : apsp_workspace_bytes(g->nodes, g->edges));
  if (st != ECL_OK) return s.finish(st);
  int* ctl = reinterpret_cast<int*>(s.ws);
  int* W = inplace ? dist : reinterpret_cast<int*>(s.ws + cbytes);
  const int grid = s.dev.sms * 4;

  s.start_timer();
  ECL_LAUNCH_NEXT(apsp_fill, grid, 256, 0, s.stream, W, (long)N, N, s.n);
  if (s.m > 0) ECL_LAUNCH_NEXT(apsp_edges, (s.n + 255) / 256, 256, 0, s.stream, W, (long)N, s.n, s.m, s.nindex, s.nlist, s.eweight, s.status);
  s.mark();
  st = apsp_tile(s.n) == 64 ? apsp_launch<64>(W, N, ctl, s.dev, s.stream, s.status)
                            : apsp_launch<128>(W, N, ctl, s.dev, s.stream, s.status);
  if (st != ECL_OK) return s.finish(st);
  s.mark();
  s.stop_timer();
  if (!inplace) {
    const cudaMemcpyKind kind = g->location == ECL_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    if (cudaMemcpy2DAsync(dist, (size_t)ld * sizeof(int), W, (size_t)N * sizeof(int), (size_t)s.n * sizeof(int),
                          (size_t)s.n, kind, s.stream) != cudaSuccess)
      return s.finish(ECL_ERR_CUDA);
  }
  return s.finish();
}

extern "C" ecl_status ecl_compute_apsp(int32_t nodes, int32_t edges, const int32_t* nidx, const int32_t* nlist,
                                       const int32_t* eweight, int32_t* adjmat) {
  if (nodes < 1 || !adjmat) return ECL_ERR_INVALID_ARG;
  const int64_t upper = ((int64_t)nodes + 63) / 64 * 64;  // the reference's padded layout
  ecl_graph_view g{nodes, edges, nidx, nlist, eweight, ECL_HOST, 0};
  ecl_opts o{};
  const ecl_status st = ecl_apsp(&g, adjmat, upper, &o);
  if (st != ECL_OK) return st;
  for (int64_t i = 0; i < upper; i++) {
    for (int64_t j = (i < nodes ? nodes : 0); j < upper; j++) adjmat[i * upper + j] = ECL_APSP_INF;
  }
  return ECL_OK;
}
