// Entry-balanced CSR scans: every warp takes tiles of 256 consecutive entries
// of nlist, whatever rows they belong to, and finds each entry's row from the
// row that holds the tile's first entry (flat_rows, one small pass over
// nindex) and the row starts inside the tile.
//
// Why not rows per lane, warp or chunk record: a power-law graph's rows differ
// by five orders of magnitude, so a scan dealt by rows needs three paths and a
// second launch for the records, reads short rows with 4 of 32 bytes of each
// sector per load, and a small graph's few long rows run one after another on
// a few warps.  Dealt by entries, all loads of nlist are whole 32-byte sectors
// (two 16-byte loads a lane where the array is aligned) and all warps have the
// same work.  The price is about 100 instructions a tile to find the rows.
#pragma once

#include "common.cuh"
#include "ecl_b200.h"

namespace ecl {
namespace dev {

constexpr int kFlatTile = 256;                  // entries per warp and tile
constexpr int kFlatLane = kFlatTile / 32;       // consecutive entries per lane
constexpr int kFlatRowsMax = 2048;              // rows of a tile looked at one by one; more: binary search

__host__ __device__ constexpr int flat_tiles(int m) { return m / kFlatTile + (m % kFlatTile != 0); }

struct FlatCsr {
  int n, m;
  const int* nindex;
  const int* nlist;
  const int* tilerow;  // [flat_tiles(m)] row of each tile's first entry, -1: none (filled by flat_rows)
};

// tilerow[t] = v for every tile t whose first entry lies in row v (the others
// keep -1: the array is preset).  Malformed rows raise ECL_ERR_BAD_GRAPH and
// own no tile.  A row of many tiles is spread over its warp.
__device__ __forceinline__ void flat_rows_range(int n, int m, const int* nindex, int* tilerow, int first, int stride,
                                                Status* status) {
  const int lane = threadIdx.x & 31;
  for (int base = first; base < n; base += stride) {  // `first` is a multiple of 32 per warp
    const int v = base + lane;
    int t0 = 0, t1 = 0;  // tiles whose first entry is in v's row
    if (v < n) {
      const int beg = __ldg(&nindex[v]), end = __ldg(&nindex[v + 1]);
      if (beg < 0 || end < beg || end > m) {
        raise(status, ECL_ERR_BAD_GRAPH, v);
      } else if (end > beg) {
        t0 = beg / kFlatTile + (beg % kFlatTile != 0);
        t1 = (end - 1) / kFlatTile + 1;
      }
    }
    const bool many = t1 - t0 > 32;
    if (!many)
      for (int t = t0; t < t1; t++) tilerow[t] = v;  // race-free: a tile has one row, no reader in this launch
    unsigned todo = __ballot_sync(kFull, many);
    while (todo) {
      const int who = __ffs(todo) - 1;
      todo &= todo - 1;
      const int wv = __shfl_sync(kFull, v, who), w0 = __shfl_sync(kFull, t0, who), w1 = __shfl_sync(kFull, t1, who);
      for (int t = w0 + lane; t < w1; t += 32) tilerow[t] = wv;  // race-free: as above
    }
  }
}

// One tile: f(e0, row, u) with e0 the lane's first entry and, for its
// kFlatLane entries, the row (-1: the entry is in no row, or past the end) and
// the entry's value nlist[e0 + k] (0 where the row is -1).  s_mark: this
// warp's kFlatTile words of shared memory.  All lanes call, and all call f.
// `stop` = min(m, nindex[n]), the end of the last row.
template <class F>
__device__ __forceinline__ void flat_tile(const FlatCsr& g, int stop, bool vec, int t, int* s_mark, F&& f) {
  const int lane = threadIdx.x & 31;
  const int first = t * kFlatTile;
  const int e0 = first + min(lane * kFlatLane, g.m - first);  // at most m, which may be near 2^31
  int u[kFlatLane];
  if (vec && e0 <= g.m - kFlatLane) {
    const int4 a = __ldcs(reinterpret_cast<const int4*>(g.nlist + e0));
    const int4 b = __ldcs(reinterpret_cast<const int4*>(g.nlist + e0 + 4));
    u[0] = a.x, u[1] = a.y, u[2] = a.z, u[3] = a.w, u[4] = b.x, u[5] = b.y, u[6] = b.z, u[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < kFlatLane; k++) u[k] = e0 < g.m - k ? __ldcs(&g.nlist[e0 + k]) : 0;
  }
  const int v0 = g.tilerow[t];  // (not by __ldg: an earlier launch wrote it)
  int v1 = first < g.m - kFlatTile ? g.tilerow[t + 1] : -1;
  if (v1 < 0 || v1 >= g.n) v1 = g.n - 1;
  int row[kFlatLane];
  if (v1 - v0 <= kFlatRowsMax) {
    int4* m4 = reinterpret_cast<int4*>(s_mark + lane * kFlatLane);
    m4[0] = m4[1] = make_int4(-1, -1, -1, -1);
    __syncwarp();
    for (int v = v0 + 1 + lane; v <= v1; v += 32) {
      const int beg = __ldg(&g.nindex[v]), end = __ldg(&g.nindex[v + 1]);
      if (end > beg && beg >= first && beg - first < kFlatTile) s_mark[beg - first] = v;
    }
    __syncwarp();
    const int4 a = m4[0], b = m4[1];
    row[0] = a.x, row[1] = a.y, row[2] = a.z, row[3] = a.w, row[4] = b.x, row[5] = b.y, row[6] = b.z, row[7] = b.w;
    __syncwarp();  // read before the next tile clears it
#pragma unroll
    for (int k = 1; k < kFlatLane; k++)
      if (row[k] < 0) row[k] = row[k - 1];
    int carry = row[kFlatLane - 1];  // last row start in this lane or before it (rows ascend)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(kFull, carry, o);
      if (lane >= o) carry = max(carry, x);
    }
    carry = __shfl_up_sync(kFull, carry, 1);
    carry = lane == 0 ? v0 : max(carry, v0);
#pragma unroll
    for (int k = 0; k < kFlatLane; k++)
      if (row[k] < 0) row[k] = carry;
  } else {
    // a long run of empty rows: the last row that starts at or before the entry
#pragma unroll
    for (int k = 0; k < kFlatLane; k++) {
      int lo = v0, hi = v1;
      while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (__ldg(&g.nindex[mid]) <= e0 + k)
          lo = mid;
        else
          hi = mid - 1;
      }
      row[k] = lo;
    }
  }
  if (v0 < 0) {  // entries before the first row are no part of the graph
#pragma unroll
    for (int k = 0; k < kFlatLane; k++)
      if (row[k] < 0) u[k] = 0;
  }
#pragma unroll
  for (int k = 0; k < kFlatLane; k++)
    if (e0 >= stop - k) {
      row[k] = -1;
      u[k] = 0;
    }
  f(e0, row, u);
}

}  // namespace dev
}  // namespace ecl
