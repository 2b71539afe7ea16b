// Stable LSD radix sort in one cooperative launch: see radix_sort.cuh.
#include "radix_sort.cuh"

#include <algorithm>

namespace ecl {
namespace {

using namespace dev;

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = kRadixTile / kThreads;  // keys a lane holds per tile
constexpr int kDigits = 256;
constexpr int kQuarters = kThreads / kDigits;     // threads that share a digit
constexpr int kPerQuarter = kWarps / kQuarters;

__device__ __forceinline__ int digit_of(unsigned long long k, int shift) { return (int)(k >> shift) & 0xff; }

// Lanes of the warp that are `in` and hold the same 8-bit digit as this one.
__device__ __forceinline__ unsigned same_digit(int d, bool in) {
  unsigned m = __ballot_sync(kFull, in);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool one = (d >> b) & 1;
    const unsigned v = __ballot_sync(kFull, one);
    m &= one ? v : ~v;
  }
  return m;
}

// With h spread evenly and (nearly) without repeats, the passes need not look at
// all of it: the lowest two digits (one, of more than kSkipTwo keys) are left
// out, and at the end each key finds its place in its run of keys equal so far,
// of kSkipTwo / 65536 at most on average.  A pass costs 7 us and more, the end
// 5.  Measured (with a block per 4096 keys), all digits / one left out / two: 20 k keys 73 / - / 54 us, 723 k
// 96 / 87 / 77, 2 M of four degrees 227 / 203 / 215, R-MAT-22 (2.4 M keys) 336 /
// 305 / 266: beyond a million keys that can share one degree the runs get long.
constexpr int kSkipTwo = 1 << 20;

// Every block sorts its own contiguous share of the keys.  A pass: rank the
// share (a warp its 256 keys of a tile, 32 at a time), publish its digit
// counts, grid barrier, base of each digit = the smaller digits' totals + the
// earlier blocks' counts, write, second barrier.
// A share of one tile stays in registers from ranking to writing.  Bound by
// latency for small n (two barriers and three dependent memory rounds a pass),
// by the ranking and the scattered 12-byte writes for large (ranking by ballots
// instead of __match_any_sync: R-MAT-22 0.39 -> 0.35 ms).  Measured, whole
// sort, four launches a pass -> this, all digits: 1000 keys 136 -> 32 us, 150 k
// 197 -> 69, 723 k 224 -> 98, R-MAT-22 (2.4 M keys, seven passes) 382 -> 342.
// kShort: every share is at most a tile, and a warp takes only as many slices of
// it as there are for all warps.
template <bool kShort>
__global__ void __launch_bounds__(kThreads, 1) rs_sort(unsigned long long* k0, int* v0, unsigned long long* k1, int* v1,
                                                       int* __restrict__ order, int n_max,
                                                       const int* __restrict__ n_dev, const int* __restrict__ max_high,
                                                       unsigned* __restrict__ counts, bool spread, GridBarrier* bar, int* failed,
                                                       Status* __restrict__ status) {
  __shared__ unsigned s_base[kDigits];               // where the next tile's keys of each digit go
  __shared__ unsigned short s_warp[kWarps][kDigits];  // per-warp digit counts of a tile, then their prefix sums
  __shared__ unsigned s_part[kQuarters][kDigits];
  __shared__ unsigned s_sum[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1;
  const int dig = threadIdx.x & (kDigits - 1), quarter = threadIdx.x / kDigits;
  const int blocks = gridDim.x;
  const int n = max(0, min(ld(n_dev), n_max));
  const int high = ld(max_high);
  // digits of h that the passes leave to the end (see kSkipTwo)
  const int skip = !spread ? 0 : (n <= kSkipTwo ? 2 : 1);
  int passes = 5;
  while (passes < 8 && (high >> (8 * (passes - 4))) != 0) passes++;
  passes -= skip;
  const int share = ((n + blocks - 1) / blocks + 31) & ~31;
  const int beg = (int)min((long long)n, (long long)share * blockIdx.x), end = (int)min((long long)n, (long long)beg + share);
  const bool one = share <= kRadixTile;  // uniform over the grid
  const int per = kShort ? (share + kThreads - 1) / kThreads : kItems;  // slices of 32 keys a warp takes of a tile
  unsigned long long k[kItems];
  int v[kItems];
  unsigned rank[kItems];
  for (int p = 0; p < passes; p++) {
    const int shift = 8 * (p + skip);
    const bool last = p == passes - 1;
    const unsigned long long* kin = (p & 1) ? k1 : k0;
    const int* vin = (p & 1) ? v1 : v0;
    unsigned long long* kout = (p & 1) ? k0 : k1;
    int* vout = last && skip == 0 ? order : ((p & 1) ? v0 : v1);
    // Loads the tile at t0, ranks each key among its warp's keys of the same
    // digit, and leaves in s_warp[w][d] the tile's keys of digit d in earlier
    // warps; returns the tile's keys of digit `dig`.  All threads call.
    auto rank_tile = [&](int t0, bool values) -> unsigned {
      const int i0 = t0 + warp * per * 32 + lane;
#pragma unroll
      for (int j = 0; j < kItems; j++) {
        const int i = j < per ? i0 + 32 * j : end;
        k[j] = i < end ? kin[i] : 0ull;  // race-free: written before the last grid barrier
        if (values) v[j] = i < end ? vin[i] : 0;  // race-free: as above
      }
      for (int d = lane; d < kDigits / 2; d += 32) reinterpret_cast<unsigned*>(s_warp[warp])[d] = 0;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kItems; j++) {
        if (j >= per || i0 - lane + 32 * j >= end) break;  // the same for the whole warp
        const bool in = i0 + 32 * j < end;
        const int d = digit_of(k[j], shift);
        const unsigned same = same_digit(d, in);
        const unsigned seen = in ? s_warp[warp][d] : 0u;
        rank[j] = seen + __popc(same & lt);
        __syncwarp();
        if (in && lane == __ffs(same) - 1) s_warp[warp][d] = (unsigned short)(seen + __popc(same));
        __syncwarp();
      }
      __syncthreads();
      unsigned c[kPerQuarter], mine = 0;
#pragma unroll
      for (int w = 0; w < kPerQuarter; w++) {
        c[w] = s_warp[quarter * kPerQuarter + w][dig];
        mine += c[w];
      }
      s_part[quarter][dig] = mine;
      __syncthreads();
      unsigned run = 0, all = 0;
#pragma unroll
      for (int q = 0; q < kQuarters; q++) {
        if (q < quarter) run += s_part[q][dig];
        all += s_part[q][dig];
      }
#pragma unroll
      for (int w = 0; w < kPerQuarter; w++) {
        s_warp[quarter * kPerQuarter + w][dig] = (unsigned short)run;
        run += c[w];
      }
      __syncthreads();
      return all;
    };
    unsigned own = 0;
    for (int t0 = beg; t0 < end; t0 += kRadixTile) own += rank_tile(t0, one);
    unsigned before = 0, total = own;
    if (blocks > 1) {
      if (quarter == 0) st(&counts[blockIdx.x * kDigits + dig], own);
      if (!grid_sync<true>(bar, status)) {
        if (threadIdx.x == 0) st(failed, 1);
        return;
      }
      // every quarter adds up its share of the blocks' counts, all loads in flight
      unsigned t = 0, e = 0;
      for (int b0 = quarter; b0 < blocks; b0 += 16 * kQuarters) {
        unsigned c[16];
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int b = b0 + j * kQuarters;
          c[j] = b < blocks ? ld(&counts[b * kDigits + dig]) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 16; j++) {
          t += c[j];
          if (b0 + j * kQuarters < (int)blockIdx.x) e += c[j];
        }
      }
      __syncthreads();  // s_part: every thread is past rank_tile's reads
      s_part[quarter][dig] = t;
      if (quarter == 0) s_base[dig] = 0;
      __syncthreads();
      if (e) atomicAdd(&s_base[dig], e);  // shared memory
      total = s_part[0][dig] + s_part[1][dig] + s_part[2][dig] + s_part[3][dig];
      static_assert(kQuarters == 4, "the sum above");
      __syncthreads();
      before = s_base[dig];
    }
    unsigned incl = total;  // inclusive over the digits of this thread's warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    if (quarter == 0) {
      unsigned lower = incl - total;
      for (int w = 0; w < warp; w++) lower += s_sum[w];
      s_base[dig] = lower + before;
    }
    __syncthreads();
    for (int t0 = beg; t0 < end; t0 += kRadixTile) {
      unsigned tile = 0;
      if (!one) tile = rank_tile(t0, true);
      const int i0 = t0 + warp * per * 32 + lane;
#pragma unroll
      for (int j = 0; j < kItems; j++) {
        if (j >= per || i0 + 32 * j >= end) continue;
        const int d = digit_of(k[j], shift);
        const unsigned pos = s_base[d] + s_warp[warp][d] + rank[j];
        if (!last || skip > 0) kout[pos] = k[j];  // race-free: a place has one key, read behind the next grid barrier
        vout[pos] = v[j];  // race-free: as above
      }
      __syncthreads();
      if (!one && quarter == 0) s_base[dig] += tile;
      __syncthreads();
    }
    if ((!last || skip > 0) && !grid_sync<true>(bar, status)) {
      if (threadIdx.x == 0) st(failed, 1);
      return;
    }
  }
  if (skip == 0) return;
  // runs of keys equal in the sorted digits: each key to its place among them
  const unsigned long long* kin = (passes & 1) ? k1 : k0;
  const int* vin = (passes & 1) ? v1 : v0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += blocks * kThreads) {
    const unsigned long long key = kin[i];  // race-free: written before the last grid barrier
    int pos = i;
    for (int j = i - 1; j >= 0; j--) {
      const unsigned long long x = kin[j];  // race-free: as above
      if ((x ^ key) >> (8 * skip)) break;
      pos -= x > key;
    }
    for (int j = i + 1; j < n; j++) {
      const unsigned long long x = kin[j];  // race-free: as above
      if ((x ^ key) >> (8 * skip)) break;
      pos += x < key;
    }
    order[pos] = vin[i];  // race-free: a place has one key; vin as above
  }
}

}  // namespace

ecl_status radix_order(unsigned long long* k0, int* v0, unsigned long long* k1, int* v1, int* order, int n,
                       const int* n_dev, const int* max_high, unsigned* temp, bool spread, GridBarrier* bar, int* failed,
                       const DeviceInfo& dev, cudaStream_t stream, Status* status) {
  // A block per kRadixShare keys: ranking a share is a serial chain of its slices, so
  // blocks are worth their barrier arrivals; a single block needs no barrier at
  // all.  Whole sort with a block per 4096 keys -> this: 5 k keys 36 -> 34 us,
  // 20 k 52 -> 34, 100 k 51 -> 39; the slices spread over the warps, one block of
  // 1000 keys 28 -> 22.
  const int blocks = std::max(1, std::min({dev.sms, kRadixMaxBlocks, n / kRadixShare}));
  auto kernel = (long long)n <= (long long)blocks * (kRadixTile - 32) ? rs_sort<true> : rs_sort<false>;
  ECL_CUDA_TRY(launch_cooperative(kernel, blocks, kThreads, stream, k0, v0, k1, v1, order, n, n_dev, max_high, temp,
                                  spread, bar, failed, status));
  return ECL_OK;
}

}  // namespace ecl
