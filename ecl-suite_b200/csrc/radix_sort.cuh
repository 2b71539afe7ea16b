// Stable LSD radix sort of (uint64 key, int32 value) pairs, 8-bit digits, in
// ONE cooperative launch: the order of the values by key is all it returns.
//
// Keys are ~((d << 32) | h) with 32 varying bits h and a count d whose largest
// value is known on the device only: the passes are those over h (two to four
// of them) and those that the largest d needs (one below 256), so the pass
// count is decided inside the launch and costs the host nothing.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "grid_sync.cuh"
#include "runtime.cuh"

namespace ecl {

// Keys a block places per step (1024 threads x 8 keys).
constexpr int kRadixTile = 8192;
constexpr int kRadixMaxBlocks = 256;  // blocks the count table holds
constexpr int kRadixShare = 1024;     // a block per this many keys
// Words of radix_order()'s count table for n keys.
constexpr size_t radix_temp_words(int n) {
  return (size_t)256 * (n / kRadixShare < kRadixMaxBlocks ? n / kRadixShare + 1 : kRadixMaxBlocks);
}

// order[0 .. *n_dev) = the values of the pairs (k0, v0)[0 .. *n_dev) by
// ascending key, equal keys in their input order.  *n_dev <= n (which sizes
// the launch), *max_high = the largest d; (k1, v1) is scratch of n pairs, k0
// and v0 are overwritten; spread: the h of different keys differ, but for a
// few, and are spread evenly (the time depends on it, the order does not);
// `temp` holds radix_temp_words(n) and `bar` is zeroed.
// The order is whole (every value once) whatever status->code says; only when
// a grid barrier times out it is not: ECL_ERR_NO_CONVERGENCE is raised in
// `status`, *failed (zeroed before) becomes 1, and readers must check it.
ecl_status radix_order(unsigned long long* k0, int* v0, unsigned long long* k1, int* v1, int* order, int n,
                       const int* n_dev, const int* max_high, unsigned* temp, bool spread, dev::GridBarrier* bar,
                       int* failed, const DeviceInfo& dev, cudaStream_t stream, dev::Status* status);

}  // namespace ecl
