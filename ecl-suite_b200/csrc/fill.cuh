// Byte fills of several arrays in one launch.
#pragma once

#include "runtime.cuh"

namespace ecl {

constexpr int kFills = 4;

struct Fill {
  void* p = nullptr;
  size_t bytes = 0;
  int value = 0;  // of every byte
};

// As a memset of each range, in stream order.  One launch, after which the next
// kernel is placed early (launch_next), instead of a memset node each: a solve
// of a small graph spent 2.5 us on every one.
void fill_ranges(const Fill (&f)[kFills], const DeviceInfo& dev, cudaStream_t stream);

}  // namespace ecl
