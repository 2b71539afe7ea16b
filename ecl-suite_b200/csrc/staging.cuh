// Copies between the device and pageable host memory through page-locked
// blocks of this library.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace ecl {

struct StageBlock;

// One user of a block: takes it from the process's pool at its first copy that
// wants one and gives it back in release() or its destructor.  Not for
// several threads at once; the pool is.
class Staging {
 public:
  Staging() = default;
  Staging(const Staging&) = delete;
  Staging& operator=(const Staging&) = delete;
  ~Staging() { release(); }

  // False: not a copy for a block (small, host memory that is page-locked
  // already, no block free, no threads to copy with); nothing was done and the
  // caller makes the plain copy.  True: *err is the copy's outcome.
  // to_device: `src` has been read on return, the device copy is in the
  // stream.  to_host: all bytes have arrived on return.
  bool to_device(void* dst, const void* src, size_t bytes, cudaStream_t stream, cudaError_t* err);
  bool to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream, cudaError_t* err);
  // Waits for the block's copies and gives it back.
  void release();

 private:
  bool ready(const void* host, size_t bytes);
  StageBlock* block_ = nullptr;
  size_t used_ = 0;  // pieces that have had a copy issued
};

}  // namespace ecl
