// Page-locked blocks for copies of pageable memory: see staging.cuh.
//
// The driver copies pageable memory with one thread through its own blocks,
// about 18 GB/s either way.  Here four threads fill (or empty) a piece while
// the copy engine works on the one before it.  Measured, 16 host cores:
// 4.8 MB to the device 303 -> 197 us, to the host 271 -> 156; 512 kB 42 -> 34
// and 52 -> 31; 256 kB 26 -> 25 and 33 -> 21.  One thread gains nothing (312
// and 313 us), eight no more than four (189 and 168).
#include "staging.cuh"

#include <omp.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

namespace ecl {

namespace {

constexpr size_t kPiece = size_t(1) << 20;
constexpr int kPieces = 4;  // per block
constexpr int kMaxBlocks = 4;  // 16 MB of page-locked memory at most
constexpr size_t kStageMin = size_t(256) << 10;  // below, the plain copy is as fast
constexpr int kCopyThreads = 4;

}  // namespace

struct StageBlock {
  char* base = nullptr;
  int device = -1;  // of the events
  cudaEvent_t done[kPieces] = {};
};

namespace {

// Blocks are made when first wanted (4 ms each) and kept until the process
// ends, kMaxBlocks in all: a copy that finds none free is made without.
class Pool {
 public:
  StageBlock* take() {
    std::lock_guard<std::mutex> lk(mu_);
    if (nfree_ > 0) return free_[--nfree_];
    if (made_ == kMaxBlocks) return nullptr;
    void* p = nullptr;
    if (cudaHostAlloc(&p, kPiece * kPieces, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    StageBlock* b = &blocks_[made_++];
    b->base = static_cast<char*>(p);
    return b;
  }
  void give(StageBlock* b) {
    std::lock_guard<std::mutex> lk(mu_);
    free_[nfree_++] = b;
  }
  ~Pool() {
    for (int i = 0; i < nfree_; i++) cudaFreeHost(free_[i]->base);
  }

 private:
  std::mutex mu_;
  StageBlock blocks_[kMaxBlocks];
  StageBlock* free_[kMaxBlocks] = {};
  int nfree_ = 0, made_ = 0;
};

Pool g_pool;

int copy_threads() { return omp_in_parallel() ? 1 : std::min(kCopyThreads, omp_get_max_threads()); }

void copy_parallel(char* dst, const char* src, size_t bytes) {
#pragma omp parallel num_threads(copy_threads())
  {
    const size_t t = (size_t)omp_get_thread_num(), nt = (size_t)omp_get_num_threads();
    const size_t beg = bytes * t / nt & ~size_t(63), end = t + 1 == nt ? bytes : (bytes * (t + 1) / nt & ~size_t(63));
    memcpy(dst + beg, src + beg, end - beg);
  }
}

}  // namespace

bool Staging::ready(const void* host, size_t bytes) {
  if (bytes < kStageMin || copy_threads() < kCopyThreads) return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (at.type != cudaMemoryTypeUnregistered) return false;
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess) return false;
  if (block_ && block_->device != device) return false;  // (its events are another device's)
  if (block_) return true;
  block_ = g_pool.take();
  if (!block_) return false;
  used_ = 0;
  if (block_->device != device) {
    for (cudaEvent_t& e : block_->done) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    block_->device = -1;
    for (cudaEvent_t& e : block_->done)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        release();
        return false;
      }
    block_->device = device;
  }
  return true;
}

bool Staging::to_device(void* dst, const void* src, size_t bytes, cudaStream_t stream, cudaError_t* err) {
  if (!ready(src, bytes)) return false;
  *err = cudaSuccess;
  for (size_t at = 0; at < bytes && *err == cudaSuccess; at += kPiece) {
    const size_t len = std::min(kPiece, bytes - at), slot = used_ % kPieces;
    char* p = block_->base + slot * kPiece;
    if (used_ >= kPieces) *err = cudaEventSynchronize(block_->done[slot]);
    if (*err != cudaSuccess) break;
    copy_parallel(p, static_cast<const char*>(src) + at, len);
    *err = cudaMemcpyAsync(static_cast<char*>(dst) + at, p, len, cudaMemcpyHostToDevice, stream);
    if (*err == cudaSuccess) *err = cudaEventRecord(block_->done[slot], stream);
    used_++;
  }
  return true;
}

bool Staging::to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream, cudaError_t* err) {
  if (!ready(dst, bytes)) return false;
  *err = cudaSuccess;
  const size_t pieces = (bytes + kPiece - 1) / kPiece, first = used_;
  size_t issued = 0;
  for (size_t k = 0; k < pieces; k++) {
    // a piece's earlier copy is ordered before in this stream, or emptied below
    for (; issued < pieces && issued < k + kPieces && *err == cudaSuccess; issued++, used_++) {
      const size_t slot = (first + issued) % kPieces;
      if (first + issued >= kPieces && issued < kPieces) *err = cudaEventSynchronize(block_->done[slot]);
      if (*err == cudaSuccess)
        *err = cudaMemcpyAsync(block_->base + slot * kPiece, static_cast<const char*>(src) + issued * kPiece,
                               std::min(kPiece, bytes - issued * kPiece), cudaMemcpyDeviceToHost, stream);
      if (*err == cudaSuccess) *err = cudaEventRecord(block_->done[slot], stream);
    }
    const size_t slot = (first + k) % kPieces;
    if (*err == cudaSuccess) *err = cudaEventSynchronize(block_->done[slot]);
    if (*err != cudaSuccess) break;
    copy_parallel(static_cast<char*>(dst) + k * kPiece, block_->base + slot * kPiece, std::min(kPiece, bytes - k * kPiece));
  }
  return true;
}

void Staging::release() {
  if (!block_) return;
  for (size_t k = 0; k < std::min(used_, (size_t)kPieces); k++) cudaEventSynchronize(block_->done[k]);
  g_pool.give(block_);
  block_ = nullptr;
}

}  // namespace ecl
