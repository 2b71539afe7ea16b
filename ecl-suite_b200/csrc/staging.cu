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

#include "runtime.cuh"

namespace ecl {

namespace {

constexpr size_t kPiece = size_t(1) << 20;
constexpr int kPieces = 4;       // per block
constexpr int kMaxBlocks = 4;    // 16 MB of page-locked memory for a context at most ...
constexpr int kMaxContexts = 8;  // ... and for this many of them (one for each device)
constexpr size_t kStageMin = size_t(256) << 10;  // below, the plain copy is as fast
constexpr int kCopyThreads = 4;

}  // namespace

struct StageBlock {
  char* base = nullptr;
  unsigned long long ctx = 0;  // context of the memory and the events (0: not made)
  cudaEvent_t done[kPieces] = {};
  bool taken = false;
};

namespace {

// Blocks are made when first wanted (4 ms each) and kept until the process
// ends, kMaxBlocks for a context: a copy that finds none is made without.  A
// block belongs to the context it was made in.  When that context has ended
// (cudaDeviceReset), the memory and the events ended with it: the block is made
// anew, and nothing of the old one is touched, not even to free it.
class Pool {
 public:
  StageBlock* take(unsigned long long ctx) {
    std::lock_guard<std::mutex> lk(mu_);
    int made = 0;
    for (StageBlock& b : blocks_) {
      if (b.ctx != ctx) continue;
      made++;
      if (b.taken) continue;
      b.taken = true;
      return &b;
    }
    if (made == kMaxBlocks) return nullptr;
    StageBlock* room = nullptr;
    for (StageBlock& b : blocks_)
      if (!room && !b.taken && (b.ctx == 0 || gone(b))) room = &b;
    if (!room || !make(room, ctx)) return nullptr;
    room->taken = true;
    return room;
  }
  void give(StageBlock* b) {
    std::lock_guard<std::mutex> lk(mu_);
    b->taken = false;
  }
  ~Pool() {
    const unsigned long long ctx = context_id();
    for (StageBlock& b : blocks_)
      if (ctx != 0 && b.ctx == ctx) cudaFreeHost(b.base);
  }

 private:
  // Another context's block is taken to be gone when its memory is no longer
  // page-locked; a live one stays for its own context.
  static bool gone(const StageBlock& b) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, b.base) == cudaSuccess) return at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false;
  }
  static bool make(StageBlock* b, unsigned long long ctx) {
    *b = StageBlock{};
    void* p = nullptr;
    if (cudaHostAlloc(&p, kPiece * kPieces, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    for (cudaEvent_t& e : b->done)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        for (cudaEvent_t made : b->done)
          if (made) cudaEventDestroy(made);
        cudaFreeHost(p);
        *b = StageBlock{};
        return false;
      }
    b->base = static_cast<char*>(p);
    b->ctx = ctx;
    return true;
  }

  std::mutex mu_;
  StageBlock blocks_[kMaxBlocks * kMaxContexts];
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
  const unsigned long long ctx = context_id();
  if (ctx == 0) return false;
  if (block_) return block_->ctx == ctx;
  block_ = g_pool.take(ctx);
  used_ = 0;
  return block_ != nullptr;
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
