// Byte fills of several arrays in one launch: see fill.cuh.
#include "fill.cuh"

namespace ecl {
namespace {

constexpr int kTPB = 256;

struct Fills {
  Fill f[kFills];
};

// Whole 16-byte words by all threads, the bytes before and after them by the
// first ones.  Bound by the stores (128 MB of MST flags: 20 us, as memset).
__global__ void __launch_bounds__(kTPB) fill_kernel(const __grid_constant__ Fills a) {
  dev::dep_wait();
  const size_t t = (size_t)blockIdx.x * kTPB + threadIdx.x, nt = (size_t)gridDim.x * kTPB;
#pragma unroll
  for (int r = 0; r < kFills; r++) {
    unsigned char* p = static_cast<unsigned char*>(a.f[r].p);
    const size_t bytes = a.f[r].bytes;
    const unsigned char v = (unsigned char)a.f[r].value;
    const size_t to16 = (16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15, head = to16 < bytes ? to16 : bytes;
    const size_t words = (bytes - head) / 16, tail = (bytes - head) % 16;
    const int w = v * 0x01010101;
    int4* q = reinterpret_cast<int4*>(p + head);
    for (size_t i = t; i < words; i += nt) q[i] = make_int4(w, w, w, w);
    if (t < head) p[t] = v;
    if (t < tail) p[head + words * 16 + t] = v;
  }
}

}  // namespace

void fill_ranges(const Fill (&f)[kFills], const DeviceInfo& dev, cudaStream_t stream) {
  Fills a;
  size_t bytes = 0;
  for (int r = 0; r < kFills; r++) {
    a.f[r] = f[r];
    bytes += f[r].bytes;
  }
  const size_t blocks = bytes / (kTPB * 64) + 1;  // 64 bytes a thread
  ECL_LAUNCH_NEXT(fill_kernel, (int)std::min(blocks, (size_t)dev.sms * 16), kTPB, 0, stream, a);
}

}  // namespace ecl
