// Device memory of the operators (internal to libsgpp_gb300): stream-ordered allocations, so
// that creating and destroying operators in several host threads never synchronises the whole
// device (cudaFree does), and small pinned host blocks recycled instead of freed.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace sgmev {

// stream-ordered allocation on `s` from the library's own memory pool on the current device
// (created once per device; it keeps freed memory for reuse and is trimmed when an allocation
// fails); *p is nullptr on failure
cudaError_t dev_malloc(void** p, size_t bytes, cudaStream_t s);

template <typename T>
inline cudaError_t dev_malloc(T** p, size_t bytes, cudaStream_t s) {
  return dev_malloc(reinterpret_cast<void**>(p), bytes, s);
}

// bytes that dev_malloc could give out on the current device: free ones and the pool's own unused blocks
size_t dev_available();
// cudaFreeAsync on `s` (nullptr is accepted); the memory is reused once `s` reaches this point
void dev_free(void* p, cudaStream_t s);

// A non-blocking stream of the current device for one operator, and its return once it is idle (up to
// 32 streams per device are kept). An operator that takes over an earlier one's stream finds that
// one's freed memory on its own stream; blocks freed on streams that are gone cost the pool a
// search through all of them on every allocation, so that creating an operator took 0.25 ms in a
// fresh process and 2.4 ms after 48 others had come and gone.
cudaStream_t stream_acquire();
void stream_release(cudaStream_t s);

// Pinned host buffers of kPinnedBuffer bytes, for small host vectors that the kernels read and write in
// place (up to 16 idle ones are kept); nullptr when there is no memory for one
constexpr size_t kPinnedBuffer = 96 * 1024;
double* pinned_buffer();
void pinned_buffer_release(double* p);

// 64-byte pinned host blocks for scalars read back from the device
void* pinned_block();
void pinned_release(void* p);

}  // namespace sgmev
