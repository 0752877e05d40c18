// Device buffers of finished batch calls (prims.cu), kept for the next ones: cudaMalloc and cudaFree
// cost a call of few stencils more than its copies and its kernel (497 us a call of 300 edge
// pairs, 332 us with the pool). At most POOL_BUFS of at most POOL_BYTES each: 32 MB are a batch of
// 24 000 Hessians, whose call takes 1.1 to 1.7 ms, against 0.17 to 0.3 ms of allocation and release.
// A buffer belongs to one call at a time, which hands it back after its last synchronous
// copy (after an error it is freed). The kept ones are freed when any allocation of the library finds
// the device full, on abd_release_buffers, and when the library is unloaded.
//
// A kept address is only as good as its allocation: after cudaDeviceReset, or in another
// context of the same device, it may be nobody's or somebody else's (a reset gives the same
// addresses out again). A buffer is therefore known by the identifier that the driver gave its
// allocation, which no later one in the process gets, and by its context; both are
// asked for when it is taken and before it is freed.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>

namespace abd {

constexpr int POOL_BUFS = 4;
constexpr size_t POOL_BYTES = (size_t)32 << 20;

struct BatchBuf {
  void* p = nullptr;
  size_t bytes = 0;
  void* ctx = nullptr;        // context and identifier of the allocation (0: not known, never kept)
  unsigned long long id = 0;
};
BatchBuf batch_take(size_t bytes);             // throws CudaError
void batch_give(const BatchBuf& b, bool keep);  // keep: the work on it has ended
void batch_release();                           // frees the kept buffers

}  // namespace abd
