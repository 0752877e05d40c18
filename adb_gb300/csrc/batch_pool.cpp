#include "batch_pool.h"

#include <cuda.h>

#include <mutex>
#include <utility>
#include <vector>

#include "abd_engine.h"

namespace abd {
namespace {

// The driver's calls by way of the runtime: the library does not link against the driver.
struct Driver {
  CUresult (*attribute)(void*, CUpointer_attribute, CUdeviceptr) = nullptr;
  CUresult (*current)(CUcontext*) = nullptr;
  Driver() {
    cudaDriverEntryPointQueryResult q;
    void *a = nullptr, *c = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &a, 4000, cudaEnableDefault, &q) != cudaSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &c, 4000, cudaEnableDefault, &q) != cudaSuccess) {
      (void)cudaGetLastError();
      return;  // nothing is known of any buffer: none is kept
    }
    attribute = reinterpret_cast<decltype(attribute)>(a);
    current = reinterpret_cast<decltype(current)>(c);
  }
};
const Driver& driver() {
  static const Driver d;
  return d;
}

void* current_context() {
  CUcontext c = nullptr;
  return driver().current && driver().current(&c) == CUDA_SUCCESS ? c : nullptr;
}
// Identifier of the allocation at p, 0 where there is none.
unsigned long long buffer_id(void* p) {
  unsigned long long id = 0;
  const CUdeviceptr a = (CUdeviceptr)p;
  return driver().attribute && driver().attribute(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, a) == CUDA_SUCCESS ? id : 0;
}
bool alive(const BatchBuf& b) { return b.id && buffer_id(b.p) == b.id; }

struct Pool {
  std::mutex m;
  std::vector<BatchBuf> idle;
  Pool() { idle.reserve(POOL_BUFS + 1); }
  ~Pool() { trim(); }
  static void drop(const BatchBuf& b) {
    if (alive(b) && cudaFree(b.p) != cudaSuccess) (void)cudaGetLastError();
  }
  void trim() {
    std::lock_guard<std::mutex> l(m);
    for (const BatchBuf& b : idle) drop(b);
    idle.clear();
  }
};
Pool g_pool;

}  // namespace

void* device_alloc(size_t bytes) {
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    batch_release();
    CK(cudaMalloc(&p, bytes));
  }
  return p;
}

void batch_release() { g_pool.trim(); }

BatchBuf batch_take(size_t bytes) {
  void* ctx = current_context();
  if (!ctx && cudaFree(nullptr) == cudaSuccess) ctx = current_context();  // a thread's first call
  if (ctx) {
    std::lock_guard<std::mutex> l(g_pool.m);
    std::vector<BatchBuf>& idle = g_pool.idle;
    for (;;) {
      int best = -1;
      for (int i = 0; i < (int)idle.size(); ++i)
        if (idle[i].ctx == ctx && idle[i].bytes >= bytes && (best < 0 || idle[i].bytes < idle[best].bytes)) best = i;
      if (best < 0) break;
      const BatchBuf b = idle[best];
      idle.erase(idle.begin() + best);
      if (alive(b)) return b;
    }
  }
  BatchBuf b;
  b.bytes = bytes;
  b.p = device_alloc(bytes);
  b.ctx = current_context();
  b.id = b.ctx ? buffer_id(b.p) : 0;
  return b;
}

void batch_give(const BatchBuf& b, bool keep) {
  BatchBuf out = b;
  if (keep && b.id && b.bytes <= POOL_BYTES) {
    std::lock_guard<std::mutex> l(g_pool.m);
    g_pool.idle.push_back(b);
    if ((int)g_pool.idle.size() <= POOL_BUFS) return;
    size_t least = 0;  // the smallest one goes
    for (size_t i = 1; i < g_pool.idle.size(); ++i)
      if (g_pool.idle[i].bytes < g_pool.idle[least].bytes) least = i;
    out = g_pool.idle[least];
    g_pool.idle.erase(g_pool.idle.begin() + (ptrdiff_t)least);
    Pool::drop(out);
    return;
  }
  if (cudaFree(out.p) != cudaSuccess) (void)cudaGetLastError();
}

}  // namespace abd

extern "C" int abd_release_buffers(void) {
  abd::batch_release();
  return ABD_OK;
}
