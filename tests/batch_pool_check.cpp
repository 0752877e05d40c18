// CPU check of the pool of device buffers (batch_pool.cpp) over a device that this file plays:
// allocations with identifiers that are never given twice, addresses that are, a device of a
// stated size, contexts, and a reset. Prints what went wrong; exit status 1 if anything did.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstring>
#include <map>

#include "../adb_gb300/csrc/abd_engine.h"
#include "../adb_gb300/csrc/batch_pool.h"

namespace {
struct Alloc {
  size_t bytes;
  unsigned long long id;
};
std::map<size_t, Alloc> live;  // by address
unsigned long long next_id = 1;
size_t room = (size_t)1 << 30, used = 0;
int allocs = 0, wrong_frees = 0, bad = 0;
void* context = (void*)0x10;

CUresult attribute(void* out, CUpointer_attribute what, CUdeviceptr p) {
  if (what != CU_POINTER_ATTRIBUTE_BUFFER_ID || !live.count(p)) return CUDA_ERROR_INVALID_VALUE;
  memcpy(out, &live[p].id, sizeof(unsigned long long));
  return CUDA_SUCCESS;
}
CUresult current(CUcontext* c) {
  *c = (CUcontext)context;
  return CUDA_SUCCESS;
}
void reset() {
  live.clear();
  used = 0;
}
void expect(bool ok, const char* what) {
  if (!ok) {
    printf("wrong: %s\n", what);
    ++bad;
  }
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  ++allocs;
  if (used + n > room) return cudaErrorMemoryAllocation;
  size_t at = 1 << 20;  // the lowest free address
  for (auto& a : live) {
    if (a.first >= at + n) break;
    at = a.first + a.second.bytes;
  }
  live[at] = Alloc{n, next_id++};
  used += n;
  *p = (void*)at;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  if (!live.count((size_t)p)) {
    ++wrong_frees;
    return cudaErrorInvalidValue;
  }
  used -= live[(size_t)p].bytes;
  live.erase((size_t)p);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
  *f = !strcmp(name, "cuPointerGetAttribute") ? (void*)attribute : (void*)current;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
}
void abd::check(cudaError_t e, const char* where) {
  if (e != cudaSuccess) throw CudaError{e, where};
}

int main() {
  using namespace abd;
  const size_t MB = (size_t)1 << 20;
  // kept and taken again
  BatchBuf a = batch_take(MB);
  batch_give(a, true);
  int n = allocs;
  BatchBuf b = batch_take(MB / 2);
  expect(b.p == a.p && allocs == n, "a kept buffer serves the next call");
  batch_give(b, true);
  // at most POOL_BUFS stay
  BatchBuf many[6];
  for (int i = 0; i < 6; ++i) many[i] = batch_take((i + 2) * MB);
  for (int i = 0; i < 6; ++i) batch_give(many[i], true);
  expect((int)live.size() <= POOL_BUFS, "no more than POOL_BUFS are kept");
  BatchBuf big = batch_take(POOL_BYTES + 1);
  batch_give(big, true);
  expect((int)live.size() <= POOL_BUFS, "a buffer past POOL_BYTES is freed");
  // another context of the device
  context = (void*)0x20;
  n = allocs;
  BatchBuf other = batch_take(MB);
  expect(allocs == n + 1, "a buffer of another context is not used");
  batch_give(other, false);
  context = (void*)0x10;
  // a reset, after which somebody else gets the old addresses
  reset();
  void* theirs[8];
  for (void*& t : theirs) cudaMalloc(&t, MB);
  n = allocs;
  BatchBuf c = batch_take(MB / 4);
  bool mine = true;
  for (void* t : theirs) mine &= c.p != t;
  expect(mine && allocs == n + 1, "after a reset a kept address is not used");
  batch_give(c, true);
  for (int i = 0; i < 6; ++i) many[i] = batch_take((i + 2) * MB);
  for (int i = 0; i < 6; ++i) batch_give(many[i], true);
  bool intact = true;
  for (void* t : theirs) intact &= live.count((size_t)t) != 0;
  expect(intact, "after a reset nobody else's allocation is freed");
  // a full device: the kept buffers make room
  room = used + 4 * MB;
  bool got = true;
  try {
    batch_give(batch_take(20 * MB), false);
  } catch (const CudaError&) {
    got = false;
  }
  expect(got, "a batch call gets the room of the kept buffers");
  room = (size_t)1 << 30;
  for (int i = 0; i < 4; ++i) many[i] = batch_take((i + 2) * MB);
  for (int i = 0; i < 4; ++i) batch_give(many[i], true);
  room = used + 4 * MB;
  DBuf<char> handle;  // a simulation's buffer
  try {
    handle.ensure(10 * MB);
  } catch (const CudaError&) {
  }
  expect(handle.p != nullptr, "a simulation gets the room of the kept buffers");
  handle.release();
  room = (size_t)1 << 30;
  batch_give(batch_take(MB), true);
  batch_release();
  expect(used == 8 * MB, "a release leaves nothing kept");  // their eight
  expect(wrong_frees == 0, "nothing is freed twice");
  return bad != 0;
}
