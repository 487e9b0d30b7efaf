// A CUDA runtime that allocates addresses only, for the host tests of
// nsp_b200/csrc/outpool.cpp: the lowest free address is given out first, every
// allocation has a number, and a thread can be told that it has no context.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>

#include "internal.h"
#include "spgemm_host.h"

namespace {
bool no_host_memory = false;
}
// what outpool.cpp's containers allocate with
void *operator new(size_t bytes) {
  if (no_host_memory) throw std::bad_alloc();
  if (void *p = std::malloc(bytes)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

namespace {

struct Alloc {
  size_t bytes;
  unsigned long long id;
};
std::recursive_mutex mu;
std::map<size_t, Alloc> mem;  // by address
unsigned long long next_id = 1;
size_t capacity = (size_t)180 << 30;
thread_local bool no_context = false;
int capture = 0;           // 0 none, 1 another thread's thread-local or a relaxed one, 2 global
bool capture_ends = false; // a call that is not allowed in it was made
int waits = 0;             // calls that waited for the device

// A call that a capture of this kind (and any stricter one) does not allow.
bool forbidden(int from) {
  if (capture < from) return false;
  capture_ends = true;
  return true;
}

size_t used() {
  size_t sum = 0;
  for (auto &a : mem) sum += a.second.bytes;
  return sum;
}

cudaError_t take(void **p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (used() + bytes > capacity) return cudaErrorMemoryAllocation;
  size_t at = 4096;
  for (auto &a : mem) {
    if (a.first - at >= bytes) break;
    at = a.first + a.second.bytes;
  }
  const bool was = no_host_memory;  // the fake's own books are another matter
  no_host_memory = false;
  mem[at] = Alloc{bytes, next_id++};
  no_host_memory = was;
  *p = reinterpret_cast<void *>(at);
  return cudaSuccess;
}

std::map<size_t, Alloc>::iterator find(size_t at) {
  auto it = mem.upper_bound(at);
  if (it == mem.begin()) return mem.end();
  --it;
  return at < it->first + it->second.bytes ? it : mem.end();
}

CUresult attribute(void *out, CUpointer_attribute what, CUdeviceptr p) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  auto it = find((size_t)p);
  if (it == mem.end() || what != CU_POINTER_ATTRIBUTE_BUFFER_ID) return CUDA_ERROR_INVALID_VALUE;
  *static_cast<unsigned long long *>(out) = it->second.id;
  return CUDA_SUCCESS;
}

CUresult range(CUdeviceptr *base, size_t *size, CUdeviceptr p) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (no_context) return CUDA_ERROR_INVALID_CONTEXT;
  auto it = find((size_t)p);
  if (it == mem.end()) return CUDA_ERROR_NOT_FOUND;
  *base = it->first;
  *size = it->second.bytes;
  return CUDA_SUCCESS;
}

}  // namespace

namespace nspb {
thread_local int g_last_cuda = 0;
const DevInfo &dev_info() {
  static DevInfo d;
  d.total_mem = capacity;
  return d;
}
}  // namespace nspb

extern "C" {

cudaError_t cudaGetDevice(int *dev) {
  *dev = 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t bytes) {
  no_context = false;
  if (forbidden(2)) return cudaErrorStreamCaptureUnsupported;
  return take(p, bytes);
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  no_context = false;
  if (forbidden(2)) return cudaErrorStreamCaptureUnsupported;
  ++waits;
  return mem.erase(reinterpret_cast<size_t>(p)) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaDeviceSynchronize(void) {
  if (forbidden(1)) return cudaErrorStreamCaptureUnsupported;
  ++waits;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *) {
  *pool = reinterpret_cast<cudaMemPool_t>(&mem);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t, cudaStream_t) {
  return take(p, bytes);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  return mem.erase(reinterpret_cast<size_t>(p)) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaMemGetInfo(size_t *free_b, size_t *total) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  *total = capacity;
  *free_b = capacity - used();
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *at, const void *p) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  std::memset(at, 0, sizeof(*at));
  at->type = find(reinterpret_cast<size_t>(p)) == mem.end() ? cudaMemoryTypeUnregistered
                                                            : cudaMemoryTypeDevice;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **fn, unsigned long long,
                                    cudaDriverEntryPointQueryResult *q) {
  *fn = !std::strcmp(name, "cuPointerGetAttribute")  ? reinterpret_cast<void *>(&attribute)
        : !std::strcmp(name, "cuMemGetAddressRange") ? reinterpret_cast<void *>(&range)
                                                     : nullptr;
  *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}

// ---- for the tests ----
void *fake_malloc(size_t bytes) {
  void *p = nullptr;
  return take(&p, bytes) == cudaSuccess ? p : nullptr;
}
int fake_free(void *p) { return (int)cudaFree(p); }
size_t fake_used(void) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  return used();
}
void fake_capacity(size_t bytes) { capacity = bytes; }
void fake_capture(int kind) {
  capture = kind;
  capture_ends = false;
}
int fake_capture_ends(void) { return capture_ends; }
int fake_waits(void) { return waits; }
void fake_no_host_memory(int yes) { no_host_memory = yes; }
void fake_no_context(void) { no_context = true; }
int fake_scratch(void **p, size_t bytes) { return nspb::scratch_alloc(p, bytes, nullptr); }
int fake_device(void **p, size_t bytes) { return nspb::device_alloc(p, bytes); }
int fake_alloc_out(void **p, size_t bytes) { return nspb::alloc_out(p, bytes); }
}
