// The library's device memory: blocks for the outputs that it allocates, kept
// between calls, and its scratch.
//
// A product that allocates C pays cudaMalloc for it, and its caller cudaFree:
// for C of 555 MB that was 2.3 ms of a 3.9 ms call whose kernels take 1.5 ms,
// and for the 20 products of a batch 4 to 20 ms of 10 to 26. nspb_free
// therefore keeps a block that alloc_out handed out, and alloc_out gives it to
// the next request of about its size.
//
// What callers rely on stays:
//  - the block is an allocation of its own (cudaMalloc): cudaFree on it works,
//    and then it is simply gone. The driver numbers every allocation of the
//    process; a block is kept, given out again or freed here only while its
//    address still has the number it was allocated with, so one that its caller
//    freed as well is never touched, also when the address (and the size)
//    belong to someone else by then. nspb_free of a block that is kept already
//    is an error, as a second cudaFree was.
//  - nspb_free waits for the device like cudaFree, so that work in flight on
//    any stream has read a block before it is given out again, and where
//    cudaFree may be called it may be: it waits by freeing a block of 512 bytes
//    (4 us; the next one is allocated first, so that the driver does not give
//    up and map again the memory that it takes such blocks from: a product of
//    7 points on 149 x 131 x 97 nodes took 3.0 ms instead of 1.04).
//    cudaDeviceSynchronize would end every capture in progress on the device,
//    also those of other threads and relaxed ones, a plan's for instance. Where
//    cudaFree is not allowed (a global capture), the error is cudaFree's own.
// The blocks kept on a device hold at most a sixteenth of its memory, only
// while a quarter of it is free, the longest unused leave first, and all of
// them when an allocation of the library fails, for an output, for scratch or
// for a plan, which is then tried again: what a call could have while nspb_free
// gave every block back, it still has. nspb_trim gives them back at any time.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

#include "internal.h"
#include "spgemm_host.h"

namespace nspb {

namespace {

constexpr int kMaxDevices = 64;
constexpr size_t kGrain = 512;
constexpr size_t kSlack = 2u << 20;      // a block may exceed a request by this, or by an eighth
constexpr size_t kAskFree = 64u << 20;   // blocks from here on are kept only with memory to spare
constexpr size_t kMaxLive = 4096;

struct Block {
  void *p;
  size_t bytes;
  unsigned long long id;  // the driver's number of the allocation
};

struct Pool {
  std::mutex mu;
  std::vector<Block> kept;                   // oldest first
  size_t kept_bytes = 0;
  std::unordered_map<void *, Block> live;    // handed out and not seen by nspb_free
  Block token{nullptr, 0, 0};                // wait_for_device
};

// Bookkeeping that finds no host memory: the block is not kept (or not known as
// an output, so that nspb_free takes it to cudaFree). No exception leaves here,
// the callers are C functions.
template <typename F>
bool noted(F &&f) noexcept {
  try {
    f();
    return true;
  } catch (...) {
    return false;
  }
}

// Never destroyed: outputs may outlive the library's static objects.
Pool &pool_of(int dev) {
  alignas(Pool) static unsigned char room[sizeof(Pool) * kMaxDevices];
  static Pool *pools = [] {
    Pool *first = reinterpret_cast<Pool *>(room);
    for (int i = 0; i < kMaxDevices; ++i) new (first + i) Pool;
    return first;
  }();
  return pools[dev];
}

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return dev >= 0 && dev < kMaxDevices ? dev : -1;
}

// The number of the allocation that p lies in (unique in the process, and
// readable from a thread that has no context yet); 0 when it lies in none.
unsigned long long allocation_id(void *p) {
  using Attribute = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
  static const Attribute attribute = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<Attribute>(fn);
  }();
  unsigned long long id = 0;
  if (!attribute || attribute(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID,
                              reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS)
    return 0;
  return id;
}

bool still_block(const Block &b) { return b.id != 0 && allocation_id(b.p) == b.id; }

// Waits until the device has done all work given to it, as cudaFree does.
bool wait_for_device(Pool &pl) {
  void *p = nullptr;
  if (cudaMalloc(&p, kGrain) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  Block old{nullptr, 0, 0};
  {
    std::lock_guard<std::mutex> lock(pl.mu);
    old = pl.token;
    pl.token = Block{p, kGrain, allocation_id(p)};
  }
  if (!still_block(old)) {  // the first, or the device was reset
    old.p = nullptr;
    if (cudaMalloc(&old.p, kGrain) != cudaSuccess) old.p = nullptr;
  }
  if (old.p && cudaFree(old.p) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

cudaError_t drop(Pool &pl, size_t down_to) {
  cudaError_t first = cudaSuccess;
  while (!pl.kept.empty() && pl.kept_bytes > down_to) {
    const Block b = pl.kept.front();
    pl.kept.erase(pl.kept.begin());
    pl.kept_bytes -= b.bytes;
    const cudaError_t e = still_block(b) ? cudaFree(b.p) : cudaSuccess;
    if (first == cudaSuccess) first = e;
  }
  return first;
}

cudaError_t drop_all(Pool &pl) {
  const cudaError_t e = drop(pl, 0);
  if (still_block(pl.token)) cudaFree(pl.token.p);
  pl.token = Block{nullptr, 0, 0};
  return e;
}

}  // namespace

// cudaFree of every block kept on the current device; whether there was one.
static bool give_back() {
  const int dev = current_device();
  if (dev < 0) return false;
  Pool &pl = pool_of(dev);
  std::lock_guard<std::mutex> lock(pl.mu);
  const bool any = !pl.kept.empty();
  drop_all(pl);
  return any;
}

// Runs an allocation, and again without the kept blocks if there is no memory.
template <typename F>
static int allocate(F &&f) {
  cudaError_t e = f();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (give_back()) e = f();
  }
  if (e == cudaSuccess) return NSPB_OK;
  g_last_cuda = (int)e;
  cudaGetLastError();
  return NSPB_ERR_ALLOC;
}

int device_alloc(void **p, size_t bytes) {
  return allocate([&] { return cudaMalloc(p, bytes); });
}

// Library-owned stream-ordered pool per device; freed blocks stay cached.
static cudaMemPool_t scratch_pool() {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    if (cudaMemPoolCreate(&p, &props) != cudaSuccess) return nullptr;
    uint64_t keep = UINT64_MAX;
    cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    pools[dev] = p;
  }
  return pools[dev];
}

int scratch_alloc(void **p, size_t bytes, cudaStream_t s) {
  cudaMemPool_t pool = scratch_pool();
  if (!pool) return NSPB_ERR_ALLOC;
  return allocate([&] { return cudaMallocFromPoolAsync(p, bytes < 256 ? 256 : bytes, pool, s); });
}

void scratch_free(void *p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

int alloc_out(void **p, size_t bytes) {
  bytes = (std::max<size_t>(bytes, 4) + kGrain - 1) / kGrain * kGrain;
  const int dev = current_device();
  if (dev >= 0) {
    Pool &pl = pool_of(dev);
    std::lock_guard<std::mutex> lock(pl.mu);
    const size_t most = bytes + std::max(bytes / 8, std::min(bytes, kSlack));
    for (;;) {
      auto best = pl.kept.end();
      for (auto it = pl.kept.begin(); it != pl.kept.end(); ++it)
        if (it->bytes >= bytes && it->bytes <= most && (best == pl.kept.end() || it->bytes < best->bytes))
          best = it;
      if (best == pl.kept.end()) break;
      const Block b = *best;
      pl.kept_bytes -= b.bytes;
      pl.kept.erase(best);
      if (!still_block(b)) continue;  // its caller freed it as well
      *p = b.p;
      noted([&] { pl.live[b.p] = b; });
      return NSPB_OK;
    }
  }
  const int st = device_alloc(p, bytes);
  if (st) return st;
  if (dev >= 0) {
    Pool &pl = pool_of(dev);
    std::lock_guard<std::mutex> lock(pl.mu);
    // blocks that went to cudaFree directly leave entries behind
    if (pl.live.size() >= kMaxLive) pl.live.clear();
    noted([&] { pl.live[*p] = Block{*p, bytes, allocation_id(*p)}; });
  }
  return NSPB_OK;
}

// Takes the block of an output (1), or leaves it to cudaFree (0): it is not
// one, or there is no room for it. -1: it is kept already.
static int keep_out(void *p) {
  const int dev = current_device();
  if (dev < 0) return 0;
  Pool &pl = pool_of(dev);
  Block b;
  {
    std::lock_guard<std::mutex> lock(pl.mu);
    auto it = pl.live.find(p);
    if (it == pl.live.end()) {
      for (const Block &k : pl.kept)
        if (k.p == p && still_block(k)) return -1;
      return 0;
    }
    b = it->second;
    pl.live.erase(it);
  }
  const size_t cap = dev_info().total_mem / 16;
  if (b.bytes > cap || !still_block(b)) return 0;
  if (b.bytes >= kAskFree) {
    size_t free_b = 0, total = 0;
    if (cudaMemGetInfo(&free_b, &total) != cudaSuccess || free_b < total / 4) {
      cudaGetLastError();
      return 0;
    }
  }
  if (!wait_for_device(pl)) return 0;  // a capture in progress, or an earlier fault
  std::lock_guard<std::mutex> lock(pl.mu);
  drop(pl, cap - b.bytes);
  if (!noted([&] { pl.kept.push_back(b); })) return 0;
  pl.kept_bytes += b.bytes;
  return 1;
}

}  // namespace nspb

using namespace nspb;

extern "C" int nspb_free(void *p) {
  if (!p) return NSPB_OK;
  const int kept = keep_out(p);
  if (kept > 0) return NSPB_OK;
  const cudaError_t e = kept < 0 ? cudaErrorInvalidValue : cudaFree(p);
  if (e != cudaSuccess) {
    g_last_cuda = (int)e;
    cudaGetLastError();
    return NSPB_ERR_CUDA;
  }
  return NSPB_OK;
}

extern "C" int nspb_trim(void) {
  const int dev = current_device();
  if (dev < 0) return NSPB_ERR_NO_DEVICE;
  Pool &pl = pool_of(dev);
  std::lock_guard<std::mutex> lock(pl.mu);
  const cudaError_t e = drop_all(pl);
  if (e != cudaSuccess) {
    g_last_cuda = (int)e;
    cudaGetLastError();
    return NSPB_ERR_CUDA;
  }
  return NSPB_OK;
}
