// Device memory of plans.
//
// cudaMalloc and cudaFree map and unmap memory and wait for the device: making and
// destroying the plan of a 49,266-element model took about 4 ms of them, three times its
// kernels. Plans take their memory from one pool per device instead, which keeps up to
// kKeep bytes of what they free and returns the rest. Allocation and release both go
// through one stream of the pool: a block is free once every stream is done with it
// (device_free's contract), so the next owner needs no ordering of its own. Blocks above
// kPooled, which it would not keep, come from cudaMalloc: growing a pool by them took longer
// (first assembly of a C3D20 plan with 0.9 GB of element blocks 5.8 ms, from cudaMalloc 1.6).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <unordered_set>

#include "cxg_internal.cuh"

namespace cxg {

namespace {

constexpr uint64_t kKeep = 512ull << 20;
constexpr size_t kPooled = 256ull << 20;
constexpr int kMaxDevices = 64;

struct Pool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;
};
std::mutex g_mu;
Pool g_pools[kMaxDevices];
std::unordered_set<void*> g_large;  // the blocks in use that cudaMalloc gave

// The current device's pool, made on first use; null where the device has none.
cudaError_t pool_of(Pool* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_mu);
  Pool& p = g_pools[dev];
  if (!p.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    Pool n;
    uint64_t keep = kKeep;
    if ((e = cudaStreamCreateWithFlags(&n.stream, cudaStreamNonBlocking)) != cudaSuccess) return e;
    if ((e = cudaMemPoolCreate(&n.pool, &props)) == cudaSuccess)
      e = cudaMemPoolSetAttribute(n.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      if (n.pool) cudaMemPoolDestroy(n.pool);
      cudaStreamDestroy(n.stream);
      return e;
    }
    p = n;
  }
  *out = p;
  return cudaSuccess;
}

// alloc(), and where it finds no memory once more with what the pool keeps returned.
template <class F>
cudaError_t or_trim(F alloc) {
  cudaError_t e = alloc();
  Pool p;
  if (e != cudaErrorMemoryAllocation || pool_of(&p) != cudaSuccess) return e;
  cudaGetLastError();
  cudaStreamSynchronize(p.stream);  // the frees before it
  if (cudaMemPoolTrimTo(p.pool, 0) != cudaSuccess) return e;
  return alloc();
}

}  // namespace

cudaError_t device_malloc(void** out, size_t bytes) {
  *out = nullptr;
  return or_trim([&] { return cudaMalloc(out, bytes); });
}

cudaError_t device_malloc_async(void** out, size_t bytes, cudaStream_t s) {
  *out = nullptr;
  return or_trim([&] { return cudaMallocAsync(out, bytes, s); });
}

cudaError_t device_alloc(void** out, size_t bytes) {
  *out = nullptr;
  if (bytes > kPooled) {
    const cudaError_t e = device_malloc(out, bytes);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_mu);
    g_large.insert(*out);
    return e;
  }
  Pool p;
  cudaError_t e = pool_of(&p);
  if (e != cudaSuccess) return e;
  e = or_trim([&] { return cudaMallocFromPoolAsync(out, std::max<size_t>(bytes, 16), p.pool, p.stream); });
  if (e == cudaSuccess) e = cudaStreamSynchronize(p.stream);
  return e;
}

void device_free(void* ptr) {
  {
    std::unique_lock<std::mutex> lock(g_mu);
    if (g_large.erase(ptr)) {
      lock.unlock();
      cudaFree(ptr);
      return;
    }
  }
  Pool p;
  if (ptr && pool_of(&p) == cudaSuccess) cudaFreeAsync(ptr, p.stream);
}

bool kernel_reads(int device, const void* ptr) {
  cudaPointerAttributes at;
  if (!ptr || reinterpret_cast<uintptr_t>(ptr) % sizeof(double) != 0) return false;
  if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == device);
}

void device_free_all(int device, void* const* blocks, int n) {
  int current = device;
  cudaGetDevice(&current);
  if (current != device) cudaSetDevice(device);
  cudaDeviceSynchronize();
  for (int i = 0; i < n; ++i) device_free(blocks[i]);
  Pool p;
  if (pool_of(&p) == cudaSuccess) cudaStreamSynchronize(p.stream);  // applies the pool's threshold
  if (current != device) cudaSetDevice(current);
}

}  // namespace cxg
