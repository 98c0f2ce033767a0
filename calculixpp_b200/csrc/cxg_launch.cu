// Launch figures kept per thread, and launches that overlap the drain of the kernel before.
//
// A small assembly is two kernels of 6 and 8 us. Asking the runtime for attributes,
// occupancy and SM count on every call took 5 us of the host, and the second kernel's
// start-up followed the first one's end.
#include <cuda_runtime.h>

#include <mutex>
#include <unordered_map>

#include "cxg_internal.cuh"

namespace cxg {

namespace {

struct Key {
  const void* kern;
  size_t smem;
  int threads, device;
  bool operator==(const Key& o) const {
    return kern == o.kern && smem == o.smem && threads == o.threads && device == o.device;
  }
};
struct Hash {
  size_t operator()(const Key& k) const {
    return (reinterpret_cast<size_t>(k.kern) >> 4) * 1099511628211ull ^ (k.smem << 20) ^ (static_cast<size_t>(k.threads) << 8) ^
           static_cast<size_t>(k.device);
  }
};
struct Shape {
  int per_sm, sms;
};
thread_local std::unordered_map<Key, Shape, Hash> g_shapes;

struct Limit {
  const void* kern;
  int device;
  bool operator==(const Limit& o) const { return kern == o.kern && device == o.device; }
};
struct LimitHash {
  size_t operator()(const Limit& k) const { return reinterpret_cast<size_t>(k.kern) ^ static_cast<size_t>(k.device) << 1; }
};
std::mutex g_limits_mu;
std::unordered_map<Limit, size_t, LimitHash> g_limits;

}  // namespace

// The limit belongs to the kernel, not to a launch or a thread: lowered for one launch it would
// fail another thread's, or a later one whose shape is already known. So it only ever rises.
cudaError_t allow_smem(const void* kern, size_t smem) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_limits_mu);
  size_t& limit = g_limits[Limit{kern, dev}];
  if (smem <= limit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e == cudaSuccess) limit = smem;
  return e;
}

cudaError_t kernel_shape(const void* kern, int threads, size_t smem, int* per_sm, int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const Key key{kern, smem, threads, dev};
  const auto it = g_shapes.find(key);
  if (it != g_shapes.end()) {
    *per_sm = it->second.per_sm;
    *sms = it->second.sms;
    return cudaSuccess;
  }
  Shape sh{};
  if ((e = allow_smem(kern, smem)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sh.per_sm, kern, threads, smem)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sh.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  g_shapes.emplace(key, sh);
  *per_sm = sh.per_sm;
  *sms = sh.sms;
  return cudaSuccess;
}

cudaError_t launch_kernel(const void* kern, int64_t grid, int threads, size_t smem, cudaStream_t s, void** args) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, kern, args);
}

}  // namespace cxg
