// A stand-in for the parts of the CUDA runtime that the library's host-only files use: two
// devices of 1 GB, host memory for device memory, and a log of the calls that matter. The
// tests build those files against it (tests/test_host_runtime.py), so the order of calls and
// the answers to failing ones are checked without a GPU.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <map>
#include <string>

namespace cxg {
cudaError_t device_alloc(void** out, size_t bytes);
cudaError_t device_malloc(void** out, size_t bytes);
void device_free(void* ptr);
void device_free_all(int device, void* const* blocks, int n);
bool kernel_reads(int device, const void* ptr);
cudaError_t kernel_shape(const void* kern, int threads, size_t smem, int* per_sm, int* sms);
cudaError_t launch_kernel(const void* kern, int64_t grid, int threads, size_t smem, cudaStream_t s, void** args);
}  // namespace cxg

namespace {

constexpr size_t kDevice = size_t{1} << 30;

struct Block {
  int device;
  size_t bytes;
  bool pooled;
};
int g_device = 0;
size_t g_used[2] = {0, 0}, g_idle[2] = {0, 0};  // in use, and kept by the device's pool
std::map<void*, Block> g_blocks;
std::map<std::pair<const void*, int>, int> g_limit;
std::string g_log;

void note(const std::string& s) { g_log += s + "@" + std::to_string(g_device) + " "; }

cudaError_t take(void** p, size_t bytes, bool pooled) {
  const size_t idle = pooled ? std::min(g_idle[g_device], bytes) : 0;  // reused first
  if (g_used[g_device] + g_idle[g_device] - idle + bytes > kDevice) return cudaErrorMemoryAllocation;
  g_idle[g_device] -= idle;
  g_used[g_device] += bytes;
  *p = std::malloc(16);
  g_blocks[*p] = {g_device, bytes, pooled};
  return cudaSuccess;
}

}  // namespace

extern "C" {

cudaError_t cudaGetDevice(int* d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  g_device = d;
  note("set");
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return note("wait"), cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return note("malloc"), take(p, n, false); }
cudaError_t cudaFree(void* p) {
  note("free");
  g_used[g_blocks[p].device] -= g_blocks[p].bytes;
  g_blocks.erase(p);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(static_cast<size_t>(g_device + 1)), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* m, const cudaMemPoolProps* p) {
  return *m = reinterpret_cast<cudaMemPool_t>(static_cast<size_t>(p->location.id + 1)), cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return note("pool"), take(p, n, true); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return note("async"), take(p, n, false); }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) {
  note("trim");
  g_idle[g_device] = 0;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  note("give");
  const Block b = g_blocks[p];
  if (s != reinterpret_cast<cudaStream_t>(static_cast<size_t>(b.device + 1))) note("WRONG-POOL");
  g_used[b.device] -= b.bytes;
  g_idle[b.device] += b.bytes;
  g_blocks.erase(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void* p) {
  auto b = g_blocks.upper_bound(const_cast<void*>(p));
  *at = {};
  if (b == g_blocks.begin() || static_cast<const char*>(p) >= static_cast<char*>((--b)->first) + 16) return cudaErrorInvalidValue;
  at->type = cudaMemoryTypeDevice;
  at->device = b->second.device;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* kern, cudaFuncAttribute, int n) {
  note("limit" + std::to_string(n));
  g_limit[{kern, g_device}] = n;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { return *s = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kern, void**) {
  if (c->dynamicSmemBytes <= static_cast<size_t>(g_limit[{kern, g_device}])) return note("launch"), cudaSuccess;
  return note("refused"), cudaErrorInvalidValue;
}

// ---- what the tests call
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
int t_alloc(void** p, size_t n) { return cxg::device_alloc(p, n); }
int t_malloc(void** p, size_t n) { return cxg::device_malloc(p, n); }
void t_free(void* p) { cxg::device_free(p); }
void t_free_all(int device, void* const* p, int n) { cxg::device_free_all(device, p, n); }
int t_kernel_reads(int device, const void* p) { return cxg::kernel_reads(device, p); }
int t_shape(const void* kern, size_t smem) {
  int per_sm, sms;
  return cxg::kernel_shape(kern, 128, smem, &per_sm, &sms);
}
int t_launch(const void* kern, size_t smem) { return cxg::launch_kernel(kern, 1, 128, smem, nullptr, nullptr); }

}  // extern "C"
