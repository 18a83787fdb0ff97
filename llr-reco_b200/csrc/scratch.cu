// Per-call device scratch of the stand-alone operators (batched prox, signal model, wavelet shrink,
// hard projection, DTI fit), stream-ordered from one private memory pool per device.
//
// The device's default pool gives its memory back to the driver at every synchronisation (release
// threshold 0), so an operator that allocated there mapped fresh pages on each call: the DTI fit's
// 2 KB table made a 0.62 ms call take 1.0-2.9 ms.  The private pool keeps at most kKeepBytes of
// unused memory mapped (kKeepMost once a call has asked for it, see scratch_keep); what is above it goes
// back at the next synchronisation, all of it when a context or a network is destroyed, when a caller of the
// operators alone asks for it (llr_device_free of a null pointer), or when an allocation of the library
// runs out of memory.
// Allocation and free are stream-ordered, so calls on several streams and threads never share a
// block at the same time.
#include <mutex>

#include "llr_internal.h"

namespace llr {

namespace {

constexpr int kMaxDevices = 64;
// The Gram scratch of 16384 blocks of 61 columns (248 MB, a 192 x 192 x 96 volume in 6^3 blocks)
// stays mapped between calls; below 0.2 % of the device's memory.
constexpr unsigned long long kKeepBytes = 256ull << 20;
constexpr unsigned long long kKeepMost = 768ull << 20;

std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices];
unsigned long long g_keep[kMaxDevices];

// The pool of the stream's device, created on first use; null when there is none (the caller
// then takes the default pool).
cudaMemPool_t pool_of(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_pool[dev]) return g_pool[dev];
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t p = nullptr;
  if (cudaMemPoolCreate(&p, &props) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  unsigned long long keep = kKeepBytes;
  if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) cudaGetLastError();
  g_pool[dev] = p;
  g_keep[dev] = keep;
  return p;
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  if (bytes == 0) bytes = 16;
  // Under capture the allocation becomes a node of the caller's graph, which owns the memory.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  int dev = -1;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
      cudaStreamGetDevice(s, &dev) != cudaSuccess) {
    cudaGetLastError();
    return cudaMallocAsync(p, bytes, s);
  }
  cudaMemPool_t pool = pool_of(dev);
  if (!pool) return cudaMallocAsync(p, bytes, s);
  cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, s);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    cudaStreamSynchronize(s);
    cudaMemPoolTrimTo(pool, 0);
    e = cudaMallocFromPoolAsync(p, bytes, pool, s);
  }
  return e;
}

void scratch_keep(size_t bytes, cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  int dev = -1;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
      cudaStreamGetDevice(s, &dev) != cudaSuccess || !pool_of(dev)) {
    cudaGetLastError();
    return;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  unsigned long long keep = bytes < kKeepMost ? bytes : kKeepMost;
  if (keep <= g_keep[dev]) return;
  if (cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) g_keep[dev] = keep;
  else cudaGetLastError();
}

void scratch_trim() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_pool[dev]) cudaMemPoolTrimTo(g_pool[dev], 0);
}

cudaError_t device_alloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  scratch_trim();
  return cudaMalloc(p, bytes ? bytes : 16);
}

}  // namespace llr
