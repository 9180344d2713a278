// Device and pinned host memory of the library's trees.
//
// A tree is about 40 device arrays.  cudaMalloc and cudaFree took 10 to 60 us
// each, 1.3 ms of the 2.4 ms of a one-shot call on 200 points, so the arrays come
// from a stream-ordered pool per device: what one tree gives back the next one
// takes, from any thread and on any stream (the pool orders a block's reuse after
// its free).  Up to kKeepBytes of free memory stay with the pool; the rest goes
// back to the device at the next synchronisation, and all of it when an
// allocation fails.  Pinned blocks are kept in a short list.
#include <cuda_runtime.h>

#include <mutex>

#include "vd_common.cuh"

namespace vd {
namespace {

constexpr unsigned long long kKeepBytes = 512ull << 20;
constexpr int kMaxDevices = 64;
constexpr int kPinnedKept = 16;

std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};
int g_state[kMaxDevices] = {};  // 0 not asked yet, 1 pool, -1 none (plain allocations)
void* g_pinned[kPinnedKept] = {};
int g_npinned = 0;

// The current device's pool, null where there is none.
cudaMemPool_t pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_mu);
  if (g_state[dev] == 0) {
    int has = 0;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = kKeepBytes;
    if (cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && has &&
        cudaMemPoolCreate(&g_pool[dev], &props) == cudaSuccess &&
        cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) {
      g_state[dev] = 1;
    } else {
      cudaGetLastError();
      g_pool[dev] = nullptr;
      g_state[dev] = -1;
    }
  }
  return g_pool[dev];
}

}  // namespace

void* pool_alloc(size_t bytes, cudaStream_t st) {
  void* p = nullptr;
  cudaMemPool_t mp = pool();
  if (!mp) {
    if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
  }
  if (cudaMallocFromPoolAsync(&p, bytes, mp, st) == cudaSuccess) return p;
  // what finished work has freed goes back to the device, then once more
  cudaGetLastError();
  cudaStreamSynchronize(st);
  cudaMemPoolTrimTo(mp, 0);
  if (cudaMallocFromPoolAsync(&p, bytes, mp, st) == cudaSuccess) return p;
  cudaGetLastError();
  return nullptr;
}

void pool_free(void* p, cudaStream_t st) {
  if (!p) return;
  if (pool() && cudaFreeAsync(p, st) == cudaSuccess) return;
  cudaGetLastError();
  cudaFree(p);  // waits for the device
}

void* pinned_alloc() {
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (g_npinned > 0) return g_pinned[--g_npinned];
  }
  void* p = nullptr;
  if (cudaMallocHost(&p, kPinnedBytes) == cudaSuccess) return p;
  cudaGetLastError();
  return nullptr;
}

void pinned_free(void* p) {
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (g_npinned < kPinnedKept) {
      g_pinned[g_npinned++] = p;
      return;
    }
  }
  cudaFreeHost(p);
}

}  // namespace vd
