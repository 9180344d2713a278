// Device and pinned host memory of the library's trees.
//
// A tree is about 40 device arrays.  cudaMalloc and cudaFree took 10 to 60 us
// each, 1.3 ms of the 2.4 ms of a one-shot call on 200 points, so the arrays come
// from a stream-ordered pool: what one tree gives back the next one takes, from
// any thread and on any stream (the pool orders a block's reuse after its free).
// Up to kKeepBytes of free memory stay with the pool; the rest goes back to the
// device at the next synchronisation (a tree that is freed makes one), and all of
// it when an allocation fails or the caller asks (vd_trim_memory).  Pinned blocks
// are kept in a short list.
//
// Pool and list belong to a CUDA context and end with it (cudaDeviceReset, or a
// device's primary context given up by all of its users), so they are looked up
// by the current context's id, which no later context has again.  A context that
// is not met any more costs its entry here and nothing else.
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "vd_common.cuh"

namespace vd {
namespace {

constexpr unsigned long long kKeepBytes = 512ull << 20;
constexpr int kContexts = 32;
constexpr int kPinnedKept = 16;

struct ContextMemory {
  unsigned long long id;  // 0: entry not in use
  cudaMemPool_t pool;     // null where there is none (plain allocations)
  void* pinned[kPinnedKept];
  int npinned;
};
std::mutex g_mu;
ContextMemory g_mem[kContexts] = {};
int g_next = 0;  // entry that the next new context takes
std::atomic<bool> g_plain{false};  // some block came from cudaMalloc

typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long*);

ContextMemory* entry_of(unsigned long long id) {  // g_mu held
  for (int i = 0; i < kContexts && id != 0; ++i)
    if (g_mem[i].id == id) return &g_mem[i];
  return nullptr;
}

// The current context's entry, made when it is met first; null without a context
// (then allocations are plain).  g_mu held.
ContextMemory* current_entry() {
  unsigned long long id = context_id();
  int dev = 0, has = 0;
  if (id == 0 && cudaGetDevice(&dev) == cudaSuccess) {
    cudaSetDevice(dev);  // a thread's first call: binds its device's context (other threads may be capturing)
    id = context_id();
  }
  if (id == 0) return nullptr;
  if (ContextMemory* e = entry_of(id)) return e;
  ContextMemory& e = g_mem[g_next];
  g_next = (g_next + 1) % kContexts;
  e = ContextMemory{};
  cudaMemPoolProps props = {};
  unsigned long long keep = kKeepBytes;
  if (cudaGetDevice(&dev) == cudaSuccess) {
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess || !has ||
        cudaMemPoolCreate(&e.pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(e.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
      cudaGetLastError();
      e.pool = nullptr;
    }
  }
  e.id = id;
  return &e;
}

// The current context's pool, null where there is none.
cudaMemPool_t pool() {
  std::lock_guard<std::mutex> lock(g_mu);
  const ContextMemory* e = current_entry();
  return e ? e->pool : nullptr;
}

}  // namespace

// Context ids come from the driver API (cuCtxGetCurrent, cuCtxGetId), reached
// through the runtime's driver entry points so that the library needs no libcuda
// link.
unsigned long long context_id() {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(f);
  });
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
    return 0;
  return id;
}

void* pool_alloc(size_t bytes, cudaStream_t st) {
  void* p = nullptr;
  cudaMemPool_t mp = pool();
  if (!mp) {
    g_plain = true;
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
  // (looking up the context of each block freed was 0.5 % of a call on 200 points)
  if ((!g_plain || pool()) && cudaFreeAsync(p, st) == cudaSuccess) return;
  cudaGetLastError();
  cudaFree(p);  // waits for the device
}

int pool_trim() {
  std::lock_guard<std::mutex> lock(g_mu);
  ContextMemory* e = current_entry();
  if (!e) return E_OK;  // nothing is kept without a context
  if (cudaDeviceSynchronize() != cudaSuccess) return E_CUDA;  // frees still in their streams
  while (e->npinned > 0) cudaFreeHost(e->pinned[--e->npinned]);
  return e->pool && cudaMemPoolTrimTo(e->pool, 0) != cudaSuccess ? E_CUDA : E_OK;
}

void* pinned_alloc(unsigned long long* context) {
  {
    std::lock_guard<std::mutex> lock(g_mu);
    ContextMemory* e = current_entry();
    *context = e ? e->id : 0;
    if (e && e->npinned > 0) return e->pinned[--e->npinned];
  }
  void* p = nullptr;
  if (cudaMallocHost(&p, kPinnedBytes) == cudaSuccess) return p;
  cudaGetLastError();
  return nullptr;
}

void pinned_free(void* p, unsigned long long context) {
  {
    std::lock_guard<std::mutex> lock(g_mu);
    ContextMemory* e = entry_of(context);
    if (e && e->npinned < kPinnedKept) {
      e->pinned[e->npinned++] = p;
      return;
    }
  }
  // a block of another context than the current one may be gone with its
  // context, and its address in use again: it is left alone
  if (context == 0 || context == context_id()) cudaFreeHost(p);
}

}  // namespace vd
