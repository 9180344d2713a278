"""CPU: the library's memory across CUDA contexts, on a stand-in for the runtime.

vd_memory.cu is compiled as host C++ against a stand-in that keeps, per device, a
context with an id and remembers which pools and pinned blocks have ended with their
context.  A context ends when its device is reset: whatever is handed out afterwards
has to belong to a living one, on every device.
"""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "voronoids_gb300", "csrc")

STAND_IN = r"""
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include "vd_common.cuh"

namespace {
unsigned long long last_id = 2, ctx_of[2] = {1, 2};  // of devices 0 and 1
int dev = 0, faults = 0, pinned_made = 0;
bool bound = true;  // the thread has a current context
std::map<void*, unsigned long long> pools, blocks, pinned;  // handle or block -> its context
bool alive(const std::map<void*, unsigned long long>& m, void* p) {
  auto i = m.find(p);
  return i != m.end() && (i->second == ctx_of[0] || i->second == ctx_of[1]);
}
CUresult ctx_get(CUcontext* c) { *c = bound ? (CUcontext)(size_t)ctx_of[dev] : nullptr; return CUDA_SUCCESS; }
CUresult ctx_id(CUcontext c, unsigned long long* id) { *id = (size_t)c; return CUDA_SUCCESS; }
}  // namespace
namespace vd { void note_launches(long long) {} }

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { dev = d; bound = true; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 1; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* q) {
  *p = (cudaMemPool_t)malloc(1);
  pools[*p] = ctx_of[q->location.id];
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) { memset(v, 0, 8); return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t mp, size_t) { if (!alive(pools, mp)) ++faults; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t mp, cudaStream_t) {
  if (!alive(pools, mp) || pools[mp] != ctx_of[dev]) { ++faults; return cudaErrorInvalidValue; }
  *p = malloc(n);
  blocks[*p] = ctx_of[dev];
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); blocks[*p] = ctx_of[dev]; return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return alive(blocks, p) ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = malloc(n);
  pinned[*p] = ctx_of[dev];
  ++pinned_made;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { if (!alive(pinned, p)) ++faults; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *f = strcmp(name, "cuCtxGetId") == 0 ? (void*)ctx_id : (void*)ctx_get;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

void on_device(int d) { dev = d; }
void unbind(void) { bound = false; }
void reset(void) { ctx_of[dev] = ++last_id; }
int fault_count(void) { return faults; }
int made_count(void) { return pinned_made; }
unsigned long long owner;
void* take(void) { return vd::pinned_alloc(&owner); }
unsigned long long taken_owner(void) { return owner; }
void give(void* p, unsigned long long c) { vd::pinned_free(p, c); }
int usable(void* p) { return alive(pinned, p) && pinned[p] == ctx_of[dev]; }
int trim(void) { return vd::pool_trim(); }
void* array(void) { return vd::pool_alloc(64, nullptr); }
void array_free(void* p) { vd::pool_free(p, nullptr); }
}
"""


@pytest.fixture()
def mem(tmp_path):
    """The stand-in and vd_memory.cu in one library, loaded anew for each test."""
    inc = [d for d in ("/usr/local/cuda/include", os.path.join(os.environ.get("CUDA_HOME", ""), "include"))
           if os.path.exists(os.path.join(d, "cuda_runtime.h"))]
    if not inc or not shutil.which("g++"):
        pytest.skip("no CUDA headers or no g++")
    src, lib = tmp_path / "stand_in.cpp", tmp_path / "memory.so"
    src.write_text(STAND_IN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", inc[0], "-I", CSRC, "-o", str(lib),
                    "-x", "c++", str(src), os.path.join(CSRC, "vd_memory.cu")], check=True)
    L = ctypes.CDLL(str(lib))
    for f in (L.take, L.array):
        f.restype = ctypes.c_void_p
    L.taken_owner.restype = ctypes.c_ulonglong
    for f in (L.usable, L.array_free):
        f.argtypes = [ctypes.c_void_p]
    L.give.argtypes = [ctypes.c_void_p, ctypes.c_ulonglong]
    return L


def test_blocks_are_used_again_within_a_context(mem):
    p = mem.take()
    mem.give(p, mem.taken_owner())
    assert mem.take() == p and mem.usable(p) and mem.made_count() == 1


def test_nothing_outlives_its_context(mem):
    for _ in range(80):  # more contexts than the library remembers
        blocks = [(mem.take(), mem.taken_owner()) for _ in range(20)]  # and more blocks than it keeps
        assert all(mem.usable(p) for p, _ in blocks)
        a = mem.array()
        assert a
        mem.array_free(a)
        for b in blocks:
            mem.give(*b)
        mem.reset()
    assert mem.fault_count() == 0


def test_a_reset_of_one_device_leaves_the_other_alone(mem):
    mem.on_device(0)
    p0, c0 = mem.take(), mem.taken_owner()
    mem.on_device(1)
    p1, c1 = mem.take(), mem.taken_owner()
    mem.give(p0, c0)  # from a thread on the other device
    mem.give(p1, c1)
    mem.on_device(0)
    mem.reset()
    mem.on_device(1)
    assert mem.take() == p1 and mem.usable(p1) and mem.array()
    mem.on_device(0)
    assert mem.usable(mem.take()) and mem.array()
    assert mem.fault_count() == 0


def test_a_block_given_back_after_its_context_ended_is_not_handed_out(mem):
    p, c = mem.take(), mem.taken_owner()
    mem.reset()
    mem.give(p, c)
    assert mem.usable(mem.take())
    assert mem.fault_count() == 0


def test_a_trim_after_a_reset_touches_nothing_dead(mem):
    p, c = mem.take(), mem.taken_owner()
    mem.give(p, c)
    assert mem.array() and mem.trim() == 0
    assert mem.usable(mem.take()) and mem.made_count() == 2  # the kept block was given back
    mem.reset()
    assert mem.trim() == 0 and mem.array() and mem.fault_count() == 0


def test_a_thread_without_a_context_gets_its_devices(mem):
    p = mem.take()
    mem.give(p, mem.taken_owner())
    mem.unbind()  # as in a new thread
    assert mem.take() == p and mem.usable(p) and mem.array() and mem.fault_count() == 0
