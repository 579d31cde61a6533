"""What the library keeps from one simulation for the next (wendy_gb300/csrc/
wg_blocks.cu, host code): compiled here against a stand-in for the CUDA runtime
with two devices and an allocator that can be made to fail."""
import ctypes.util
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "wendy_gb300", "csrc")

RUNTIME = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include "wg_blocks.cuh"
using namespace wg;
static int now = 0;             // the current device
static size_t room = 1u << 30;  // bytes that can still be allocated
static std::set<void*> live;
static size_t size_of(void* p) { return *static_cast<size_t*>(p); }
static cudaError_t get(void** p, size_t b) {
  if (b > room) return cudaErrorMemoryAllocation;
  room -= b;
  *p = malloc(sizeof(size_t));
  *static_cast<size_t*>(*p) = b;
  live.insert(*p);
  return cudaSuccess;
}
static cudaError_t put(void* p) {
  room += size_of(p);
  live.erase(p);
  free(p);
  return cudaSuccess;
}
struct Handle { int dev; };
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = now; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t b) { return get(p, b); }
cudaError_t cudaFree(void* p) { return put(p); }
cudaError_t cudaHostAlloc(void** p, size_t b, unsigned) { return get(p, b); }
cudaError_t cudaFreeHost(void* p) { return put(p); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(new Handle{now});
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(new Handle{now});
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}
template <typename T>
static int device_of(T h) { return reinterpret_cast<Handle*>(h)->dev; }
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
"""

STREAMS = r"""
int main() {
  // made on device 0, given back while device 1 is current: the next user of
  // device 1 gets streams of its own device, the next of device 0 these again
  StreamSet a, b, c;
  CHECK(stream_set_take(&a) == cudaSuccess);
  now = 1;
  stream_set_give(a);
  CHECK(stream_set_take(&b) == cudaSuccess);
  CHECK(device_of(b.stream) == 1 && device_of(b.ev0) == 1 && device_of(b.ev1) == 1);
  now = 0;
  CHECK(stream_set_take(&c) == cudaSuccess);
  CHECK(c.stream == a.stream && device_of(c.ev0) == 0);
  return 0;
}
"""

ROOM = r"""
int main() {
  // a closed simulation's memory is all the device has: every kind of allocation
  // takes it back before it fails
  const size_t most = (size_t)400 << 20;
  room = most;
  void* p = nullptr;
  for (int k = 0; k < 4; ++k) {
    CHECK(block_alloc(&p, most - 1000) == cudaSuccess);
    block_free(p);
    CHECK(room == 1000 && live.size() == 1);  // kept
    if (k == 0) CHECK(device_alloc(&p, 2000) == cudaSuccess && cudaFree(p) == cudaSuccess);
    if (k == 1) CHECK(page_locked_alloc(&p, 2000) == cudaSuccess && cudaFreeHost(p) == cudaSuccess);
    if (k == 2) CHECK(host_block_alloc(&p, 2000) == cudaSuccess && host_block_free(p) == cudaSuccess);
    if (k == 3) blocks_trim();
    blocks_trim();
    CHECK(room == most && live.empty());
  }
  CHECK(device_alloc(&p, most + 1) == cudaErrorMemoryAllocation);
  return 0;
}
"""

TWICE = r"""
int main() {
  // a second release is refused, and what is kept stays intact
  void *p = nullptr, *q = nullptr;
  CHECK(host_block_alloc(&p, 5000) == cudaSuccess);
  CHECK(host_block_free(p) == cudaSuccess);
  CHECK(host_block_free(p) != cudaSuccess && live.count(p) == 1);
  CHECK(host_block_alloc(&q, 5000) == cudaSuccess && q == p);
  void* other = nullptr;
  CHECK(cudaHostAlloc(&other, 5000, 0) == cudaSuccess);
  CHECK(host_block_free(other) == cudaSuccess && live.count(other) == 0);
  CHECK(host_block_free(q) == cudaSuccess && host_block_free(nullptr) == cudaSuccess);
  return 0;
}
"""


def _run(tmp_path, main):
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "kept.cpp", tmp_path / "kept"
    src.write_text(RUNTIME + main)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(cuda, "include"),
                    "-x", "c++", os.path.join(CSRC, "wg_blocks.cu"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_streams_stay_with_their_device(tmp_path):
    _run(tmp_path, STREAMS)


def test_kept_memory_is_given_back_before_an_allocation_fails(tmp_path):
    _run(tmp_path, ROOM)


def test_a_second_release_is_refused(tmp_path):
    _run(tmp_path, TWICE)


def test_no_source_allocates_past_what_is_kept():
    # wg_blocks.cu alone calls the allocators that fail while memory is kept idle
    for f in sorted(os.listdir(CSRC)):
        if f != "wg_blocks.cu" and f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as src:
                code = [line.split("//")[0] for line in src]
            assert not [c for c in code
                        if re.search(r"\bcuda(Malloc|MallocHost|HostAlloc)\(", c)], f


@pytest.mark.gpu
def test_trim_gives_the_memory_of_closed_simulations_back():
    import ctypes

    import wendy_gb300
    from wendy_gb300 import ics
    rt = ctypes.CDLL(ctypes.util.find_library("cudart") or "libcudart.so")
    rt.cudaMemGetInfo.argtypes = [ctypes.POINTER(ctypes.c_size_t)] * 2

    def free_bytes():
        f, t = ctypes.c_size_t(), ctypes.c_size_t()
        assert rt.cudaMemGetInfo(ctypes.byref(f), ctypes.byref(t)) == 0
        return f.value

    x, v, m = ics.sech2_disk(1 << 20, seed=1)
    wendy_gb300.Simulation(x, v, m, 1., -1.).close()
    kept = free_bytes()
    wendy_gb300.trim()
    assert free_bytes() >= kept + (100 << 20)
