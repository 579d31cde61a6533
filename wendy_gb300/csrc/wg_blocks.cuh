// wg_blocks.cuh -- device and page-locked memory, streams and events kept from
// one simulation for the next.
//
// Setting up and tearing down a simulation took five device and five
// page-locked allocations, a stream and two events, and as many releases,
// each release waiting for the device: 0.6 ms for a hundred sheets, 3 ms for
// 1e6, against 0.1 ms of device time for a force evaluation.  What a simulation
// releases is kept here, up to kKeepDevice and kKeepHost bytes and kKeepSets
// streams per process, oldest dropped first, and handed to the next one that
// asks for it.  It is given back to the system when an allocation of the
// library fails, when the free memory is asked for, and by blocks_trim() (wg_trim
// for other users of the device's memory in the process).
// Callers hand back only memory and streams with no work in flight, so that
// nothing depends on the stream that used them last.  All functions may be
// called from several threads.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace wg {

constexpr size_t kKeepDevice = (size_t)512 << 20;
constexpr size_t kKeepHost = (size_t)64 << 20;
constexpr int kKeepSets = 8;

// Device memory on the current device.  Contents are undefined.
cudaError_t block_alloc(void** p, size_t bytes);
void block_free(void* p);
template <typename T>
cudaError_t block_alloc(T** p, size_t bytes) {
  return block_alloc(reinterpret_cast<void**>(p), bytes);
}

// Page-locked host memory.
cudaError_t host_block_alloc(void** p, size_t bytes);
// An error if p was released already; memory page-locked by others is released as
// cudaFreeHost does.
cudaError_t host_block_free(void* p);
template <typename T>
cudaError_t host_block_alloc(T** p, size_t bytes) {
  return host_block_alloc(reinterpret_cast<void**>(p), bytes);
}

// cudaMalloc and cudaMallocHost for memory that is not handed on (released with
// cudaFree and cudaFreeHost): what is kept idle is given back before they fail.
cudaError_t device_alloc(void** p, size_t bytes);
cudaError_t page_locked_alloc(void** p, size_t bytes);
template <typename T>
cudaError_t device_alloc(T** p, size_t bytes) {
  return device_alloc(reinterpret_cast<void**>(p), bytes);
}
template <typename T>
cudaError_t page_locked_alloc(T** p, size_t bytes) {
  return page_locked_alloc(reinterpret_cast<void**>(p), bytes);
}

// A non-blocking stream and two timing events, of the device that is current
// when they are taken (they may be given back from any other).
struct StreamSet {
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int dev = -1;
};
cudaError_t stream_set_take(StreamSet* s);
void stream_set_give(const StreamSet& s);

// Gives everything kept back to the system.
void blocks_trim();

}  // namespace wg
