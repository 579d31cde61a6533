// wg_blocks.cu -- see wg_blocks.cuh.  Host code only: it compiles without the rest
// of the library, against any implementation of the runtime calls it makes.
#include <list>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "wg_blocks.cuh"

namespace wg {

namespace {

struct Block {
  void* p;
  size_t bytes;
  int dev;  // -1: page-locked host memory
};

struct Kept {
  std::mutex mu;
  std::unordered_map<void*, Block> out;  // handed out
  std::list<Block> idle;                 // kept, oldest first
  size_t idle_device = 0, idle_host = 0;
  std::vector<StreamSet> sets;
};

Kept& kept() {
  static Kept* k = new Kept();  // outlives every user of the library
  return *k;
}

int device_now() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return dev;
}

void release(const Block& b) {
  if (b.dev < 0)
    cudaFreeHost(b.p);
  else
    cudaFree(b.p);
}

// An idle block of at least `bytes` on dev, at most half as large again (or
// 64 KiB more), the tightest; true if there was one.
bool take(Kept& k, int dev, size_t bytes, Block* out) {
  std::lock_guard<std::mutex> lock(k.mu);
  auto best = k.idle.end();
  for (auto it = k.idle.begin(); it != k.idle.end(); ++it)
    if (it->dev == dev && it->bytes >= bytes && it->bytes <= bytes + bytes / 2 + (64 << 10) &&
        (best == k.idle.end() || it->bytes < best->bytes))
      best = it;
  if (best == k.idle.end()) return false;
  *out = *best;
  (dev < 0 ? k.idle_host : k.idle_device) -= best->bytes;
  k.idle.erase(best);
  k.out[out->p] = *out;
  return true;
}

// From the system; what is kept idle is given back to it if there is no room.
cudaError_t fresh(bool host, void** p, size_t bytes) {
  auto raw = [&] {
    return host ? cudaHostAlloc(p, bytes, cudaHostAllocDefault) : cudaMalloc(p, bytes);
  };
  cudaError_t e = raw();
  if (e != cudaSuccess) {
    cudaGetLastError();
    blocks_trim();
    e = raw();
  }
  return e;
}

cudaError_t alloc(int dev, void** p, size_t bytes) {
  Kept& k = kept();
  Block b;
  if (take(k, dev, bytes, &b)) {
    *p = b.p;
    return cudaSuccess;
  }
  const cudaError_t e = fresh(dev < 0, p, bytes);
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> lock(k.mu);
    k.out[*p] = Block{*p, bytes, dev};
  }
  return e;
}

bool give(void* p) {
  if (!p) return true;
  Kept& k = kept();
  std::vector<Block> drop;
  {
    std::lock_guard<std::mutex> lock(k.mu);
    const auto it = k.out.find(p);
    if (it == k.out.end()) return false;
    const Block b = it->second;
    k.out.erase(it);
    size_t& held = b.dev < 0 ? k.idle_host : k.idle_device;
    const size_t limit = b.dev < 0 ? kKeepHost : kKeepDevice;
    if (b.bytes > limit) {
      drop.push_back(b);
    } else {
      for (auto o = k.idle.begin(); o != k.idle.end() && held + b.bytes > limit;) {
        if ((o->dev < 0) == (b.dev < 0)) {
          drop.push_back(*o);
          held -= o->bytes;
          o = k.idle.erase(o);
        } else {
          ++o;
        }
      }
      k.idle.push_back(b);
      held += b.bytes;
    }
  }
  for (const Block& b : drop) release(b);
  return true;
}

}  // namespace

cudaError_t block_alloc(void** p, size_t bytes) {
  const int dev = device_now();
  if (dev < 0) return cudaErrorNoDevice;
  return alloc(dev, p, bytes);
}
void block_free(void* p) { give(p); }

cudaError_t host_block_alloc(void** p, size_t bytes) { return alloc(-1, p, bytes); }
cudaError_t host_block_free(void* p) {
  if (give(p)) return cudaSuccess;
  Kept& k = kept();
  {
    std::lock_guard<std::mutex> lock(k.mu);
    for (const Block& b : k.idle)
      if (b.p == p) return cudaErrorInvalidValue;
  }
  return cudaFreeHost(p);
}

cudaError_t device_alloc(void** p, size_t bytes) { return fresh(false, p, bytes); }
cudaError_t page_locked_alloc(void** p, size_t bytes) { return fresh(true, p, bytes); }

cudaError_t stream_set_take(StreamSet* s) {
  Kept& k = kept();
  const int dev = device_now();
  {
    std::lock_guard<std::mutex> lock(k.mu);
    for (auto it = k.sets.begin(); it != k.sets.end(); ++it)
      if (it->dev == dev) {
        *s = *it;
        k.sets.erase(it);
        return cudaSuccess;
      }
  }
  s->dev = dev;
  cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev1);
  return e;
}

void stream_set_give(const StreamSet& s) {
  if (s.stream && s.ev0 && s.ev1 && s.dev >= 0) {
    Kept& k = kept();
    std::lock_guard<std::mutex> lock(k.mu);
    if (k.sets.size() < (size_t)kKeepSets) {
      k.sets.push_back(s);
      return;
    }
  }
  if (s.ev0) cudaEventDestroy(s.ev0);
  if (s.ev1) cudaEventDestroy(s.ev1);
  if (s.stream) cudaStreamDestroy(s.stream);
}

void blocks_trim() {
  Kept& k = kept();
  std::list<Block> idle;
  std::vector<StreamSet> sets;
  {
    std::lock_guard<std::mutex> lock(k.mu);
    idle.swap(k.idle);
    sets.swap(k.sets);
    k.idle_device = k.idle_host = 0;
  }
  for (const Block& b : idle) release(b);
  for (const StreamSet& s : sets) {
    cudaEventDestroy(s.ev0);
    cudaEventDestroy(s.ev1);
    cudaStreamDestroy(s.stream);
  }
}

}  // namespace wg
