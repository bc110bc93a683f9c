// A buffer that is destroyed while the host has no memory left goes back to its pool and ends
// no process.  Runs without a GPU: the device call it ends in reports an error, which is dropped.
#include <cstdio>

#include "common.cuh"

extern bool g_no_memory;  // operator new fails (block_cache_new.cpp)

namespace femgpu {
thread_local cudaMemPool_t g_alloc_pool = nullptr;
thread_local BlockCache* g_alloc_cache = nullptr;
}  // namespace femgpu

int main() {
  femgpu::BlockCache cache;
  {
    femgpu::DBuf<int> buf;  // as an allocation of 1000 ints leaves it
    buf.p = reinterpret_cast<int*>(256);
    buf.n = 1000;
    buf.cache = &cache;
    buf.cls = femgpu::BlockCache::class_of(4000);
    g_no_memory = true;
  }
  g_no_memory = false;
  if (cache.bytes != 0 || !cache.kept[femgpu::BlockCache::class_of(4000)].empty()) return 1;
  std::puts("ok");
  return 0;
}
