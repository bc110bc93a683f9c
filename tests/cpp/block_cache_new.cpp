// operator new for block_cache.cu, which fails while g_no_memory is set.
#include <cstdlib>
#include <new>

bool g_no_memory = false;

void* operator new(std::size_t n) {
  void* p = g_no_memory ? nullptr : std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
