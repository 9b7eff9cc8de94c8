// Preloaded over operator new: while `fail_new` is set, every allocation fails as if memory had run out.
#include <cstdlib>
#include <new>

extern "C" {
volatile int fail_new = 0;
volatile int failed = 0;
}
void* operator new(std::size_t n) {
  if (fail_new) {
    failed = failed + 1;
    throw std::bad_alloc();
  }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
