// Test infrastructure only: the stand-in CUDA runtime (stub_cudart.cpp) with host
// allocations that can be made to fail inside parallel regions.
#include "stub_cudart.cpp"

#include <new>
#include <omp.h>

namespace {
std::atomic<int> g_team_nomem{0};
}

extern "C" void stub_cudart_team_nomem(int on) { g_team_nomem = on; }

void *operator new(std::size_t n) {
  if (g_team_nomem.load() && omp_in_parallel()) throw std::bad_alloc();
  if (void *p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void *operator new[](std::size_t n) { return operator new(n); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
void operator delete[](void *p) noexcept { std::free(p); }
void operator delete[](void *p, std::size_t) noexcept { std::free(p); }
