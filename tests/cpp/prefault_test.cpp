// csrc/prefault.cpp where memory runs out: the n-th allocation that it makes fails, for every n. Prints how many calls came
// back, how many threw, and how many bytes they changed.
#include <sys/mman.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include "prefault.h"

static int left = -1;  // allocations until one fails (negative: none does)
void *operator new(std::size_t n) {
  if (left == 0) throw std::bad_alloc();
  if (left > 0) left--;
  if (void *p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main() {
  const size_t bytes = 24u << 20;
  int calls = 0, threw = 0, changed = 0;
  for (int n = -1; n < 12; n++) {
    char *p = static_cast<char *>(mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (p == MAP_FAILED) return 1;
    p[bytes / 3] = 7;
    left = n;
    try {
      lmw::prefault(p + 5, bytes - 9);
      calls++;
    } catch (...) {
      threw++;
    }
    left = -1;
    for (size_t i = 0; i < bytes; i += 4096) changed += p[i] != (i == bytes / 3 ? 7 : 0) ? 1 : 0;
    munmap(p, bytes);
  }
  std::printf("%d %d %d\n", calls, threw, changed);
  return 0;
}
