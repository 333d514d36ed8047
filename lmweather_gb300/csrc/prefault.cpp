#include "prefault.h"

#include <algorithm>
#include <cstdint>
#include <thread>
#ifdef __linux__
#include <sys/mman.h>
#include <unistd.h>
#endif

namespace lmw {

void prefault(void *p, size_t bytes) noexcept {
#ifdef __linux__
  constexpr size_t kLeast = 1 << 20;
  if (bytes < kLeast) return;
  const size_t page = static_cast<size_t>(sysconf(_SC_PAGESIZE));
  const uintptr_t a = reinterpret_cast<uintptr_t>(p) / page * page, e = reinterpret_cast<uintptr_t>(p) + bytes;
  unsigned char first = 1, last = 1;
  if (mincore(reinterpret_cast<void *>(a), 1, &first) != 0 || mincore(reinterpret_cast<void *>((e - 1) / page * page), 1, &last) != 0) return;
  const uintptr_t mid = (a + (e - a) / 2) / page * page;
  unsigned char half = 1;
  if (mincore(reinterpret_cast<void *>(mid), 1, &half) != 0 || ((first & last & half) & 1)) return;
  constexpr int kPopulateWrite = 23;  // MADV_POPULATE_WRITE (Linux 5.14); where it is unknown the copy faults the pages
  auto fill = [=](uintptr_t from, uintptr_t to) {
    if (to > from) madvise(reinterpret_cast<void *>(from), to - from, kPopulateWrite);
  };
  const int parts = bytes >= 8 * kLeast ? 4 : 1;
  const uintptr_t len = ((e - a) / parts + page - 1) / page * page;
  std::thread others[3];
  try {
    for (int k = 1; k < parts; k++) others[k - 1] = std::thread(fill, std::min(a + k * len, e), std::min(a + (k + 1) * len, e));
  } catch (...) {  // no thread (std::system_error) or no memory for one (std::bad_alloc)
  }
  fill(a, std::min(a + len, e));
  for (auto &t : others)
    if (t.joinable()) t.join();
#else
  (void)p;
  (void)bytes;
#endif
}

}  // namespace lmw
