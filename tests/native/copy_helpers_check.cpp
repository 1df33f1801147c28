// Host-side check of the serving loop's copy helpers (copy_helpers.h): every
// copy is made before run returns, with several callers at once, with fewer
// threads than asked for, and without memory to share them; nothing is thrown.
// Built and run by tests/test_copy_helpers_host.py; prints "ok".
#include <sys/resource.h>
#include <unistd.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <new>

#include "copy_helpers.h"

static thread_local bool no_memory = false;
void* operator new(size_t n) {
  void* p = no_memory ? nullptr : malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

using ighost::CopyHelpers;
static int fails = 0;
#define CHECK(c)                                       \
  do {                                                 \
    if (!(c)) {                                        \
      std::printf("FAIL line %d: %s\n", __LINE__, #c); \
      fails++;                                         \
    }                                                  \
  } while (0)

constexpr size_t BYTES = 4096;

static bool copies_right(CopyHelpers& h, size_t n, uint8_t salt, bool starve = false) {
  std::vector<uint8_t> from(n * BYTES), to(n * BYTES, 0);
  for (size_t i = 0; i < from.size(); i++) from[i] = (uint8_t)(i * 31 + i / BYTES + salt);
  std::vector<CopyHelpers::Copy> copies;
  for (size_t i = 0; i < n; i++) copies.push_back({&to[i * BYTES], &from[i * BYTES]});
  no_memory = starve;
  bool thrown = false;
  try {
    h.run(copies, BYTES);
  } catch (...) {
    thrown = true;
  }
  no_memory = false;
  return !thrown && from == to;
}

int main() {
  const size_t M = CopyHelpers::MIN_COPIES;
  {
    // no room for a thread's stack: none starts, the copies are made all the same
    long pages = 0;
    FILE* f = std::fopen("/proc/self/statm", "r");
    CHECK(f && std::fscanf(f, "%ld", &pages) == 1);
    if (f) std::fclose(f);
    rlimit old, tight;
    getrlimit(RLIMIT_AS, &old);
    tight = old;
    tight.rlim_cur = (rlim_t)pages * (rlim_t)sysconf(_SC_PAGESIZE) + (2u << 20);
    CHECK(setrlimit(RLIMIT_AS, &tight) == 0);
    {
      CopyHelpers h;
      bool thrown = false;
      try {
        h.start(8);
      } catch (...) {
        thrown = true;
      }
      CHECK(!thrown && h.threads() == 0);
      CHECK(copies_right(h, 3 * M, 1));
    }
    setrlimit(RLIMIT_AS, &old);
  }
  {
    CopyHelpers h;
    h.start(8);
    CHECK(h.threads() == 8);
    for (size_t n : {(size_t)0, (size_t)1, M - 1, M, 8 * M}) CHECK(copies_right(h, n, 2));
    CHECK(copies_right(h, 8 * M, 3, true));  // no memory for the job
    CHECK(copies_right(h, 8 * M, 4));
    std::atomic<int> bad{0};
    std::vector<std::thread> callers;
    for (int t = 0; t < 4; t++)
      callers.emplace_back([&, t] {
        for (int k = 0; k < 50; k++) bad += !copies_right(h, M + 7 * k % 40, (uint8_t)(t * 50 + k), k % 5 == 0);
      });
    for (std::thread& t : callers) t.join();
    CHECK(bad == 0);
  }
  if (fails) return 1;
  std::printf("ok\n");
  return 0;
}
