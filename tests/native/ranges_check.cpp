// Host-side check of the conditions under which a batch's rows and responses
// are read and written in place (ranges.h).  Built and run by
// tests/test_ranges_host.py; prints "ok".
#include <cstdio>

#include "ranges.h"

static int fails = 0;
#define CHECK(c)                                       \
  do {                                                 \
    if (!(c)) {                                        \
      std::printf("FAIL line %d: %s\n", __LINE__, #c); \
      fails++;                                         \
    }                                                  \
  } while (0)

int main() {
  using namespace ighost;
  const char* p = reinterpret_cast<const char*>((uintptr_t)1 << 20);

  CHECK(!overlap(p, 16, p + 16, 16) && !overlap(p + 16, 16, p, 16));  // neighbours
  CHECK(overlap(p, 17, p + 16, 16) && overlap(p + 16, 16, p, 17));    // one byte
  CHECK(overlap(p, 64, p + 16, 8) && overlap(p + 16, 8, p, 64));      // one inside the other
  CHECK(overlap(p, 1, p, 1) && !overlap(p, 0, p, 16) && !overlap(p, 16, p + 8, 0));
  const char* top = reinterpret_cast<const char*>(UINTPTR_MAX - 15);  // ends at the last address
  CHECK(overlap(top, 16, top + 15, 1) && !overlap(top, 16, p, 16));

  CHECK(rows_and_out_in_place(p, 4096, p + 4096, 4096));
  CHECK(rows_and_out_in_place(p + 4096, 4096, p, 4096));
  CHECK(rows_and_out_in_place(p, 4096, p + 4104, 64));      // responses on any 64-bit word
  CHECK(!rows_and_out_in_place(p, 4096, p + 4100, 64));     // 4-byte aligned responses
  CHECK(!rows_and_out_in_place(p + 8, 4096, p + 8192, 64)); // rows off their 16 bytes
  CHECK(!rows_and_out_in_place(p, 4096, p + 4088, 64));     // the last row's last word
  CHECK(!rows_and_out_in_place(p, 4096, p, 64));

  if (fails) return 1;
  std::printf("ok\n");
  return 0;
}
