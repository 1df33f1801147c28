// Host-side check of the choice between the one-CTA Respond kernel's two forms
// (batch_policy.h).  Built and run by tests/test_batch_policy_host.py; prints "ok".
#include <cstdio>

#include "batch_policy.h"

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
  int asked = 0;
  auto runs = [&] { return asked++, false; };
  auto ended = [&] { return asked++, true; };

  CHECK(alone_limit(152, false, LastBatch{}, 7, runs) == 152 && asked == 0);       // none before
  const LastBatch last{true, 7};
  CHECK(alone_limit(152, false, last, 7, runs) == 152 && asked == 0);              // its own stream: it ends first
  CHECK(alone_limit(152, false, last, 8, runs) == 0 && asked == 1);                // another stream, still running
  CHECK(alone_limit(152, false, last, 8, ended) == 152 && asked == 2);
  CHECK(alone_limit(152, true, last, 7, ended) == 0 && asked == 2);                // captured: no query either
  CHECK(alone_limit(152, true, LastBatch{}, 7, ended) == 0 && asked == 2);
  CHECK(alone_limit(152, false, LastBatch{true, 0}, 8, runs) == 0);                // id 0 is an id like any other

  // whole rows: few columns, more queries than SMs
  CHECK(whole_rows(1, 153, 152) && whole_rows(4, 153, 152) && whole_rows(2, 0xFFFFFFFFu, 152));
  CHECK(!whole_rows(1, 152, 152) && !whole_rows(8, 153, 152) && !whole_rows(16, 5000, 152));

  if (fails) return 1;
  std::printf("ok\n");
  return 0;
}
