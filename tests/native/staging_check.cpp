// Check of the staging memory a context keeps (nbg_staging.hpp) with an
// allocator that counts and can refuse.  Prints "ok" and exits 0, or prints the
// first failure and exits 1.
#include <cstdio>
#include <cstdlib>

#include "nbg_staging.hpp"

static int live = 0, calls = 0;
static size_t last = 0;
static bool refuse = false;

static void* take(size_t n) {
  calls++;
  last = n;
  if (refuse) return nullptr;
  live++;
  return std::malloc(n);
}
static void give(void* p) {
  live--;
  std::free(p);
}

#define CHECK(cond)                                     \
  if (!(cond)) {                                        \
    std::printf("FAIL line %d: %s\n", __LINE__, #cond); \
    return 1;                                           \
  }

int main() {
  const size_t limit = 1 << 20;
  nbg::StagingBlock b{take, give, limit};
  unsigned char* p = b.get(100);
  CHECK(p && live == 1 && calls == 1 && last == 64 * 1024);
  CHECK(b.get(64 * 1024) == p && calls == 1);  // fits: the same block
  p = b.get(100000);
  CHECK(p && live == 1 && calls == 2 && b.bytes == 100000);  // grown, the old one given back
  CHECK(b.get(limit) && live == 1 && b.bytes == limit);
  CHECK(b.get(limit + 1) == nullptr && live == 1 && b.bytes == limit);  // over the limit: refused, the block stays
  CHECK(b.get(1) && calls == 3);
  b.free();
  CHECK(live == 0 && b.p == nullptr);
  refuse = true;
  CHECK(b.get(10) == nullptr && b.bytes == 0 && live == 0);  // a refusal is no error
  CHECK(b.get(10) == nullptr && live == 0);
  refuse = false;
  CHECK(b.get(10) && live == 1);
  b.free();
  b.free();
  CHECK(live == 0);
  std::puts("ok");
  return 0;
}
