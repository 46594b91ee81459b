// csrc/grow_buf.h over a fake allocator of limited memory.  Prints "ok", or
// the line of the first check that fails.
#include "grow_buf.h"

#include <cstdio>
#include <map>

static size_t limit, used, frees;
static std::map<void *, size_t> live;

struct FakeMem {
  static void *alloc(size_t n) {
    if (used + n > limit) return nullptr;
    void *p = ::operator new(n);
    live[p] = n;
    used += n;
    return p;
  }
  static void free(void *p) {
    used -= live.at(p);
    live.erase(p);
    ::operator delete(p);
    frees++;
  }
};
using Buf = bz2g::GrowBuf<FakeMem>;

#define CHECK(x)                    \
  if (!(x)) {                       \
    std::printf("%d\n", __LINE__);  \
    return 1;                       \
  }

int main() {
  limit = 1000;
  Buf a, b, spare;
  CHECK(a.try_reserve(100) && a.cap == 100 && used == 100);
  CHECK(a.try_reserve(50) && a.cap == 100 && frees == 0);  // large enough
  CHECK(spare.try_reserve(600));
  // refused: a call can do without the spare, so it is no error, and nothing is held
  CHECK(!spare.try_reserve(2000) && spare.p == nullptr && spare.cap == 0 && used == 100);
  CHECK(spare.try_reserve(600));
  // what others need is taken from the spare
  CHECK(reserve_or_free(b, 700, spare) && b.cap == 700 && spare.cap == 0 && used == 800);
  // and where that is not enough, the call fails with nothing lost but the buffer
  CHECK(!reserve_or_free(b, 950, spare) && b.cap == 0 && a.cap == 100);
  CHECK(spare.try_reserve(300) && !reserve_or_free(b, 950, spare) && spare.cap == 0);
  CHECK(reserve_or_free(b, 900, spare) && used == 1000);
  CHECK(!reserve_or_free(spare, 10, spare));  // the spare itself gives nothing up
  a.release();
  b.release();
  CHECK(used == 0 && live.empty());
  std::printf("ok\n");
}
