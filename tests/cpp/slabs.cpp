// Prints slab_count of csrc/slabs.h for tests/test_slabs_cpu.py: per line of
// "blocks bytes workers on_device" read from the input.
#include <cstdio>

#include "slabs.h"

int main() {
  long long nb, bytes;
  int workers, dev;
  while (std::scanf("%lld %lld %d %d", &nb, &bytes, &workers, &dev) == 4)
    std::printf("%d\n", bz2g::slab_count((int)nb, bytes, workers, dev != 0));
}
