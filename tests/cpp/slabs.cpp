// Prints what csrc/slabs.h decides, for tests/test_slabs_cpu.py.
//   slabs         slab_count per line "blocks bytes workers on_device" read
//   slabs queue   slab sizes per line "blocks length slabs cap" read: a queue
//                 of equal blocks, rooms that never bind
#include <climits>
#include <cstdio>

#include "slabs.h"

int main(int argc, char **) {
  long long nb, bytes;
  int workers, dev;
  if (argc > 1) {
    long long len;
    int slabs, cap;
    while (std::scanf("%lld %lld %d %d", &nb, &len, &slabs, &cap) == 4) {
      auto needs = [&](int) {
        return bz2g::BlockNeeds{(len + 15) / 16 * 16, len, 1, 1, 1};
      };
      const bz2g::BlockNeeds room{INT64_MAX, INT64_MAX, INT_MAX, INT_MAX, INT_MAX};
      const auto at = bz2g::cut_queue((int)nb, room, bz2g::queue_share((int)nb, slabs, needs),
                                      needs, [&](int) { return cap; });
      for (size_t k = 0; k + 1 < at.size(); k++) std::printf("%d ", at[k + 1] - at[k]);
      std::printf("\n");
    }
    return 0;
  }
  while (std::scanf("%lld %lld %d %d", &nb, &bytes, &workers, &dev) == 4)
    std::printf("%d\n", bz2g::slab_count((int)nb, bytes, workers, dev != 0));
}
