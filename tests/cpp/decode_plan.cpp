// Prints what csrc/decode_plan.h plans, for tests/test_decode_plan_cpu.py.
//   grids M...      column_grids of each M
//   chunks BITS...  chunk_grid
//   crc N...        crc_grid
//   tiles BITS...   jump_tiles of blocks of these bits
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "decode_plan.h"

using namespace bz2g;

int main(int argc, char **argv) {
  if (!std::strcmp(argv[1], "tiles")) {
    std::vector<int64_t> bits;
    for (int i = 2; i < argc; i++) bits.push_back(std::atoll(argv[i]));
    for (const int32_t t : jump_tiles(bits)) std::printf("%d ", t);
    std::printf("\n");
    return 0;
  }
  for (int i = 2; i < argc; i++) {
    const long long v = std::atoll(argv[i]);
    if (!std::strcmp(argv[1], "grids")) {
      const ColumnGrids g = column_grids((int)v);
      std::printf("%d %d %d %d %d\n", g.lf, g.walk, g.gather, g.repeat, g.unrle);
    } else if (!std::strcmp(argv[1], "chunks")) {
      std::printf("%d\n", chunk_grid(v));
    } else {
      std::printf("%d\n", crc_grid(v));
    }
  }
}
