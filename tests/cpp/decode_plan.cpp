// Prints what csrc/decode_plan.h plans, for tests/test_decode_plan_cpu.py.
//   grids M...      column_grids of each M
//   chunks BITS...  chunk_grid
//   crc N...        crc_grid
//   tiles BITS...   jump_tiles of blocks of these bits
//   jumps ROOM BITS...  the pieces they run in, then whether they pay
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "decode_plan.h"

using namespace bz2g;

int main(int argc, char **argv) {
  if (!std::strcmp(argv[1], "jumps")) {
    std::vector<int64_t> bits;
    for (int i = 3; i < argc; i++) bits.push_back(std::atoll(argv[i]));
    const std::vector<int32_t> first = jump_tiles(bits);
    const std::vector<int> at = jump_pieces(first, std::atoll(argv[2]));
    for (const int q : at) std::printf("%d ", q);
    std::printf("\n%d\n", !at.empty() && jumps_pay(first, (int)at.size() - 1));
    return 0;
  }
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
