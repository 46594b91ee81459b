// How a call's blocks are cut into slabs (host code without CUDA;
// csrc/compressor.cu drives them).
#pragma once

#include <stdint.h>

#include <algorithm>
#include <vector>

namespace bz2g {

// Workspace a block takes in a slab (raw: its bytes rounded up to 16), and
// what a slab has.
struct BlockNeeds {
  int64_t raw, elems;
  int raw_tiles, tiles, group_tiles;
};

// Fewest blocks of a slab: with fewer the launches of another slab cost more
// than they overlap.
constexpr int kMinSlabBlocks = 16;
// Bytes of a call from which it takes a second slab, and per slab beyond that.
// Every slab at work has a host thread, and where the program keeps the cores
// busy (OpenMP's threads spin for some ms after a parallel loop) a thread
// beyond the caller's costs about 1.1 ms, whatever the slab.  So a call is cut
// only where even then it takes no longer than as one slab did before there
// were several, sooner for host input, whose copies overlap too.  In ms, one
// slab then / cut on an idle host / on a busy one: 30 MB on the device 3.1 /
// 1.8 / 2.9 (two slabs), 110 MB 6.6 / 4.2 / 6.2 (three); 45 MB from the host
// 4.6 / 2.8 / 4.1 (two), 110 MB 8.6 / 5.2 / 7.2 (four), but 60 MB 5.4 / 3.2 /
// 5.7 with three.  Cut by 16 blocks alone, 6.4 MB in blocks of 100,000 took
// 2.1 / 1.4 / 4.4, now 1.2 on both.
constexpr int64_t kTwoSlabBytes = 32 * 900000;
constexpr int64_t kDeviceSlabBytes = 32 * 900000;
constexpr int64_t kHostSlabBytes = 26 * 900000;
// Blocks per slab of host input, from four slabs on.
constexpr int kHostSlabBlocks = 128;

// Slabs of a call that fits the workers' slabs once: split evenly over the
// workers, so that their stages (and, from host memory, the copies) overlap.
// Host input takes several per worker once they hold kHostSlabBlocks, so that
// the first kernels need not wait for a quarter of the input.
inline int slab_count(int nblocks, int64_t bytes, int workers, bool on_device) {
  const int rounds = on_device ? 1 : std::max(1, nblocks / (workers * kHostSlabBlocks));
  const int64_t each = on_device ? kDeviceSlabBytes : kHostSlabBytes;
  const int64_t by_bytes = bytes < kTwoSlabBytes ? 1 : std::max<int64_t>(2, bytes / each);
  const int64_t most = std::min<int64_t>(nblocks / kMinSlabBlocks, by_bytes);
  return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)workers * rounds, most));
}

// First block of each slab, and the end, for a queue of n blocks.  A slab is
// closed when it holds cap(its first block) blocks or `share` bytes, or when
// the next block finds no room.
template <typename Needs, typename Cap>
std::vector<int> cut_queue(int n, const BlockNeeds &room, int64_t share, Needs needs, Cap cap) {
  std::vector<int> at{0};
  BlockNeeds sum{};
  int cnt = 0, most = 0;
  for (int q = 0; q < n; q++) {
    const BlockNeeds b = needs(q);
    if (cnt > 0 && (cnt == most || sum.raw >= share || sum.raw + b.raw > room.raw ||
                    sum.elems + b.elems > room.elems || sum.tiles + b.tiles > room.tiles ||
                    sum.raw_tiles + b.raw_tiles > room.raw_tiles ||
                    sum.group_tiles + b.group_tiles > room.group_tiles)) {
      at.push_back(q);
      sum = BlockNeeds{};
      cnt = 0;
    }
    if (cnt++ == 0) most = cap(q);
    sum = {sum.raw + b.raw, sum.elems + b.elems, sum.raw_tiles + b.raw_tiles, sum.tiles + b.tiles,
           sum.group_tiles + b.group_tiles};
  }
  if (n > 0) at.push_back(n);
  return at;
}

// The bytes at which a queue's slabs are closed so that it makes `slabs` of
// them: counted as the slabs count them, or a queue of short blocks would be
// closed before its last ones.
template <typename Needs>
int64_t queue_share(int n, int slabs, Needs needs) {
  int64_t sum = 0;
  for (int q = 0; q < n; q++) sum += needs(q).raw;
  return std::max<int64_t>(1, (sum + slabs - 1) / slabs);
}

}  // namespace bz2g
