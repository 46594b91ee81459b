// Launch shapes of the decoder, from a batch's own blocks (host code without
// CUDA; csrc/decode.cu has the kernels).
#pragma once

#include <stdint.h>

#include <algorithm>
#include <vector>

namespace bz2g {

constexpr int kDecMaxSel = 18002;
// Per-block capacity of the last column (the reference's 900,000-byte raw
// blocks can exceed 900,000 RLE1 bytes by up to a quarter).
constexpr int kDecCap = 1200000;
constexpr int kDecGroupSyms = 50;
constexpr int kChunkGroups = 32;  // groups per warp of k_dec_syms and k_dec_emit
constexpr int kMaxChunks = (kDecMaxSel + kChunkGroups - 1) / kChunkGroups;
constexpr int kSymWarps = 4;
constexpr int kLfChunk = 4096;    // last-column bytes per CTA of k_dec_lf_hist, _rank
constexpr int kWalkThreads = 128;
constexpr int kWalkChunk = 64;    // bytes per pool chunk of the walks
constexpr int kGatherChunks = 128;  // pool chunks per CTA of k_dec_gather
constexpr int kUnTile = 8192;     // RLE1 bytes per CTA of k_dec_unrle1_count, _write
constexpr int kCrcParts = 32;     // CTAs that share a block's CRC, at most
constexpr int kCrcChunk = 4096;   // output bytes they take at a time

inline int dec_ceil(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// Walkers of the inverse BWT: one per walk_step(m) positions, and origPtr's.
constexpr int walk_step(int m) { return m > kDecCap / 2 ? 128 : 64; }
constexpr int walker_count(int m, int orig) {
  return (m + walk_step(m) - 1) / walk_step(m) + (orig % walk_step(m) != 0);
}

// CTAs per block of k_dec_syms and k_dec_emit (whose warps take further chunks
// a grid apart, so this is no bound): a code has at least a bit, and
// `max_bits` is the most bits between two block candidates.
inline int chunk_grid(int64_t max_bits) {
  const int64_t groups = std::min<int64_t>(kDecMaxSel, max_bits / kDecGroupSyms + 1);
  return dec_ceil(dec_ceil(groups, kChunkGroups), kSymWarps);
}

// CTAs per block of the stages after the entropy decode, for blocks of at most
// m last-column bytes.  Grids for the largest block the format allows cost
// more than the work for short ones: 5 MB in blocks of 1,000 bytes took 6.6 ms,
// of which 4 launched CTAs that returned at once.
struct ColumnGrids {
  int lf, walk, gather, repeat, unrle;
};
inline ColumnGrids column_grids(int m) {
  // (128 bytes a walker give fewer walkers than 64 for a shorter block)
  const int walkers = dec_ceil(std::min(m, kDecCap / 2), 64) + 1;
  const int most = std::max(walkers, dec_ceil(m, 128) + 1);
  return {dec_ceil(m, kLfChunk), dec_ceil(most, kWalkThreads),
          dec_ceil(most + m / kWalkChunk + 1, kGatherChunks), std::min(16, dec_ceil(m, 4096)),
          dec_ceil(m, kUnTile)};
}

// CTAs per block of k_dec_crc, for blocks of at most n output bytes.
inline int crc_grid(int64_t n) {
  return (int)std::min<int64_t>(kCrcParts, std::max<int64_t>(1, dec_ceil(n, kCrcChunk)));
}

// Tiles of the jumps over whole groups (k_dec_jumps): kJumpTile bit positions
// of a block per CTA, blocks one after another.
constexpr int kJumpTile = 4096;
// No block is longer: header with symbol map, selectors of at most 6 bits, six
// tables of 258 lengths of at most 63 steps, 50 codes of at most 20 bits per
// group.  (Bytes that follow a stream's last block count as its own until then.)
constexpr int64_t kMaxBlockBits = 105 + 16 + 256 + 18 + 6 * kDecMaxSel + 6 * (5 + 258 * 127) +
                                  (int64_t)kDecMaxSel * kDecGroupSyms * 20;

// First tile of each block, and their number, for blocks of the given bits.
inline std::vector<int32_t> jump_tiles(const std::vector<int64_t> &bits) {
  std::vector<int32_t> first(bits.size() + 1, 0);
  for (size_t q = 0; q < bits.size(); q++)
    first[q + 1] = first[q] + (int32_t)(std::min(bits[q], kMaxBlockBits) / kJumpTile) + 1;
  return first;
}

// Jumps or chains (k_dec_groups) for a batch.  Jumps cost work with the bits
// of all blocks, chains the time of the longest block until the blocks fill
// the GPU, and tables for every block; so the total over the longest block
// decides, whatever their size, and blocks of few tiles take jumps.  Whole
// decodes by jumps / chains, ms:
//   blocks            8            40           100          140          300
//   text, 900,000     1.6 / 4.4    3.3 / 5.4    6.8 / 7.5    9.3 / 9.2    19 / 15
//   text, 100,000     0.74 / 1.0   0.99 / 1.4   1.4 / 1.5    1.9 / 1.7    2.9 / 2.3
//   noise, 900,000    4.1 / 13.2   10.8 / 16.1  22.5 / 20.6
//   noise, 100,000    1.0 / 2.0    1.8 / 2.3    3.2 / 2.9    4.0 / 3.2    8.0 / 5.0
// The lines cross at about 130 blocks of text and 80 of noise, which cannot be
// told apart by their bits; 1,000 blocks of 5,000 bytes take 1.1 / 1.6.
// Jumps of more tiles than their scratch holds run in pieces of whole blocks;
// each piece takes the chain of jumps through its longest block anew.  Only
// noise has such blocks in numbers for which it pays (two pieces: 40 blocks
// 11.2 / 14.9, 60 blocks 16.1 / 15.8).
constexpr int kJumpRatio = 125;
constexpr int kJumpRatioPieces = 55;
constexpr int kJumpBlock = 3;
constexpr int kJumpMaxTiles = 51200;  // a piece's: 2.5 GB of scratch
constexpr int64_t kJumpTileBytes = 6 * 2 * kJumpTile;  // two bytes per table and position

// Blocks at which the pieces begin, and the end; empty when a block alone has
// more tiles than the scratch.
inline std::vector<int> jump_pieces(const std::vector<int32_t> &first, int64_t room_tiles) {
  std::vector<int> at{0};
  for (int q = 0; q + 1 < (int)first.size(); q++) {
    if (first[q + 1] - first[q] > room_tiles) return {};
    if (first[q + 1] - first[at.back()] > room_tiles) at.push_back(q);
  }
  at.push_back((int)first.size() - 1);
  return at;
}

inline bool jumps_pay(const std::vector<int32_t> &first, int pieces) {
  const int64_t n = (int64_t)first.size() - 1;
  int64_t longest = 1;
  for (int64_t q = 0; q < n; q++) longest = std::max<int64_t>(longest, first[q + 1] - first[q]);
  return first.back() <= (pieces > 1 ? kJumpRatioPieces : kJumpRatio) * longest + kJumpBlock * n;
}

}  // namespace bz2g
