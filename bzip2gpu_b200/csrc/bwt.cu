// BWT of every block of a slab: sorted cyclic rotations by prefix doubling.
//
// Reference: src/compression/fbwt.cu:47-106 (prefix doubling with a stable
// 64-bit key sort each round; ties, i.e. equal rotations, keep index order).
//
// Here:
//   1. One segmented LSD radix sort (segments = blocks) of every rotation by
//      its first P bytes (cyclic, big-endian), stable from index order, so
//      ties are index-ascending.
//   2. Ranks are group heads: head = first SA position of the group;
//      ISA[i] = head of rotation i.  Rotations in groups of size 1 are final.
//   3. The rotations still in groups of size >= 2 ("active") are compacted,
//      per block, with their SA position.  Round with shift h (prefix length
//      h -> 2h) keys them (head << kb) | ISA[(i + h) mod m] and re-sorts them
//      stably; the k-th of them in sorted order goes to the k-th active SA
//      position (groups are contiguous, so this sorts within each group).
//      Short groups need no radix sort: a block whose active groups are all
//      short (sorts_groups) sorts them one by one in shared memory
//      (k_bwt_groups), in the same rounds.
//   4. A block stops when no rotation is active, when a round splits no group
//      (the rest are equal rotations, already index-ascending), or when the
//      prefix length reaches m.
// Block-local ranks fit kb = ceil(log2(max m + 1)) bits.  When 3*kb <= 64
// (m < 2^21, every bzip2 block) key and rotation share one 64-bit item and
// the sort moves items only: the first sort keys the first P = 4 bytes
// (item = prefix << 32 | i), rounds use item = head << 2kb | rank << kb | i.
// Larger m keeps separate 64-bit keys and 32-bit rotations, with P = 8.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "engine.h"

namespace bz2g {

namespace {

constexpr int kSortWarps = kTileThreads / 32;  // 8
constexpr int kWarpSpan = kTile / kSortWarps;   // elements per warp in a tile (512)
// Digits of the doubling rounds' sorts may be 9 bits wide (fewer passes over
// the 2kb key bits); the tile and group digit tables (tile_hist, scan_base)
// are sized for kMaxRadix digits.  Shared memory of the scatter: the tile's
// keys (and values), per-warp digit counts, two digit tables.
template <int RB>
constexpr size_t scatter_smem_keys() {
  return (size_t)kTile * 8 + (size_t)kSortWarps * (1 << RB) * 4 + 2 * (1 << RB) * 4;
}
template <int RB>
constexpr size_t scatter_smem_vals() {
  return scatter_smem_keys<RB>() + (size_t)kTile * 4;
}

// Tile of this CTA: blockIdx.x, or the blockIdx.x-th entry of a list of the
// tiles that hold work (doubling rounds).
__device__ __forceinline__ int tile_id(const int32_t *list) {
  return list ? list[blockIdx.x] : (int)blockIdx.x;
}

__device__ __forceinline__ int tile_valid(const SlabDev &d, int t, const int32_t *lens, int *b_out,
                                          int *lt_out) {
  int b = d.tile_block[t];
  int lt = (int)((int64_t)t * kTile - d.off[b]);
  *b_out = b;
  *lt_out = lt;
  int v = lens[b] - lt;
  return v < 0 ? 0 : (v > kTile ? kTile : v);
}

// The valid lanes of the warp whose RB-bit digit equals this lane's: one
// ballot per digit bit (cheaper here than __match_any_sync).
template <int RB>
__device__ __forceinline__ unsigned digit_peers(int dg, bool ok) {
  unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int bit = 0; bit < RB; bit++) {
    const bool on = (dg >> bit) & 1;
    const unsigned bb = __ballot_sync(0xffffffffu, on);
    peers &= on ? bb : ~bb;
  }
  return peers;
}

// The RB bits of an item from bit `shift` on.  kHigh: a byte of the high word
// (the first sort's 8-bit digits), one byte permutation.
template <int RB, bool kHigh>
struct Digit {
  int sh;
  bool high;
  __device__ __forceinline__ explicit Digit(int shift)
      : sh(kHigh ? 0x4440 + (shift - 32) / 8 : shift & 31), high(shift >= 32) {}
  __device__ __forceinline__ int operator()(uint64_t item) const {
    const uint32_t lo = (uint32_t)item, hi = (uint32_t)(item >> 32);
    if (kHigh) return (int)__byte_perm(hi, 0, sh);
    return (int)(__funnelshift_r(high ? hi : lo, high ? 0u : hi, sh) & ((1u << RB) - 1u));
  }
};

// The first sort of the packed layout starts from index order, so its first
// pass builds each tile's items itself from the block's text (read in order:
// the item at element e of a tile is rotation lt + e) instead of reading
// them: item = (first 4 bytes of the rotation, big-endian) << 32 | rotation.
__device__ __forceinline__ uint64_t text_item(const uint8_t *T, int m, int i) {
  uint32_t k = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    int j = i + q;
    while (j >= m) j -= m;
    k = (k << 8) | T[j];
  }
  return ((uint64_t)k << 32) | (uint32_t)i;
}

// The key buffers alternate with the passes that move anything: sort_ctl[0] is
// the buffer before a sort, bit p of sort_ctl[1] says whether pass p moves
// items (k_bwt_tile_list settles both at the end of a round).
__device__ __forceinline__ int keys_before(const SlabDev &d, int pass) {
  return (d.sort_ctl[0] ^ __popc(d.sort_ctl[1] & ((1 << pass) - 1))) & 1;
}
__device__ __forceinline__ int keys_now(const SlabDev &d) { return keys_before(d, 31); }

// Packed items leave the value buffers free; vals[0] holds the digit of each
// item for the coming pass, written by the pass before it (by k_bwt_round_keys
// for a round's first), so that the histogram reads 1 or 2 bytes per item
// instead of 8.
template <int RB>
using DigitT = std::conditional_t<RB == 8, uint8_t, uint16_t>;
template <int RB>
__device__ __forceinline__ DigitT<RB> *next_digits(const SlabDev &d) {
  return reinterpret_cast<DigitT<RB> *>(d.vals[0]);
}

template <int RB>
__device__ __forceinline__ void digit_scan(const SlabDev &d, int t, int force, int pass,
                                           uint32_t *scratch);
// The group of a block's tile t: kScanTiles tiles, of this block only.
__device__ __forceinline__ int scan_group(int t, int b) { return t / kScanTiles + b; }

// gen != 0: the generating first pass (items from the text, see text_item;
// 8-bit digits).  RB: digit width, tile_hist holds 2^RB counts per tile.
// The last tile of a group to finish its counts (a counter, after a fence that
// publishes the counts) runs the scan over the group's counts (digit_scan), so
// the pass needs no scan launch of its own.
// Bound by the latency of a tile's chain of loads, counts, fence and counter
// (4 to 5 us whatever the bytes): a CTA takes kHistTiles entries of the list, two
// warps each, a thread's loads are 16 bytes of digits, all issued before the
// counting.  Reading the items (8 bytes each) a tile per CTA took 1.76 + 0.92 ms
// (8- and 9-bit digits) for 1 GiB of text and 6.3 ms for 64 MiB of long repeats;
// now 0.92 + 0.50 and 3.5, for 0.4 ms more in the scatter of the first and 0.5
// of the second.
constexpr int kHistTiles = 4;

// Counts the digits of 16 loaded bytes that lie in [from, to) of the chunk.
template <int RB>
__device__ __forceinline__ void count_chunk(uint32_t *cnt, const uint4 &v, int from, int to) {
  constexpr int kPer = 16 / (int)sizeof(DigitT<RB>);
  const uint32_t x[4] = {v.x, v.y, v.z, v.w};
  // sorted items come in long runs of equal digits: one count for all
  if (from <= 0 && to >= kPer && v.x == v.y && v.x == v.z && v.x == v.w &&
      v.x == __funnelshift_l(v.x, v.x, RB == 8 ? 8 : 16)) {
    atomicAdd(&cnt[RB == 8 ? v.x & 255u : v.x & 0xffffu], (uint32_t)kPer);
    return;
  }
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const uint32_t q = RB == 8 ? __byte_perm(x[i / 4], 0, 0x4440 + i % 4)
                               : __byte_perm(x[i / 2 % 4], 0, i & 1 ? 0x4432 : 0x4410);
    if (i >= from && i < to) atomicAdd(&cnt[q], 1u);
  }
}

template <int RB>
__global__ void __launch_bounds__(256, 6) k_radix_hist(SlabDev d, int shift, const int32_t *list,
                                                       int ntiles, int gen, int packed, int pass) {
  constexpr int kN = 1 << RB, kThreads = 256 / kHistTiles;
  __shared__ uint32_t counts[kHistTiles][kN];
  __shared__ int s_last[kHistTiles];  // this tile, where it was the last of its group, or -1
  __shared__ uint32_t scratch[40];
  const int p = threadIdx.x / kThreads, u = threadIdx.x % kThreads;
  uint32_t *cnt = counts[p];
  const int entry = blockIdx.x * kHistTiles + p;
  int t = 0, b = 0, lt = 0, valid = 0;
  if (entry < ntiles) {
    t = list ? list[entry] : entry;
    valid = tile_valid(d, t, d.sort_len, &b, &lt);
  }
  for (int i = u; i < kN; i += kThreads) cnt[i] = 0;
  if (u == 0) s_last[p] = -1;
  __syncthreads();
  // the pass before wrote this one's digits if it ran
  const bool ready = packed && !gen && (pass == 0 || ((d.sort_ctl[1] >> (pass - 1)) & 1));
  if (valid > 0 && (ready || gen)) {
    // gen: digit bits [shift, shift + 8) of the item are byte q of the
    // rotation's 4-byte prefix: the tile's text from q on, and the q bytes after it
    const int q = gen ? 3 - (shift - 32) / 8 : 0;
    const uint8_t *T = d.rle1 + d.off[b];
    const uint4 *D = gen ? reinterpret_cast<const uint4 *>(T + lt)
                         : reinterpret_cast<const uint4 *>(next_digits<RB>(d) + d.off[b] + lt);
    constexpr int kPer = 16 / (int)sizeof(DigitT<RB>);
    constexpr int kLoads = 4;
#pragma unroll
    for (int e0 = 0; e0 < kTile; e0 += kLoads * kThreads * kPer) {
      uint4 v[kLoads];
#pragma unroll
      for (int i = 0; i < kLoads; i++) {
        const int c = e0 / kPer + i * kThreads + u;
        if (c * kPer < valid) v[i] = D[c];
      }
#pragma unroll
      for (int i = 0; i < kLoads; i++) {
        const int e = e0 + (i * kThreads + u) * kPer;
        if (e < valid) count_chunk<RB>(cnt, v[i], q - e, valid - e);
      }
    }
    if (u < min(q, valid)) {
      // (of a tile shorter than q, the whole window lies past its end)
      const int m = d.m[b];
      int j = lt + max(valid, q) + u;
      while (j >= m) j -= m;
      atomicAdd(&cnt[T[j]], 1u);
    }
  } else if (valid > 0) {
    const uint64_t *K = d.keys[keys_before(d, pass)] + d.off[b] + lt;
    const Digit<RB, false> dig(shift);
#pragma unroll 8
    for (int e = u; e < valid; e += kThreads) atomicAdd(&cnt[dig(K[e])], 1u);
  }
  __syncthreads();
  if (valid > 0)
    for (int i = u; i < kN; i += kThreads) d.tile_hist[(size_t)t * kN + i] = cnt[i];
  __threadfence();
  __syncthreads();
  if (u == 0 && valid > 0) {
    const int t0 = t - lt / kTile, nt = (d.sort_len[b] + kTile - 1) / kTile;
    const int tiles = min(t0 + nt, (t | (kScanTiles - 1)) + 1) - max(t0, t & -kScanTiles);
    if (atomicAdd(&d.scan_count[scan_group(t, b)], 1) == tiles - 1) s_last[p] = t;
  }
  __syncthreads();
  for (int k = 0; k < kHistTiles; k++)
    if (s_last[k] >= 0) digit_scan<RB>(d, s_last[k], gen, pass, scratch);
}

// Adds n rows of digit counts to `run`, and (kWrite) replaces each row by what
// `run` was before it.  Thread i handles the kD = 2^RB / 256 consecutive digits
// kD*i .. kD*i+kD-1; a row's loads are independent, kU are in flight.
template <int RB, bool kWrite>
__device__ __forceinline__ void scan_rows(uint32_t *rows, int n, uint32_t *run) {
  constexpr int kN = 1 << RB, kD = kN / 256;
  constexpr int kU = kD == 1 ? 16 : 8;
  uint32_t *H = rows + kD * threadIdx.x;
  for (int k0 = 0; k0 < n; k0 += kU) {
#pragma unroll
    for (int q = 0; q < kD; q++) {
      uint32_t h[kU];
#pragma unroll
      for (int j = 0; j < kU; j++) h[j] = k0 + j < n ? __ldcg(&H[(size_t)(k0 + j) * kN + q]) : 0u;
#pragma unroll
      for (int j = 0; j < kU; j++) {
        if (kWrite && k0 + j < n) H[(size_t)(k0 + j) * kN + q] = run[q];
        run[q] += h[j];
      }
    }
  }
}

// By the CTA that counted the last tile of a group of kScanTiles tiles: each
// tile's count of a digit becomes that of the group's earlier tiles.  The last
// group of a block turns the groups' sums into where the digit's items of each
// group go (scan_base).  One CTA per block over all the block's tiles took 10
// to 25 us at the end of a launch (64 MiB of long repeats, 186 launches: 4.0 ms,
// in groups 3.5).
// force != 0 (the generating pass): the pass runs even if every tile holds one
// digit only, since it writes the items the later passes read.
template <int RB>
__device__ __forceinline__ void digit_scan(const SlabDev &d, int t, int force, int pass,
                                           uint32_t *scratch) {
  constexpr int kN = 1 << RB, kD = kN / 256;
  __shared__ int s_end;
  const int b = d.tile_block[t];
  const int len = d.sort_len[b];
  const int t0 = (int)(d.off[b] / kTile), t1 = t0 + (len + kTile - 1) / kTile;
  const int first = max(t0, t & -kScanTiles), g0 = scan_group(t0, b);
  const int g = scan_group(t, b) - g0, ng = scan_group(t1 - 1, b) - g0 + 1;
  uint32_t run[kD];
#pragma unroll
  for (int q = 0; q < kD; q++) run[q] = 0;
  __threadfence();
  scan_rows<RB, true>(d.tile_hist + (size_t)first * kN,
                      min(t1, (t | (kScanTiles - 1)) + 1) - first, run);
  uint32_t *base_rows = d.scan_base + (size_t)g0 * kN;
  uint32_t *SB = base_rows + kD * threadIdx.x;
  if (threadIdx.x == 0) d.scan_count[g0 + g] = 0;
  if (ng > 1) {
#pragma unroll
    for (int q = 0; q < kD; q++) SB[(size_t)g * kN + q] = run[q];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      s_end = atomicAdd(&d.blk_count[b], 1) == ng - 1;
      if (s_end) d.blk_count[b] = 0;
    }
    __syncthreads();
    if (!s_end) return;
    __threadfence();
#pragma unroll
    for (int q = 0; q < kD; q++) run[q] = 0;
    scan_rows<RB, false>(base_rows, ng, run);
  }
  // the digits' bases (exclusive sum over the digits of the block's counts)
  uint32_t sum = 0;
  bool one = false;
#pragma unroll
  for (int q = 0; q < kD; q++) {
    sum += run[q];
    one |= run[q] == (uint32_t)len;
  }
  uint32_t tot;
  uint32_t base = (uint32_t)d.off[b] + block_excl_sum(sum, scratch, &tot);
  int trivial = __syncthreads_or(one);
  if ((!trivial || force) && threadIdx.x == 0) atomicOr(&d.sort_ctl[1], 1 << pass);
#pragma unroll
  for (int q = 0; q < kD; q++) {
    const uint32_t c = run[q];
    run[q] = base;
    base += c;
  }
  if (ng > 1) {
    scan_rows<RB, true>(base_rows, ng, run);
  } else {
#pragma unroll
    for (int q = 0; q < kD; q++) SB[q] = run[q];
  }
}

// Stable scatter of one tile by one 8-bit digit.  Elements are warp-striped
// (lane l, item i <-> element w*512 + i*32 + l) so that ranking item by item
// over the lanes with equal digits keeps the original order; the tile is sorted locally
// in shared memory, then written so that equal digits go out contiguously.
// All of a thread's loads are issued before the ranking starts.
template <bool kVals, int RB, bool kHigh>
__global__ void __launch_bounds__(256, kVals ? 2 : 3)
    k_radix_scatter(SlabDev d, int shift, int next, int timed, const int32_t *list, int gen,
                    int pass) {
  constexpr int kN = 1 << RB, kD = kN / 256;
  if (!((d.sort_ctl[1] >> pass) & 1)) return;  // every block's items share this digit
  const int t = tile_id(list);
  int b, lt;
  const int valid = tile_valid(d, t, d.sort_len, &b, &lt);
  if (valid == 0) return;
  if (timed >= 0 && threadIdx.x == 0)
    atomicAdd((unsigned long long *)&d.kt_elems[timed], (unsigned long long)valid);
  extern __shared__ __align__(16) uint8_t smem[];
  uint64_t *sk = reinterpret_cast<uint64_t *>(smem);
  uint32_t *sv = reinterpret_cast<uint32_t *>(sk + kTile);
  uint32_t *wcnt = kVals ? sv + kTile : reinterpret_cast<uint32_t *>(sk + kTile);  // [warp][digit]
  uint32_t *goff = wcnt + kSortWarps * kN + kN;  // global digit base for this tile
  const int cur = keys_before(d, pass);
  const uint64_t *K = d.keys[cur] + d.off[b] + lt;
  const uint32_t *V = d.vals[cur] + d.off[b] + lt;
  const int w = warp_id(), ln = lane_id();
  const Digit<RB, kHigh> dig(shift);

  uint64_t key[kTileItems];
  uint32_t val[kTileItems];
  if (kHigh && gen) {
    const uint8_t *T = d.rle1 + d.off[b];
    const int m = d.m[b];
#pragma unroll
    for (int i = 0; i < kTileItems; i++) {
      const int e = w * kWarpSpan + i * 32 + ln;
      key[i] = e < valid ? text_item(T, m, lt + e) : 0;
    }
  } else {
#pragma unroll
    for (int i = 0; i < kTileItems; i++) {
      const int e = w * kWarpSpan + i * 32 + ln;
      key[i] = e < valid ? K[e] : 0;
      if (kVals) val[i] = e < valid ? V[e] : 0;
    }
  }
#pragma unroll
  for (int q = 0; q < kSortWarps * kD; q++) wcnt[q * 256 + threadIdx.x] = 0;

  __syncthreads();

  uint32_t rank2[kTileItems / 2];  // two 16-bit ranks per register (ranks < 512)
  const unsigned lt_mask = (1u << ln) - 1u;
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = w * kWarpSpan + i * 32 + ln;
    const bool ok = e < valid;
    const int dg = dig(key[i]);
    const unsigned peers = digit_peers<RB>(dg, ok);
    const uint32_t before = ok ? wcnt[w * kN + dg] : 0;
    const uint32_t r = before + __popc(peers & lt_mask);
    if (i & 1)
      rank2[i >> 1] |= r << 16;
    else
      rank2[i >> 1] = r;
    __syncwarp();
    if (ok && (peers & lt_mask) == 0) wcnt[w * kN + dg] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    const uint32_t *SB = d.scan_base + (size_t)scan_group(t, b) * kN;
    // per digit: its local base (exclusive scan over digits of the tile's
    // counts); each warp's count becomes that warp's local start for the
    // digit, and the digit's global base becomes (global - local) base, so
    // the placement and the write below read one table entry each
    __shared__ uint32_t scratch[40];
    uint32_t tot;
    if constexpr (kD == 1) {
      const int dg = threadIdx.x;
      uint32_t run = 0;
      for (int ww = 0; ww < kSortWarps; ww++) run += wcnt[ww * kN + dg];
      const uint32_t lb = block_excl_sum(run, scratch, &tot);
      uint32_t at = lb;
      for (int ww = 0; ww < kSortWarps; ww++) {
        const uint32_t c = wcnt[ww * kN + dg];
        wcnt[ww * kN + dg] = at;
        at += c;
      }
      goff[dg] = d.tile_hist[(size_t)t * kN + dg] + SB[dg] - lb;
    } else {
      // thread i: the kD consecutive digits kD*i ..
      uint32_t run[kD], sum = 0;
#pragma unroll
      for (int q = 0; q < kD; q++) {
        const int dg = kD * threadIdx.x + q;
        run[q] = 0;
        for (int ww = 0; ww < kSortWarps; ww++) run[q] += wcnt[ww * kN + dg];
        sum += run[q];
      }
      uint32_t lb = block_excl_sum(sum, scratch, &tot);
#pragma unroll
      for (int q = 0; q < kD; q++) {
        const int dg = kD * threadIdx.x + q;
        uint32_t at = lb;
        for (int ww = 0; ww < kSortWarps; ww++) {
          const uint32_t c = wcnt[ww * kN + dg];
          wcnt[ww * kN + dg] = at;
          at += c;
        }
        goff[dg] = d.tile_hist[(size_t)t * kN + dg] + SB[dg] - lb;
        lb += run[q];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = w * kWarpSpan + i * 32 + ln;
    if (e < valid) {
      const int dg = dig(key[i]);
      const uint32_t r = (i & 1) ? rank2[i >> 1] >> 16 : rank2[i >> 1] & 0xffffu;
      const uint32_t pos = wcnt[w * kN + dg] + r;
      sk[pos] = key[i];
      if (kVals) sv[pos] = val[i];
    }
  }
  __syncthreads();
  uint64_t *KO = d.keys[cur ^ 1];
  uint32_t *VO = d.vals[cur ^ 1];
  DigitT<RB> *DO = next_digits<RB>(d);
  const Digit<RB, kHigh> ndig(next);
  for (int k = threadIdx.x; k < valid; k += blockDim.x) {
    const uint64_t kk = sk[k];
    const int dg = dig(kk);
    const uint32_t g = goff[dg] + (uint32_t)k;
    KO[g] = kk;
    if (kVals) VO[g] = sv[k];
    if (!kVals && next >= 0) DO[g] = (DigitT<RB>)ndig(kk);
  }
}

// Stable sort of each block's elements by key bits [lo, hi), over `grid`
// tiles (all tiles, or the listed ones).
// gen: the first pass generates the packed first-sort items from the text.
// RB: digit width (8; 9 for packed items of the doubling rounds where that
// takes fewer passes).
template <int RB>
void radix_passes(const SlabDev &d, int lo, int hi, int has_vals, cudaStream_t st, int grid,
                  const int32_t *list, bool gen) {
  BZ_REQUIRE(RB == 8 || (!has_vals && !gen), kErrInternal, "wide digits are for packed rounds");
  const size_t smem = has_vals ? scatter_smem_vals<RB>() : scatter_smem_keys<RB>();
  int pass = 0;
  for (int shift = lo; shift < hi; shift += RB, pass++) {
    const int g = gen && shift == lo;
    const int next = shift + RB < hi ? shift + RB : -1;
    k_radix_hist<RB><<<(grid + kHistTiles - 1) / kHistTiles, 256, 0, st>>>(d, shift, list, grid, g,
                                                                          !has_vals, pass);
    BZ_LAUNCH_CHECK();
    int timed = -1;
    if (d.kt_on && *d.kt_n < kMaxTimedLaunches) {
      timed = (*d.kt_n)++;
      // the generating pass reads text bytes; the next pass's digits are written too
      d.kt_bpe[timed] = has_vals ? 24 : (g ? 9 : 16) + (next >= 0 ? (int)sizeof(DigitT<RB>) : 0);
      BZ_CUDA(cudaEventRecord(d.kt_ev[2 * timed], st));
    }
    if constexpr (RB == 8) {
      if (has_vals)
        k_radix_scatter<true, 8, false><<<grid, 256, smem, st>>>(d, shift, next, timed, list, 0, pass);
      else if (gen)
        k_radix_scatter<false, 8, true><<<grid, 256, smem, st>>>(d, shift, next, timed, list, g, pass);
      else
        k_radix_scatter<false, 8, false><<<grid, 256, smem, st>>>(d, shift, next, timed, list, 0, pass);
    } else {
      k_radix_scatter<false, RB, false><<<grid, 256, smem, st>>>(d, shift, next, timed, list, 0, pass);
    }
    BZ_LAUNCH_CHECK();
    if (timed >= 0) BZ_CUDA(cudaEventRecord(d.kt_ev[2 * timed + 1], st));
  }
}

// 9-bit digits where they take fewer passes than 8-bit ones (10-bit
// digits also save a pass for 19- and 20-bit rank fields, but their
// 4x digit tables made the deep rounds of long blocks slower)
bool wide_digits(int bits) { return (bits + 8) / 9 < (bits + 7) / 8; }

void radix_sort(const SlabDev &d, int lo, int hi, int has_vals, cudaStream_t st, int grid,
                const int32_t *list, bool gen = false) {
  if (grid <= 0) return;
  if (!has_vals && !gen && wide_digits(hi - lo))
    radix_passes<9>(d, lo, hi, has_vals, st, grid, list, gen);
  else
    radix_passes<8>(d, lo, hi, has_vals, st, grid, list, gen);
}

// ------------------------------------------------------------------- BWT
__global__ void k_bwt_init(SlabDev d) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b == 0)
    for (int k = 0; k < 10; k++) d.sort_ctl[k] = 0;
  if (b >= d.nblocks) return;
  int m = d.m[b];
  d.sort_len[b] = m > 1 ? m : 0;
  d.done[b] = m > 1 ? 0 : 1;
  d.ngroups[b] = -1;
  d.act_len[b] = 0;
  d.active_sum[b] = 0;
  d.loc[b] = d.loc_act[b] = d.loc_heads[b] = d.loc_sing[b] = d.gmax[b] = 0;
  // the histogram's counters: each pass resets them, and so does this
  d.blk_count[b] = 0;
  const int t0 = (int)(d.off[b] / kTile), t1 = t0 + (m + kTile - 1) / kTile;
  for (int g = scan_group(t0, b); m > 0 && g <= scan_group(t1 - 1, b); g++) d.scan_count[g] = 0;
  for (int k = 0; k < 8; k++) d.pstat[b * 8 + k] = 0;
  if (m == 1) d.sa[d.off[b]] = 0;
}

// The oracle's accounting of the rounds h = 1, 2, (4) that the first sort
// stands for (round h runs while the partition has a non-singleton group and
// the previous round split one), and the group count of the prefix before
// the first sort's as the fixed-point reference of the first ranking.
__device__ void prefix_account(const SlabDev &d, int b, int nq) {
  const int m = d.m[b];
  const int32_t *ps = d.pstat + b * 8;
  int64_t A = 0;
  bool stop = false;
  for (int q = 0; q < nq - 1 && !stop; q++) {
    const int G = ps[q], S = ps[4 + q];
    if (G == m) break;
    A += m - S;
    const int h = 1 << q;
    if (ps[q + 1] == G || 2 * h >= m) stop = true;
  }
  d.active_sum[b] = A;
  d.ngroups[b] = ps[nq - 2];
  if (A) atomicAdd(reinterpret_cast<unsigned long long *>(d.sort_ctl + 8), (unsigned long long)A);
}

// First keys: the first 4 (packed) or 8 bytes of each rotation.
__global__ void __launch_bounds__(256) k_bwt_keys0(SlabDev d, int packed) {
  __shared__ uint8_t sb[kTile + 8];
  int b, lt;
  int valid = tile_valid(d, blockIdx.x, d.sort_len, &b, &lt);
  if (valid == 0) return;
  const int m = d.m[b];
  const uint8_t *T = d.rle1 + d.off[b];
  for (int e = threadIdx.x; e < valid + 7; e += blockDim.x) {
    int i = lt + e;
    while (i >= m) i -= m;
    sb[e] = T[i];
  }
  __syncthreads();
  uint64_t *K = d.keys[0] + d.off[b] + lt;
  uint32_t *V = d.vals[0] + d.off[b] + lt;
  for (int e = threadIdx.x; e < valid; e += blockDim.x) {
    uint64_t k = 0;
    if (packed) {
#pragma unroll
      for (int q = 0; q < 4; q++) k = (k << 8) | sb[e + q];
      K[e] = (k << 32) | (uint32_t)(lt + e);
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) k = (k << 8) | sb[e + q];
      K[e] = k;
      V[e] = (uint32_t)(lt + e);
    }
  }
}

// ---------------------------------------------------------------- ranking
// After a sort, the sorted (key, rotation) pairs of a block sit at
// [off, off + len); element k belongs at SA position P[k] (k itself after the
// first sort; the k-th active position in later rounds).  A group starts
// where the key changes; its head is the SA position of its first element.
// Elements are read warp-striped (warp w owns [512w, 512w + 512), item i of
// lane l is element 512w + 32i + l) so every load is coalesced.

// Kinds of sorted elements: the first sort's packed items (prefix << 32 |
// rotation), a round's packed items (head << 2kb | rank << kb | rotation),
// separate keys.
enum Kind { kPrefixItems, kRoundItems, kKeys };

// What is compared: the prefix, head and rank, or the whole key.
template <int kKind>
using Key = std::conditional_t<kKind == kPrefixItems, uint32_t, uint64_t>;
// The difference (exclusive or) of two keys reaches this from the first byte on.
template <int kKind>
constexpr Key<kKind> kFirstByte = Key<kKind>(1) << (8 * (sizeof(Key<kKind>) - 1));

template <int kKind>
__device__ __forceinline__ Key<kKind> key_at(const uint64_t *K, int k, int kb) {
  if constexpr (kKind == kPrefixItems) return reinterpret_cast<const uint32_t *>(K)[2 * k + 1];
  else if constexpr (kKind == kRoundItems) return K[k] >> kb;
  else return K[k];
}

// Per tile: the group heads as a bit per element (head_bits), the last head
// (SA position) and the active (non-singleton) count of each warp span, head
// and singleton counts.  After the first sort it also counts the group heads
// and singletons of the prefix-1, -2, -4 (, -8) byte partitions: pstat[b*8 + q]
// heads and pstat[b*8 + 4 + q] singletons of prefix 2^q bytes.  An element
// heads its group of prefix P when its first P bytes differ from those before
// it, i.e. when the difference reaches the P-th byte, and is alone when the
// one after it differs so too: two differences give all partitions.  Each key is
// loaded once, all of a thread's at the start; neighbours come by shuffle
// (1 GiB of text, both rankings: 1.37 -> 1.16 ms).
template <int kKind, bool kInitial>
__global__ void __launch_bounds__(256) k_bwt_flags(SlabDev d, int kb, const int32_t *list) {
  __shared__ int red[2][kSortWarps];
  constexpr int kQ = !kInitial ? 0 : kKind == kPrefixItems ? 3 : 4;
  const int t = tile_id(list);
  int b, lt;
  const int valid = tile_valid(d, t, d.sort_len, &b, &lt);
  if (valid == 0) return;
  const int len = d.sort_len[b];
  const int64_t off = d.off[b];
  const uint64_t *K = d.keys[keys_now(d)] + off;
  const int w = warp_id(), ln = lane_id();
  uint32_t *bits = d.head_bits + (size_t)t * (kTile / 32) + w * kTileItems;
  int last = -1, heads = 0, sing = 0;
  int pc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  Key<kKind> key[kTileItems];
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = w * kWarpSpan + i * 32 + ln;
    key[i] = e < valid ? key_at<kKind>(K, lt + e, kb) : 0;
  }
  // the keys just before and after the warp's span
  Key<kKind> edge = 0;
  {
    const int k = lt + w * kWarpSpan + (ln ? kWarpSpan : -1);
    if (ln < 2 && k >= 0 && k < len) edge = key_at<kKind>(K, k, kb);
  }
  const Key<kKind> kbefore = __shfl_sync(0xffffffffu, edge, 0);
  const Key<kKind> kafter = __shfl_sync(0xffffffffu, edge, 1);
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = w * kWarpSpan + i * 32 + ln;
    const int k = lt + e;
    // the lane below, or the row above's last; the lane above, or the row below's first
    Key<kKind> kp = __shfl_up_sync(0xffffffffu, key[i], 1);
    Key<kKind> kn = __shfl_down_sync(0xffffffffu, key[i], 1);
    const Key<kKind> first = i ? __shfl_sync(0xffffffffu, key[i ? i - 1 : 0], 31) : kbefore;
    const Key<kKind> last_ = i + 1 < kTileItems
                                 ? __shfl_sync(0xffffffffu, key[i + 1 < kTileItems ? i + 1 : i], 0)
                                 : kafter;
    if (ln == 0) kp = first;
    if (ln == 31) kn = last_;
    bool hd = false, alone = false;
    if (e < valid) {
      const Key<kKind> p = k > 0 ? key[i] ^ kp : ~Key<kKind>(0);
      const Key<kKind> n = k + 1 < len ? key[i] ^ kn : ~Key<kKind>(0);
      const Key<kKind> pn = min(p, n);
      hd = p != 0;
      alone = pn != 0;
#pragma unroll
      for (int q = 0; q < kQ; q++) {
        const Key<kKind> at = kFirstByte<kKind> >> (8 * ((1 << q) - 1));
        pc[q] += p >= at;
        pc[4 + q] += pn >= at;
      }
    }
    const unsigned bm = __ballot_sync(0xffffffffu, hd);
    sing += __popc(__ballot_sync(0xffffffffu, alone));
    heads += __popc(bm);
    if (bm) last = k - ln + 31 - __clz(bm);
    if (ln == 0) bits[i] = bm;
  }
#pragma unroll
  for (int q = 0; q < 8; q++) {
    if ((q & 3) < kQ) {
      const int v = __reduce_add_sync(0xffffffffu, pc[q]);
      if (ln == 0 && v) atomicAdd(&d.pstat[b * 8 + q], v);
    }
  }
  if (ln == 0) {
    const int wvalid = min(max(valid - w * kWarpSpan, 0), kWarpSpan);
    d.warp_last[t * kSortWarps + w] =
        kInitial || last < 0 ? last : (d.kpos[d.sort_ctl[3]] + off)[last];
    d.warp_act[t * kSortWarps + w] = wvalid - sing;  // elements in groups of size >= 2
    red[0][w] = heads;
    red[1][w] = sing;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int h = 0, sg = 0;
    for (int q = 0; q < kSortWarps; q++) {
      h += red[0][q];
      sg += red[1][q];
    }
    d.tile_b[t] = h;
    d.tile_c[t] = sg;
  }
}

// Per block: carry of the last head into each warp span (512 elements of a
// tile), compaction offsets of the active elements per warp span, and the
// stop test: no active element left, no group split by this round (the rest
// are equal rotations), or prefix >= m.
// nq > 0: after the first sort (prefix_account).  Blocks sorted group by group
// (loc) are not ranked here.
__device__ void block_round_end(const SlabDev &d, int b, int active, int heads, int singles,
                                int64_t prefix_len) {
  const int m = d.m[b];
  const bool fin = active == 0 || heads == d.ngroups[b] || prefix_len >= m;
  d.ngroups[b] = heads - singles;  // groups among the rotations still active
  if (fin) {
    d.done[b] = 1;
    d.act_len[b] = 0;
  } else {
    d.act_len[b] = active;
    atomicAdd(&d.sort_ctl[2], 1);
    atomicAdd(&d.sort_ctl[6], active);
    d.active_sum[b] += active;  // rotations entering the next round
  }
}

__global__ void __launch_bounds__(256) k_bwt_rank_block(SlabDev d, int64_t prefix_len, int nq) {
  __shared__ int scratch[40];
  __shared__ int sx[256];
  const int b = blockIdx.x;
  const int len = d.sort_len[b];
  if (len <= 0 || d.loc[b]) return;
  const int nt = (len + kTile - 1) / kTile;
  const int t0 = (int)(d.off[b] / kTile);
  const int nw = nt * kSortWarps;
  int32_t *WL = d.warp_last + (int64_t)t0 * kSortWarps;
  int32_t *WA = d.warp_act + (int64_t)t0 * kSortWarps;
  int carry = -1, heads = 0, singles = 0, active = 0;
  for (int base = 0; base < nw; base += 256) {
    const int k = base + threadIdx.x;
    const int v = k < nw ? WL[k] : -1;
    const int ac = k < nw ? WA[k] : 0;
    const int inc = block_incl_max(v, scratch, -1);
    sx[threadIdx.x] = inc;
    __syncthreads();
    const int ex = threadIdx.x == 0 ? carry : max(carry, sx[threadIdx.x - 1]);
    if (k < nw) WL[k] = ex;
    const int c2 = max(carry, sx[255]);
    __syncthreads();
    carry = c2;
    int tot;
    const int ao = block_excl_sum(ac, scratch, &tot);
    if (k < nw) WA[k] = active + ao;
    active += tot;
  }
  for (int base = 0; base < nt; base += 256) {
    const int k = base + threadIdx.x;
    int tot;
    block_excl_sum(k < nt ? d.tile_b[t0 + k] : 0, scratch, &tot);
    heads += tot;
    block_excl_sum(k < nt ? d.tile_c[t0 + k] : 0, scratch, &tot);
    singles += tot;
  }
  if (threadIdx.x == 0) {
    if (nq > 0) prefix_account(d, b, nq);
    block_round_end(d, b, active, heads, singles, prefix_len);
  }
}

// Write SA and ISA for the sorted elements, and compact the elements of
// groups of size >= 2 (for blocks still sorting) into the other key/value/
// position buffers, keyed by their new head (rank of i+h added next round).
// Heads come from head_bits: an element's group starts at the last head up to
// it, and ends where the next element is a head.  Bound by latency and by the
// scattered writes of ISA (L2 57 %, DRAM 31 %): all of a thread's items and its
// warp's head bits are loaded first, 1 GiB of text, first ranking: 2.70 -> 2.40 ms.
template <int kKind, bool kInitial>
__global__ void __launch_bounds__(256) k_bwt_apply(SlabDev d, int kb, const int32_t *list) {
  const int t = tile_id(list);
  int b, lt;
  const int valid = tile_valid(d, t, d.sort_len, &b, &lt);
  if (valid == 0) return;
  const int len = d.sort_len[b];
  const int64_t off = d.off[b];
  const int cur = keys_now(d), pc = d.sort_ctl[3];
  const uint64_t *K = d.keys[cur] + off;
  const uint32_t *V = d.vals[cur] + off;
  const int32_t *P = d.kpos[pc] + off;
  const bool compact = d.done[b] == 0;
  const int w = warp_id(), ln = lane_id();
  const uint32_t *bits = d.head_bits + (size_t)t * (kTile / 32) + w * kTileItems;
  // this warp span's head carry and compaction offset (k_bwt_rank_block)
  int carry = d.warp_last[t * kSortWarps + w];
  int aoff = d.warp_act[t * kSortWarps + w];
  uint64_t *KO = d.keys[cur ^ 1] + off;
  uint32_t *VO = d.vals[cur ^ 1] + off;
  int32_t *PO = d.kpos[pc ^ 1] + off;
  int32_t *SA = d.sa + off;
  int32_t *IS = d.isa + off;
  const unsigned lt_mask = (1u << ln) - 1u, le_mask = 0xffffffffu >> (31 - ln);
  int gmax = 0;  // largest active group that ends here
  // all loads before the first use: lane i holds row i's bits (row 16: past the
  // tile, the block's next tile, or not used)
  const uint32_t my_bits = ln <= kTileItems ? bits[ln] : 0;
  uint32_t vals[kTileItems];
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = w * kWarpSpan + i * 32 + ln;
    const int k = lt + e;
    vals[i] = 0;
    if (e < valid) {
      if (kKind == kPrefixItems) vals[i] = (uint32_t)K[k];
      else if (kKind == kRoundItems) vals[i] = (uint32_t)(K[k] & ((1ull << kb) - 1));
      else vals[i] = V[k];
    }
  }
  uint32_t bm = __shfl_sync(0xffffffffu, my_bits, 0);
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = w * kWarpSpan + i * 32 + ln;
    const int k = lt + e;
    const bool ok = e < valid;
    const uint32_t bn = __shfl_sync(0xffffffffu, my_bits, i + 1);
    const uint32_t val = vals[i];
    int pos = k;
    if (!kInitial && ok) pos = P[k];
    const bool hd = (bm >> ln) & 1u;
    const bool tl = k + 1 == len || ((__funnelshift_r(bm, bn, 1) >> ln) & 1u);
    const bool active = ok && !(hd && tl);
    const uint32_t below = bm & le_mask;
    int head, next;  // up to this element, and up to the row's end
    if (kInitial) {
      head = below ? k - ln + 31 - __clz(below) : carry;
      next = bm ? k - ln + 31 - __clz(bm) : carry;
    } else {
      head = __shfl_sync(0xffffffffu, pos, below ? 31 - __clz(below) : 0);
      next = __shfl_sync(0xffffffffu, pos, bm ? 31 - __clz(bm) : 0);
      if (!below) head = carry;
      if (!bm) next = carry;
    }
    carry = next;
    bm = bn;
    const unsigned am = __ballot_sync(0xffffffffu, active);
    if (ok) {
      if (tl && !hd) gmax = max(gmax, pos - head + 1);
      SA[pos] = (int32_t)val;
      IS[val] = head;
      if (compact && active) {
        const int r = aoff + __popc(am & lt_mask);
        if (kKind != kKeys) {
          KO[r] = ((uint64_t)(uint32_t)head << (2 * kb)) | val;
        } else {
          KO[r] = (uint64_t)(uint32_t)head << kb;
          VO[r] = val;
        }
        PO[r] = pos;
      }
    }
    aoff += __popc(am);
  }
  if (compact && kKind != kKeys) {
    gmax = __reduce_max_sync(0xffffffffu, gmax);
    if (ln == 0 && gmax > 0) atomicMax(&d.gmax[b], gmax);
  }
}

// Groups of at most kGroupMax rotations can be sorted in shared memory: a CTA
// takes the groups that start in a unit of `step` items of a block's active
// list, and holds kTile, so a step is what the block's longest group leaves of
// that (2048 for every block took a CTA for half of what it can hold).  Longer
// groups leave steps that mostly reload what other CTAs hold, and every
// doubling of a group is a merge more, where the radix passes cost the same
// for any group, and their launches the same for any number of rotations.
// So groups of more than kGroupLong, or kGroupMean on average, are sorted here
// only while the slab's blocks on the radix path have few rotations in all.
// Measured, repeats that double until the end, by groups / by radix sort, ms:
//   groups of    3,500        1,800        1,280        750          500
//   1 block      3.6 / 3.8    2.9 / 3.8    2.9 / 3.8    2.6 / 3.8
//   2 blocks     5.2 / 4.2    4.4 / 4.3    4.2 / 4.3    3.8 / 4.3
//   4 blocks     8.0 / 6.1    7.4 / 6.1    6.4 / 6.1    5.7 / 6.1
//   16 blocks    26.3 / 16.0  24.5 / 16.0  21.6 / 16.1  17.9 / 16.0  15.5 / 16.1
// Text has a few long groups among very short ones, which the mean tells apart:
// with kGroupMax at 1,024 and no mean 512 MiB of it take 15.2 instead of 14.5.
constexpr int kMinStep = 512;
constexpr int kGroupMax = kTile - kMinStep;
constexpr int kGroupLong = 2048;
constexpr int kGroupMean = 512;
__device__ __forceinline__ bool sorts_groups(int gmax, int active, int groups, int radix_active) {
  if (gmax > kGroupMax) return false;
  if (gmax <= kGroupLong && active <= kGroupMean * groups) return true;
  return radix_active <= (gmax > kGroupLong ? 1 << 20 : gmax > kGroupLong / 2 ? 2 << 20 : 6 << 20);
}
__device__ __forceinline__ int group_step(int gmax) { return (kTile - gmax) & ~31; }

// Lists a block's tiles, or its units when it is sorted group by group.  The
// blocks' places are taken by a thread each, the entries written by a warp
// each.  One CTA of 1024 threads; nblocks in passes of 1024.
struct TileRuns {
  int at[1024], n[1024], first[1024], step[1024];
  int32_t *list[1024];
};

__device__ __forceinline__ void list_block(const SlabDev &d, TileRuns &r, int b, int len) {
  const bool loc = d.loc[b];
  const int unit = loc ? d.loc_step[b] : kTile;  // entries: tiles, or items / 32
  const int nt = (len + unit - 1) / unit;
  r.at[threadIdx.x] = atomicAdd(&d.sort_ctl[loc ? 7 : 5], nt);
  r.n[threadIdx.x] = nt;
  r.first[threadIdx.x] = (int)(d.off[b] / (loc ? 32 : kTile));
  r.step[threadIdx.x] = loc ? unit / 32 : 1;
  r.list[threadIdx.x] = loc ? d.loc_list : d.tile_list;
}

__device__ __forceinline__ void write_lists(const TileRuns &r, int nb) {
  for (int q = warp_id(); q < nb; q += 32)
    for (int k = lane_id(); k < r.n[q]; k += 32)
      r.list[q][r.at[q] + k] = r.first[q] + k * r.step[q];
}

// Ends a round: blocks sorted group by group settle their counts, the key and
// position buffers switch, sort_len = active rotations, and the next round's
// tiles are listed: tiles of the blocks that go on by radix sort, units of
// those whose groups are all short.
__global__ void __launch_bounds__(1024) k_bwt_tile_list(SlabDev d, int64_t prefix_len, int packed) {
  __shared__ TileRuns runs;
  // active rotations of the blocks that were on the radix path in this round
  // (those sorted by groups add theirs below)
  const int radix_active = d.sort_ctl[6];
  __syncthreads();
  for (int b0 = 0; b0 < d.nblocks; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    runs.n[threadIdx.x] = 0;
    if (b < d.nblocks) {
      if (d.loc[b] && d.sort_len[b] > 0) {
        block_round_end(d, b, d.loc_act[b], d.loc_heads[b], d.loc_sing[b], prefix_len);
        d.loc_act[b] = d.loc_heads[b] = d.loc_sing[b] = 0;
        d.loc_cur[b] ^= 1;
      }
      const int len = d.act_len[b];
      d.sort_len[b] = len;
      if (len > 0) {
        if (packed && !d.loc[b] && sorts_groups(d.gmax[b], len, d.ngroups[b], radix_active)) {
          d.loc[b] = 1;
          d.loc_cur[b] = keys_now(d) ^ 1;
        }
        d.loc_step[b] = group_step(d.gmax[b]);
        d.gmax[b] = 0;
        list_block(d, runs, b, len);
      }
    }
    __syncthreads();
    write_lists(runs, min(1024, d.nblocks - b0));
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    d.sort_ctl[0] = keys_now(d) ^ 1;
    d.sort_ctl[1] = 0;
    d.sort_ctl[3] ^= 1;
  }
}

// One round of the groups of a unit.  Items are head << 2kb | rank << kb |
// rotation; with the head replaced by the group's start in the tile (groups
// stand in no order in the list) they are all different and sorting them by
// value sorts every group by rank with ties in index order.  Each group is
// sorted by itself: ranks within 8 items by counting the smaller ones, then
// runs of 8, 16, .. merged, an item's place being its place in its run plus
// the number of smaller items in the sibling run (binary search; what follows
// a group's end is larger).  A warp takes part up to its
// longest group.  The new heads follow within the CTA, since an
// item's SA position is its group's head plus its place in the group.  About 200 instructions per rotation where
// the radix passes, ranking and compaction of a round took about 700.
__global__ void __launch_bounds__(256, 3) k_bwt_groups(SlabDev d, int kb) {
  __shared__ uint64_t key[kTile + 8];
  __shared__ uint16_t gsize[kTile];           // at a group's start
  __shared__ uint32_t starts[kTile / 32 + 1];  // bit per item: a group starts here
  __shared__ int red[3][kSortWarps];
  __shared__ int s_base;
  const int64_t u = (int64_t)d.loc_list[blockIdx.x] * 32;  // the unit's first item
  const int b = d.tile_block[u / kTile];
  const int64_t off = d.off[b];
  const int s = (int)(u - off);
  const int step = d.loc_step[b];
  const int len = d.sort_len[b];
  const int cur = d.loc_cur[b];
  const uint64_t *K = d.keys[cur] + off;
  const int w = warp_id(), ln = lane_id();
  const int avail = min(kTile, len - s);
  const unsigned le_mask = 0xffffffffu >> (31 - ln);
  const int hs = 2 * kb;  // bits of (rank, rotation)
  const uint64_t low = (1ull << hs) - 1, vmask = (1ull << kb) - 1;
  const int e0 = w * kWarpSpan + ln;  // item i of this thread: e0 + 32 i
  uint64_t mine[kTileItems];
  bool before_first = false;  // thread 0: the item before the unit is of another group
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = e0 + 32 * i;
    mine[i] = e < avail ? K[s + e] : ~0ull;
    if (e < avail) key[e] = mine[i];
  }
  if (threadIdx.x == 0) before_first = s == 0 || (K[s - 1] >> hs) != (mine[0] >> hs);
  __syncthreads();
  // group starts: the first in each of this warp's rows, and the last so far
  uint32_t gs2[kTileItems / 2];  // two 16-bit fields per register
  int wfirst = INT32_MAX, wafter = INT32_MAX, carry = -1;
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = e0 + 32 * i;
    bool st = false;
    if (e < avail) {
      if (e == 0) st = before_first;
      else st = (key[e - 1] >> hs) != (mine[i] >> hs);
    }
    const unsigned bm = __ballot_sync(0xffffffffu, st);
    if (ln == 0) starts[e >> 5] = bm;
    if (bm) {  // a row lies in the unit or after it
      if (e - ln < step) wfirst = min(wfirst, e - ln + __ffs(bm) - 1);
      else wafter = min(wafter, e - ln + __ffs(bm) - 1);
    }
    const unsigned below = bm & le_mask;
    const int g = below ? e - ln + 31 - __clz(below) : carry;
    carry = bm ? e - ln + 31 - __clz(bm) : carry;
    if (i & 1) gs2[i >> 1] |= (uint32_t)(g & 0xffff) << 16;
    else gs2[i >> 1] = (uint32_t)(g & 0xffff);
  }
  if (threadIdx.x == 0) starts[kTile / 32] = 0;
  if (ln == 0) {
    red[0][w] = wfirst;
    red[1][w] = carry;
    red[2][w] = wafter;
  }
  __syncthreads();
  int first = INT32_MAX, after = avail, before = -1;
#pragma unroll
  for (int q = 0; q < kSortWarps; q++) {
    first = min(first, red[0][q]);
    after = min(after, red[2][q]);
    if (q < w) before = max(before, red[1][q]);
  }
  if (first == INT32_MAX) return;  // one group from before covers the unit
  // [first, after): whole groups.  Keys with the group's start in front; a
  // group's last item leaves its size at its start.
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = e0 + 32 * i;
    uint32_t g = (i & 1) ? gs2[i >> 1] >> 16 : gs2[i >> 1] & 0xffffu;
    if (g == 0xffffu) g = (uint32_t)before & 0xffffu;
    if (i & 1) gs2[i >> 1] = (gs2[i >> 1] & 0xffffu) | (g << 16);
    else gs2[i >> 1] = (gs2[i >> 1] & 0xffff0000u) | g;
    const uint32_t nx = __funnelshift_r(starts[e >> 5], starts[(e >> 5) + 1], 1);
    if (e >= first && e < after) {
      mine[i] = ((uint64_t)g << hs) | (mine[i] & low);
      key[e] = mine[i];
      if (((nx >> ln) & 1u) || e + 1 == after) gsize[g] = (uint16_t)(e - (int)g + 1);
    } else if (e >= after && e < avail) {
      key[e] = ~0ull;
    }
  }
  if (threadIdx.x < 8) key[avail + threadIdx.x] = ~0ull;
  __syncthreads();
  // the fields become start | log2 of the size, rounded up, << 12
  int most = 0;
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = e0 + 32 * i;
    const uint32_t g = (i & 1) ? gs2[i >> 1] >> 16 : gs2[i >> 1] & 0xffffu;
    uint32_t lg = 0;
    if (e >= first && e < after) lg = 32 - __clz((uint32_t)gsize[g] - 1u);
    most = max(most, (int)lg);
    if (i & 1) gs2[i >> 1] += lg << 28;
    else gs2[i >> 1] += lg << 12;
  }
  most = __reduce_max_sync(0xffffffffu, most);  // this warp's longest group: up to 2^most
  if (ln == 0) red[2][w] = most;
  auto field = [&](int i) { return (i & 1) ? gs2[i >> 1] >> 16 : gs2[i >> 1] & 0xffffu; };
  // runs of 8
  uint32_t to2[kTileItems / 2];
  if (most > 0) {
#pragma unroll
    for (int i = 0; i < kTileItems; i++) {
      const int e = e0 + 32 * i;
      int to = e;
      if (e >= first && e < after) {
        const int g = field(i) & 0xfff;
        to = g + ((e - g) & ~7);
        const uint64_t *c = key + to;
#pragma unroll
        for (int q = 0; q < 8; q++) to += c[q] < mine[i];
      }
      if (i & 1) to2[i >> 1] |= (uint32_t)to << 16;
      else to2[i >> 1] = (uint32_t)to;
    }
  }
  __syncthreads();
  int all = 0;
#pragma unroll
  for (int q = 0; q < kSortWarps; q++) all = max(all, red[2][q]);
  if (most > 0) {
#pragma unroll
    for (int i = 0; i < kTileItems; i++) {
      const int e = e0 + 32 * i;
      const int to = (int)((i & 1) ? to2[i >> 1] >> 16 : to2[i >> 1] & 0xffffu);
      if (e >= first && e < after && to != e) key[to] = mine[i];
    }
  }
  __syncthreads();
  for (int l = 3; l < all; l++) {  // some group has more than 2^l items
    const int run = 1 << l;
    if (most > l) {
#pragma unroll
      for (int i = 0; i < kTileItems; i++) {
        const int e = e0 + 32 * i;
        int to = e;
        const uint32_t f = field(i);
        if (e >= first && e < after && (int)(f >> 12) > l) {
          const uint64_t x = key[e];
          mine[i] = x;
          const int at = e - (int)(f & 0xfffu);
          const bool odd = at & run;
          const int r0 = e - (at & (run - 1));          // this run
          int lo = odd ? r0 - run : r0 + run;           // its sibling
          to = odd ? e - run - lo : e - lo;
          int hi = min(lo + run, after);
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key[mid] < x) lo = mid + 1;
            else hi = mid;
          }
          to += lo;
        }
        if (i & 1) to2[i >> 1] |= (uint32_t)to << 16;
        else to2[i >> 1] = (uint32_t)to;
      }
    }
    __syncthreads();
    if (most > l) {
#pragma unroll
      for (int i = 0; i < kTileItems; i++) {
        const int e = e0 + 32 * i;
        const int to = (int)((i & 1) ? to2[i >> 1] >> 16 : to2[i >> 1] & 0xffffu);
        if (to != e) key[to] = mine[i];
      }
    }
    __syncthreads();
  }
  // new groups: group and rank alike
  carry = -1;
  int heads = 0, sing = 0, act = 0;
  uint32_t sg2[kTileItems / 2];
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = e0 + 32 * i;
    const bool in = e >= first && e < after;
    const uint64_t x = in ? key[e] : ~0ull;
    mine[i] = x;
    const bool hd = in && (e == first || (key[e - 1] >> kb) != (x >> kb));
    const bool tl = in && (key[e + 1] >> kb) != (x >> kb);
    const unsigned bm = __ballot_sync(0xffffffffu, hd);
    const unsigned below = bm & le_mask;
    const int g = below ? e - ln + 31 - __clz(below) : carry;
    carry = bm ? e - ln + 31 - __clz(bm) : carry;
    if (i & 1) sg2[i >> 1] |= (uint32_t)(g & 0xffff) << 16;
    else sg2[i >> 1] = (uint32_t)(g & 0xffff);
    const unsigned sm = __ballot_sync(0xffffffffu, hd && tl);
    const unsigned im = __ballot_sync(0xffffffffu, in);
    heads += __popc(bm);
    sing += __popc(sm);
    act += __popc(im & ~sm);
  }
  if (ln == 0) {
    red[0][w] = carry;
    red[1][w] = act;
    red[2][w] = heads | sing << 16;  // at most 512 each
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int a = 0, hh = 0, ss = 0;
    for (int q = 0; q < kSortWarps; q++) {
      const int v = red[1][q];
      red[1][q] = a;
      a += v;
      hh += red[2][q] & 0xffff;
      ss += red[2][q] >> 16;
    }
    s_base = a ? atomicAdd(&d.loc_act[b], a) : 0;
    atomicAdd(&d.loc_heads[b], hh);
    if (ss) atomicAdd(&d.loc_sing[b], ss);
  }
  __syncthreads();
  int sbefore = -1;
  for (int q = 0; q < w; q++) sbefore = max(sbefore, red[0][q]);
  int32_t *SA = d.sa + off;
  int32_t *IS = d.isa + off;
  uint64_t *KO = d.keys[cur ^ 1] + off + s_base + red[1][w];
  const unsigned lt_mask = le_mask >> 1;
  int gmax = 0;  // the longest group that goes on
#pragma unroll
  for (int i = 0; i < kTileItems; i++) {
    const int e = e0 + 32 * i;
    const bool in = e >= first && e < after;
    const uint64_t x = mine[i];
    const uint32_t sgv = (i & 1) ? sg2[i >> 1] >> 16 : sg2[i >> 1] & 0xffffu;
    const int sg = sgv == 0xffffu ? sbefore : (int)sgv;
    const int g = field(i) & 0xfff;
    const int head = in ? (int)(K[s + e] >> hs) : 0;  // the list still holds the group here
    const int nhead = head + (sg - g);
    const uint32_t val = (uint32_t)(x & vmask);
    const bool tl = in && (key[e + 1] >> kb) != (x >> kb);
    const bool active = in && !(sg == e && tl);
    if (in) {
      SA[head + (e - g)] = (int32_t)val;
      if (nhead != head) IS[val] = nhead;
    }
    const unsigned am = __ballot_sync(0xffffffffu, active);
    if (active) KO[__popc(am & lt_mask)] = ((uint64_t)(uint32_t)nhead << hs) | val;
    KO += __popc(am);
    if (tl && sg != e) gmax = max(gmax, e - sg + 1);
  }
  gmax = __reduce_max_sync(0xffffffffu, gmax);
  if (ln == 0 && gmax > 0) atomicMax(&d.gmax[b], gmax);
}

// Round keys for the compacted active rotations: add the rank of i+h.  loc: the
// list holds units of the blocks sorted group by group, else tiles.
__global__ void __launch_bounds__(256) k_bwt_round_keys(SlabDev d, int h, int packed, int kb,
                                                        const int32_t *list, int loc, int wide) {
  const int t = list[blockIdx.x];
  const int64_t u = (int64_t)t * (loc ? 32 : kTile);
  const int b = d.tile_block[u / kTile];
  const int64_t off = d.off[b];
  const int lt = (int)(u - off);
  const int len = d.sort_len[b];
  const int valid = min(loc ? d.loc_step[b] : kTile, len - lt);
  if (valid <= 0) return;
  const int m = d.m[b];
  const int cur = loc ? d.loc_cur[b] : d.sort_ctl[0];
  uint64_t *K = d.keys[cur] + off + lt;
  const uint32_t *V = d.vals[cur] + off + lt;
  const int32_t *IS = d.isa + off;
  const uint64_t mask = (1ull << kb) - 1;
  for (int e = threadIdx.x; e < valid; e += blockDim.x) {
    if (packed) {
      uint64_t item = K[e];
      int i2 = (int)(item & mask) + h;
      if (i2 >= m) i2 -= m;
      item |= (uint64_t)(uint32_t)IS[i2] << kb;
      K[e] = item;
      // the first pass's digit: the bits from kb on, the rank's low ones and,
      // where kb is less than a digit, the head's
      const uint32_t low = (uint32_t)(item >> kb);
      if (!loc && wide) next_digits<9>(d)[off + lt + e] = low & 511u;
      if (!loc && !wide) next_digits<8>(d)[off + lt + e] = (uint8_t)low;
    } else {
      int i2 = (int)V[e] + h;
      if (i2 >= m) i2 -= m;
      K[e] |= (uint32_t)IS[i2];
    }
  }
}

// Shared memory above the default, once per device.
void configure_smem() {
  static std::atomic<uint64_t> configured{0};
  int dev = 0;
  BZ_CUDA(cudaGetDevice(&dev));
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (bit && (configured.load(std::memory_order_acquire) & bit)) return;
  auto room = [](auto kernel, size_t bytes) {
    BZ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  };
  room(k_radix_scatter<true, 8, false>, scatter_smem_vals<8>());
  room(k_radix_scatter<false, 8, true>, scatter_smem_keys<8>());
  room(k_radix_scatter<false, 8, false>, scatter_smem_keys<8>());
  room(k_radix_scatter<false, 9, false>, scatter_smem_keys<9>());
  configured.fetch_or(bit, std::memory_order_release);
}

}  // namespace

void stage_bwt(const SlabDev &d, int max_m, cudaStream_t st) {
  configure_smem();
  k_bwt_init<<<(d.nblocks + 127) / 128, 128, 0, st>>>(d);
  BZ_LAUNCH_CHECK();
  if (max_m <= 1) return;
  // the tiles holding rotations (a block's workspace has room for its
  // worst-case RLE1 output, so most of its tiles are usually empty), and the
  // slab's largest m, which sets the width of the rank fields
  const int nlive = live_tiles(d, st);
  if (nlive == 0) return;
  if (nlive > 0 && d.live[2] >= 0) max_m = std::min(max_m, std::max(d.live[2], 1));
  if (max_m <= 1) return;
  int kb = 1;
  while ((1ll << kb) <= (int64_t)max_m) kb++;
  const int packed = 3 * kb <= 64;
  const int wide = wide_digits(2 * kb);  // the rounds' digits
  bool rounds_timed = d.kt_on && d.rt_ev != nullptr;
  if (rounds_timed) {
    d.rt_act[0] = 0;
    BZ_CUDA(cudaEventRecord(d.rt_ev[0], st));
  }
  const int grid0 = nlive > 0 ? nlive : d.ntiles;
  const int32_t *list0 = nlive > 0 ? d.vt_list : nullptr;
  // first sort: 4-byte prefixes in the high half of packed items, or 8-byte keys
  if (packed) {
    radix_sort(d, 32, 64, 0, st, grid0, list0, true);
  } else {
    k_bwt_keys0<<<d.ntiles, 256, 0, st>>>(d, packed);
    BZ_LAUNCH_CHECK();
    radix_sort(d, 0, 64, 1, st, d.ntiles, nullptr);
  }
  const int nq = packed ? 3 : 4;  // prefixes 1,2,4 (,8) bytes
  int64_t prefix = packed ? 4 : 8;
  int grid = grid0, lgrid = 0;
  const int32_t *list = list0;
  int r = 0;  // round being run (0: the first sort)
  for (int initial = 1;; initial = 0) {
    BZ_CUDA(cudaMemsetAsync(d.sort_ctl + 2, 0, sizeof(int32_t), st));
    BZ_CUDA(cudaMemsetAsync(d.sort_ctl + 5, 0, 3 * sizeof(int32_t), st));
    if (grid > 0) {
      auto rank = [&](auto flags, auto apply) {
        flags<<<grid, 256, 0, st>>>(d, kb, list);
        BZ_LAUNCH_CHECK();
        k_bwt_rank_block<<<d.nblocks, 256, 0, st>>>(d, prefix, initial ? nq : 0);
        BZ_LAUNCH_CHECK();
        apply<<<grid, 256, 0, st>>>(d, kb, list);
        BZ_LAUNCH_CHECK();
      };
      if (packed && initial) rank(k_bwt_flags<kPrefixItems, true>, k_bwt_apply<kPrefixItems, true>);
      else if (packed) rank(k_bwt_flags<kRoundItems, false>, k_bwt_apply<kRoundItems, false>);
      else if (initial) rank(k_bwt_flags<kKeys, true>, k_bwt_apply<kKeys, true>);
      else rank(k_bwt_flags<kKeys, false>, k_bwt_apply<kKeys, false>);
    }
    if (lgrid > 0) {
      k_bwt_groups<<<lgrid, 256, 0, st>>>(d, kb);
      BZ_LAUNCH_CHECK();
    }
    k_bwt_tile_list<<<1, 1024, 0, st>>>(d, prefix, packed);
    BZ_LAUNCH_CHECK();
    if (rounds_timed) {
      BZ_CUDA(cudaEventRecord(d.rt_ev[2 * r + 1], st));
      *d.rt_n = r + 1;
    }
    if (prefix >= max_m) break;
    BZ_CUDA(cudaMemcpyAsync(d.h_flags, d.sort_ctl + 2, 8 * sizeof(int32_t), cudaMemcpyDeviceToHost,
                            st));
    BZ_CUDA(cudaStreamSynchronize(st));
    if (rounds_timed && initial)
      std::memcpy(&d.rt_act[0], d.h_flags + 6, sizeof(int64_t));  // sort_ctl[8..9]
    if (d.h_flags[0] == 0) break;
    grid = d.h_flags[3];   // tiles holding active rotations
    lgrid = d.h_flags[5];  // units of the blocks sorted group by group
    list = d.tile_list;
    r++;
    if (rounds_timed && r >= kMaxRounds) rounds_timed = false;
    if (rounds_timed) {
      d.rt_act[r] = d.h_flags[4];  // rotations entering this round
      BZ_CUDA(cudaEventRecord(d.rt_ev[2 * r], st));
    }
    // every block's keys before any block's ranks change
    if (grid > 0) {
      k_bwt_round_keys<<<grid, 256, 0, st>>>(d, (int)prefix, packed, kb, list, 0, wide);
      BZ_LAUNCH_CHECK();
    }
    if (lgrid > 0) {
      k_bwt_round_keys<<<lgrid, 256, 0, st>>>(d, (int)prefix, packed, kb, d.loc_list, 1, 0);
      BZ_LAUNCH_CHECK();
    }
    if (packed)
      radix_sort(d, kb, 3 * kb, 0, st, grid, list);
    else
      radix_sort(d, 0, 2 * kb, 1, st, grid, list);
    prefix *= 2;
  }
}

}  // namespace bz2g
