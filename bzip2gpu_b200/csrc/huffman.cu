// Huffman table selection and code lengths, for every block of a slab.
//
// Reference: src/compression/huffman.cu:126-364 (bzip2 1.0.8 sendMTFValues
// semantics): nGroups from the symbol count; initial tables from the symbol
// histogram; 4 passes of (per 50-symbol group: cost of every table, first
// minimum wins, per-table frequencies of the chosen groups) each followed by
// length-limited (17) Huffman code lengths per table; canonical codes.
// The histogram is defined as zeroed (the reference leaves it uninitialised).
#include "engine.h"
#include "selector.h"

namespace bz2g {

namespace {

// Which blocks a launch serves: every block, the plain-selector blocks, the
// learned-selector blocks, or (learned form, after the judge) the plain
// blocks that still have passes to run in this round.
enum Which { kAll = 0, kPlain = 1, kLearned = 2, kPlainRound = 3 };

__device__ __forceinline__ bool serves(const SlabDev &d, int b, int which, int round) {
  switch (which) {
    case kAll:
      return true;
    case kPlain:
      return d.learned[b] == 0;
    case kLearned:
      return d.learned[b] != 0;
    default:
      return d.learned[b] == 0 && round < d.plain_left[b];
  }
}

// bzip2's initial tables (src/compression/huffman.cu:148-185): every length
// 15, then table n_part - 1 gets length 0 over the next range of symbols
// holding about remaining / n_part of the symbol count: it ends at the first
// symbol where the counts from its start reach that share (alpha if none
// does).  One warp: running counts in shared memory, a ballot per 32 symbols
// finds each end (one thread adding up the counts took 32 us).
constexpr int kFreqSlots = (kMaxAlpha + 31) / 32;  // 9

__device__ void init_tables(const SlabDev &d, int b, int32_t *cum) {
  const unsigned full = 0xffffffffu;
  const int ln = lane_id();
  const int s = d.s[b];
  const int ng = d.n_groups[b];
  const int alpha = d.n_in_use[b] + 2;
  uint8_t *len = d.len + (size_t)b * kMaxGroups * kMaxAlpha;
  const int32_t *freq = d.freq + (size_t)b * kMaxAlpha;
  int f[kFreqSlots];
#pragma unroll
  for (int q = 0; q < kFreqSlots; q++) f[q] = 32 * q + ln < kMaxAlpha ? freq[32 * q + ln] : 0;
  int run = 0;
#pragma unroll
  for (int q = 0; q < kFreqSlots; q++) {
    const int inc = warp_incl_sum(f[q]);
    f[q] = run + inc;  // counts of the symbols up to this one
    cum[32 * q + ln] = f[q];
    run += __shfl_sync(full, inc, 31);
  }
  for (int i = ln; i < kMaxGroups * kMaxAlpha; i += 32) len[i] = 15;
  __syncwarp();
  // counts of the symbols up to v (nothing past the alphabet's room)
  auto upto = [&](int v) { return v < 0 ? 0 : cum[min(v, kMaxAlpha - 1)]; };
  int gs = 0, remaining = s;
  for (int n_part = ng; n_part > 0; n_part--) {
    const int t_freq = remaining / n_part;
    const int base = upto(gs - 1);
    int ge = gs - 1;
    if (t_freq > 0) {
      ge = alpha;
#pragma unroll
      for (int q = kFreqSlots - 1; q >= 0; q--) {
        const int v = 32 * q + ln;
        const unsigned hit = __ballot_sync(full, v >= gs && v < alpha && f[q] - base >= t_freq);
        if (hit) ge = 32 * q + __ffs(hit) - 1;
      }
      if (gs > alpha) ge = gs - 1;  // no symbol is left
    }
    int a_freq = upto(ge) - base;
    if (ge > gs && n_part != ng && n_part != 1 && ((ng - n_part) % 2 == 1)) {
      a_freq = upto(ge - 1) - base;
      ge--;
    }
    uint8_t *row = len + (n_part - 1) * kMaxAlpha;
    for (int v = gs + ln; v <= min(ge, alpha - 1); v += 32) row[v] = 0;
    gs = ge + 1;
    remaining -= a_freq;
  }
  __syncwarp();
}

// learned_mode: blocks with six tables take the learned selector; the plain
// blocks of the learned form have 2 passes left after the two shared ones.
__global__ void k_huff_init(SlabDev d, int learned_mode) {
  __shared__ int32_t cum[32 * kFreqSlots];
  const int b = blockIdx.x;
  const int s = d.s[b];
  const int ng = s < 200 ? 2 : s < 600 ? 3 : s < 1200 ? 4 : s < 2400 ? 5 : 6;
  if (threadIdx.x == 0) {
    d.n_groups[b] = ng;
    d.n_sel[b] = (s + 49) / 50;
    d.learned[b] = (learned_mode && ng == kMaxGroups) ? 1 : 0;
    d.plain_left[b] = kIters - 2;
  }
  __syncwarp();
  init_tables(d, b, cum);
}

// One thread per 50-symbol group, its symbols in 25 registers (two 16-bit
// loads per symbol and pass before).  Costs of all tables are packed in 10-bit
// fields of one 64-bit word per symbol (50 * 17 < 1024), so a group's six
// costs are one 64-bit sum.  The frequent symbols (RUNA, RUNB and the first
// MTF indices) are counted in byte fields of a register: shared-memory adds,
// about 1.5 a cycle and SM, bound the rest.
// grid.y == 2 (the learned form's second passes): y = 1 runs, for the
// learned blocks, the plain selector's second pass over its first-pass
// tables (len2) into sel2 / rfreq2, beside y = 0's pass over len.
// list: the group tiles to run (blockIdx.x-th entry), or nullptr for all.
constexpr int kSymRegs = kGroupSize / 2;
constexpr int kPadSym = kMaxAlpha;       // fills the block's last group: costs and counts nothing
constexpr int kFreqRow = kMaxAlpha + 2;

__global__ void __launch_bounds__(kGroupTile) k_huff_select(SlabDev d, int which, int round,
                                                            const int32_t *list) {
  __shared__ __align__(16) uint32_t sy[kGroupTile * kSymRegs];  // two symbols per word
  __shared__ uint64_t plen[kMaxAlpha + 1];
  __shared__ int rf[kMaxGroups * kFreqRow];
  const int gt = list ? list[blockIdx.x] : (int)blockIdx.x;
  const int b = d.gt_block[gt];
  const int g0 = d.gt_first[gt];
  const int nsel = d.n_sel[b];
  const bool second = blockIdx.y == 1;
  if (g0 >= nsel) return;
  if (second ? !d.learned[b] : !serves(d, b, which, round)) return;
  const uint8_t *len_src = second ? d.len2 : d.len;
  uint8_t *sel_dst = second ? d.sel2 : d.sel;
  int32_t *rf_dst = second ? d.rfreq2 : d.rfreq;
  const int ng_here = min(kGroupTile, nsel - g0);
  const int s = d.s[b];
  const int ngrp = d.n_groups[b];
  const int alpha = d.n_in_use[b] + 2;
  const int64_t off = d.off[b];
  const int sym0 = g0 * kGroupSize;
  const int nsym = min(s, (g0 + ng_here) * kGroupSize) - sym0;
  const uint8_t *len = len_src + (size_t)b * kMaxGroups * kMaxAlpha;
  // a tile's symbols start on a 16-byte boundary (off is a multiple of kTile,
  // 128 groups are 12,800 bytes); the buffer has slack past a block's end
  const uint4 *src = reinterpret_cast<const uint4 *>(d.rle2 + off + sym0);
  for (int i = threadIdx.x; i < (nsym + 7) / 8; i += blockDim.x)
    reinterpret_cast<uint4 *>(sy)[i] = src[i];
  for (int v = threadIdx.x; v <= kMaxAlpha; v += blockDim.x) {
    uint64_t p = 0;
    if (v < alpha)
      for (int t = 0; t < ngrp; t++) p |= (uint64_t)len[t * kMaxAlpha + v] << (10 * t);
    plen[v] = p;
  }
  for (int i = threadIdx.x; i < kMaxGroups * kFreqRow; i += blockDim.x) rf[i] = 0;
  __syncthreads();
  const int g = threadIdx.x;
  if (g < ng_here) {
    const int n = min(kGroupSize, nsym - g * kGroupSize);
    uint32_t v2[kSymRegs];
    uint64_t cost = 0;
#pragma unroll
    for (int i = 0; i < kSymRegs; i++) {
      v2[i] = sy[g * kSymRegs + i];
      if (n < kGroupSize) {
        if (2 * i >= n) v2[i] = kPadSym | kPadSym << 16;
        else if (2 * i + 1 >= n) v2[i] = (v2[i] & 0xffffu) | kPadSym << 16;
      }
      cost += plen[v2[i] & 0xffffu] + plen[v2[i] >> 16];
    }
    uint32_t bc = 0xFFFFFFFFu;
    int bt = -1;
    for (int t = 0; t < ngrp; t++) {
      uint32_t c = (uint32_t)(cost >> (10 * t)) & 1023u;
      if (c < bc) {
        bc = c;
        bt = t;
      }
    }
    sel_dst[off / 32 + g0 + g] = (uint8_t)bt;
    uint64_t hot = 0;  // byte v: symbols v < 8 (at most 50)
    int *rft = rf + bt * kFreqRow;
#pragma unroll
    for (int i = 0; i < kSymRegs; i++) {
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const uint32_t v = q ? v2[i] >> 16 : v2[i] & 0xffffu;
        if (v < 8) hot += 1ull << (8 * v);
        else atomicAdd(&rft[v], 1);
      }
    }
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const int c = (int)((hot >> (8 * v)) & 0xffu);
      if (c) atomicAdd(&rft[v], c);
    }
  }
  __syncthreads();
  int32_t *rfreq = rf_dst + (size_t)b * kMaxGroups * kMaxAlpha;
  for (int t = 0; t < ngrp; t++)
    for (int v = threadIdx.x; v < alpha; v += blockDim.x) {
      const int c = rf[t * kFreqRow + v];
      if (c) atomicAdd(&rfreq[t * kMaxAlpha + v], c);
    }
}

// bzip2's length-limited Huffman lengths (src/compression/huffman.cu:13-124),
// one warp per block: lane t runs table t's heap (a block's tables share
// its alphabet size, so the lanes' heaps have equal sizes at every step and
// stay in step), so the warp issues about one heap's instructions for all
// six.  Heap entries carry their node's weight in the high half (weight << 32
// | node); comparisons use the weight half only, with the reference's strict
// '<', so ties resolve exactly as there: every step leaves the heap in the
// reference's state.
// The chain of heap steps is the kernel's time, so a step is made short.  A
// sift down always follows the lighter children, so the path to the bottom is
// found first, two levels per load, then its entries are compared and written
// all at once (the weights along a path do not fall, so the entries that move up
// are those not heavier than the moved one).  A sift up knows its path from the
// start.  Slots past the heap hold an infinite weight, so neither tests the
// heap's size.  One entry after another, a launch took 295 us for 258 symbols;
// this way 144 us, at about 340 instructions per merge.
// All lanes then walk the parent links for the code lengths, six tables at a
// time.
constexpr int kHeapRow = 266;  // entries per table: 16-byte rows, lanes on different banks
constexpr int kNodeN = kMaxAlpha * 2;
constexpr uint32_t kInfWeight = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t hw(uint64_t e) { return (uint32_t)(e >> 32); }

__device__ __forceinline__ uint64_t pick(bool c, uint64_t x, uint64_t y) { return c ? x : y; }

// Removes the top of a heap of n entries (n is the same for all lanes, n <
// 2^(L + 1)).  Two levels per step: a node's children and all its
// grandchildren are loaded at once, so the path to the bottom by the lighter
// children takes half as many waits.  Free of branches: entries of the path that
// do not change are written again.
template <int L>
__device__ __forceinline__ uint64_t heap_pop(uint64_t *heap, int n) {
  const uint64_t top = heap[1], tmp = heap[n];
  heap[n] = (uint64_t)kInfWeight << 32;
  uint32_t node[L + 1];
  uint64_t ch[L];  // the path's entries
  node[0] = 1;
  auto pair = [&](uint32_t at) { return *reinterpret_cast<const ulonglong2 *>(&heap[at]); };
#pragma unroll
  for (int l = 0; l < L; l += 2) {
    const uint32_t v = node[l];
    const ulonglong2 c = pair(2 * v);
    const bool r = hw(c.y) < hw(c.x);
    ch[l] = pick(r, c.y, c.x);
    node[l + 1] = 2 * v + r;
    if (l + 1 < L) {
      const ulonglong2 x = pair(4 * v), y = pair(4 * v + 2);
      const bool rx = hw(x.y) < hw(x.x), ry = hw(y.y) < hw(y.x);
      const uint64_t mx = pick(rx, x.y, x.x), my = pick(ry, y.y, y.x);
      ch[l + 1 < L ? l + 1 : l] = pick(r, my, mx);
      node[l + 2 <= L ? l + 2 : L] = 2 * node[l + 1] + (r ? ry : rx);
    }
  }
  const uint32_t tw = hw(tmp);
  bool here = true;
#pragma unroll
  for (int l = 0; l <= L; l++) {
    const bool up = l < L && hw(ch[l < L ? l : 0]) <= tw;
    heap[node[l]] = pick(up, ch[l < L ? l : 0], pick(here, tmp, ch[l > 0 ? l - 1 : 0]));
    here = up;
  }
  return top;
}

// Adds e at slot z (the same for all lanes, z < 2^(L + 1)).
template <int L>
__device__ __forceinline__ void heap_push(uint64_t *heap, int z, uint64_t e) {
  uint64_t anc[L];
#pragma unroll
  for (int l = 0; l < L; l++) anc[l] = heap[z >> (l + 1)];  // past the root: entry 0, weight 0
  const uint32_t ew = hw(e);
  bool here = true;
#pragma unroll
  for (int l = 0; l <= L; l++) {
    // slot z >> l's new entry
    const bool down = l < L && ew < hw(anc[l < L ? l : 0]);
    const uint64_t nv = pick(down, anc[l < L ? l : 0], pick(here, e, anc[l > 0 ? l - 1 : 0]));
    here = down;
    if ((z >> l) >= 1) heap[z >> l] = nv;
  }
}

// The node that joins p1 and p2, as a heap entry.
__device__ __forceinline__ uint64_t merged(uint64_t p1, uint64_t p2, int node, int16_t *parent) {
  const uint32_t w1 = hw(p1), w2 = hw(p2);
  parent[(uint32_t)p1] = parent[(uint32_t)p2] = (int16_t)node;
  parent[node] = -1;
  const uint32_t d1 = w1 & 0xff, d2 = w2 & 0xff;
  const uint32_t wn = ((w1 & 0xffffff00u) + (w2 & 0xffffff00u)) | (1 + (d1 > d2 ? d1 : d2));
  return ((uint64_t)wn << 32) | (uint32_t)node;
}

// Merges the two lightest nodes while the heap has more than `down_to`
// entries.  Node numbers count up from n_nodes.
template <int L>
__device__ __forceinline__ void merge_down(uint64_t *heap, int16_t *parent, int down_to, int &n,
                                           int &n_nodes) {
#pragma unroll 1
  while (n > down_to) {
    const uint64_t p1 = heap_pop<L>(heap, n);
    const uint64_t p2 = heap_pop<L>(heap, n - 1);
    const uint64_t e = merged(p1, p2, ++n_nodes, parent);
    heap_push<L>(heap, n - 1, e);
    n--;
  }
}

// The reference's steps one entry after another, for heaps of 256 entries and
// more and for weights that may pass 32 bits.
__device__ __forceinline__ uint64_t heap_pop_slow(uint64_t *heap, int n) {
  const uint64_t top = heap[1], tmp = heap[n];
  heap[n] = (uint64_t)kInfWeight << 32;
  n--;
  int zz = 1;
  for (;;) {
    int yy = zz << 1;
    if (yy > n) break;
    const ulonglong2 pr = *reinterpret_cast<const ulonglong2 *>(&heap[yy]);
    uint64_t c = pr.x;
    if (yy < n && hw(pr.y) < hw(pr.x)) {
      yy++;
      c = pr.y;
    }
    if (hw(tmp) < hw(c)) break;
    heap[zz] = c;
    zz = yy;
  }
  if (n > 0) heap[zz] = tmp;
  return top;
}
__device__ __forceinline__ void heap_push_slow(uint64_t *heap, int z, uint64_t e) {
  uint64_t up = heap[z >> 1];
  while (hw(e) < hw(up)) {
    heap[z] = up;
    z >>= 1;
    up = heap[z >> 1];
  }
  heap[z] = e;
}

// split (the learned form, grid.y = 2): y = 0 builds every block's tables
// into len, y = 1 the learned blocks' plain-selector tables into len2.
// split == 1 (first build): y = 0 from the counts of the first pass (the
// MLP's counts for learned blocks), y = 1 from the first plain pass's counts.
// split == 2 (second build): y = 0 from rfreq, y = 1 from rfreq2.
__global__ void __launch_bounds__(32) k_huff_lengths(SlabDev d, int which, int round, int split) {
  __shared__ __align__(16) uint64_t heap_s[kMaxGroups][kHeapRow];
  __shared__ int32_t leafw_s[kMaxGroups][kMaxAlpha + 1];
  __shared__ int16_t parent_s[kMaxGroups][kNodeN];
  const int b = blockIdx.x;
  const int ln = lane_id();
  const int ngrp = d.n_groups[b];
  const int32_t *rf_base = d.rfreq;
  uint8_t *len_base = d.len;
  if (split) {
    if (blockIdx.y == 0) {
      if (split == 1 && d.learned[b]) rf_base = d.rfreq_m;
    } else {
      if (!d.learned[b]) return;
      len_base = d.len2;
      if (split == 2) rf_base = d.rfreq2;
    }
  } else if (!serves(d, b, which, round)) {
    return;
  }
  const int alpha = d.n_in_use[b] + 2;
  for (int t = 0; t < ngrp; t++) {
    const int32_t *freq = rf_base + ((size_t)b * kMaxGroups + t) * kMaxAlpha;
    for (int i = ln; i < alpha; i += 32) {
      const int f = freq[i];
      leafw_s[t][i + 1] = (f == 0 ? 1 : f) << 8;
    }
  }
  __syncwarp();
  const bool wide = d.s[b] >= (1 << 24) - 512;  // weights may pass 32 bits
  unsigned pending = (1u << ngrp) - 1u;  // tables whose lengths are not final yet
  while (pending) {
    for (int t = 0; t < ngrp; t++)
      for (int i = ln; i < kHeapRow; i += 32) heap_s[t][i] = i ? (uint64_t)kInfWeight << 32 : 0ull;
    __syncwarp();
    const bool run = (pending >> ln) & 1u;
    uint64_t *heap = heap_s[run ? ln : 0];
    int16_t *parent = parent_s[run ? ln : 0];
    int n = alpha, n_nodes = alpha;
    if (run) {
      const int32_t *leafw = leafw_s[ln];
      for (int i = 1; i <= alpha; i++) {
        const uint64_t e = ((uint64_t)(uint32_t)leafw[i] << 32) | (uint32_t)i;
        parent[i] = -1;
        if (wide || i > 255) heap_push_slow(heap, i, e);
        else if (i > 127) heap_push<7>(heap, i, e);
        else if (i > 31) heap_push<6>(heap, i, e);
        else heap_push<4>(heap, i, e);
      }
      while (n > (wide ? 1 : 255)) {
        const uint64_t p1 = heap_pop_slow(heap, n);
        const uint64_t p2 = heap_pop_slow(heap, n - 1);
        const uint64_t e = merged(p1, p2, ++n_nodes, parent);
        heap_push_slow(heap, n - 1, e);
        n--;
      }
    }
    __syncwarp();
    if (run && !wide) {
      merge_down<7>(heap, parent, 127, n, n_nodes);
      merge_down<6>(heap, parent, 63, n, n_nodes);
      merge_down<5>(heap, parent, 31, n, n_nodes);
      merge_down<4>(heap, parent, 15, n, n_nodes);
      merge_down<3>(heap, parent, 1, n, n_nodes);
    }
    __syncwarp();
    bool too_long[kMaxGroups] = {};
    for (int i = ln + 1; i <= alpha; i += 32) {
      int j[kMaxGroups], k[kMaxGroups];
#pragma unroll
      for (int t = 0; t < kMaxGroups; t++) {
        j[t] = 0;
        k[t] = (pending >> t) & 1u ? (int)parent_s[t][i] : -1;
      }
      for (;;) {
        bool more = false;
#pragma unroll
        for (int t = 0; t < kMaxGroups; t++) {
          if (k[t] >= 0) {
            j[t]++;
            k[t] = parent_s[t][k[t]];
            more = true;
          }
        }
        if (!more) break;
      }
#pragma unroll
      for (int t = 0; t < kMaxGroups; t++) {
        if ((pending >> t) & 1u) {
          len_base[((size_t)b * kMaxGroups + t) * kMaxAlpha + i - 1] = (uint8_t)j[t];
          too_long[t] |= j[t] > kMaxCodeLen;
        }
      }
    }
    unsigned redo = 0;
#pragma unroll
    for (int t = 0; t < kMaxGroups; t++) {
      if (__any_sync(0xffffffffu, too_long[t])) {
        redo |= 1u << t;
        for (int i = ln + 1; i <= alpha; i += 32) {
          int j = leafw_s[t][i] >> 8;
          j = 1 + (j / 2);
          leafw_s[t][i] = j << 8;
        }
      }
    }
    __syncwarp();
    pending = redo;
  }
}

// Predicted coded size of a block's selection (bits): payload from the
// per-table counts and lengths, plus the table headers (5-bit start, 2 bits
// per unit of length change, 1 terminator bit per symbol).  One warp.
__device__ int64_t predicted_bits(const SlabDev &d, int b, const uint8_t *len_base,
                                  const int32_t *rf_base) {
  const int ng = d.n_groups[b];
  const int alpha = d.n_in_use[b] + 2;
  const int32_t *rf = rf_base + (size_t)b * kMaxGroups * kMaxAlpha;
  const uint8_t *len = len_base + (size_t)b * kMaxGroups * kMaxAlpha;
  int64_t e = 0;
  for (int t = 0; t < ng; t++)
    for (int v = lane_id(); v < alpha; v += 32) {
      const int l = len[t * kMaxAlpha + v];
      const int p = v ? len[t * kMaxAlpha + v - 1] : l;
      e += (int64_t)rf[t * kMaxAlpha + v] * l + 2 * abs(l - p) + 1;
    }
  for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  return e + 5 * ng;
}

// Learned form, after the second passes: a learned block whose predicted
// size exceeds that of the plain selector's first two passes takes the
// plain two-pass selection (sel2, len2) instead.  A warp for each prediction,
// the CTA for the copy (by one warp it took 77 us a slab).
__global__ void __launch_bounds__(256) k_huff_judge(SlabDev d) {
  __shared__ int64_t bits[2];
  const int b = blockIdx.x;
  if (!d.learned[b]) return;
  const int w = warp_id();
  if (w < 2) {
    const int64_t e = predicted_bits(d, b, w ? d.len2 : d.len, w ? d.rfreq2 : d.rfreq);
    if (lane_id() == 0) bits[w] = e;
  }
  __syncthreads();
  if (bits[0] <= bits[1]) return;
  const size_t tb = (size_t)b * kMaxGroups * kMaxAlpha;
  for (int i = threadIdx.x; i < kMaxGroups * kMaxAlpha; i += 256) d.len[tb + i] = d.len2[tb + i];
  const int64_t s0 = d.off[b] / 32;
  const int nsel = d.n_sel[b];
  for (int g = threadIdx.x; g < nsel; g += 256) d.sel[s0 + g] = d.sel2[s0 + g];
  if (threadIdx.x == 0) {
    d.learned[b] = 0;
    d.plain_left[b] = 0;
  }
}

// Canonical codes (src/compression/huffman.cu:135-146,352-362): for each
// length from the shortest to the longest, the symbols of that length in
// symbol order take consecutive codes; the next length starts at twice the
// running code.  One warp per table: lane l holds symbols l, l + 32, ...; a
// ballot per 32 symbols gives each symbol its place among that length's.
constexpr int kCodeSlots = (kMaxAlpha + 31) / 32;  // 9

__global__ void __launch_bounds__(kMaxGroups * 32) k_huff_codes(SlabDev d) {
  const int b = blockIdx.x;
  const int t = warp_id();
  const int ln = lane_id();
  if (t >= d.n_groups[b]) return;
  const int alpha = d.n_in_use[b] + 2;
  const uint8_t *len = d.len + ((size_t)b * kMaxGroups + t) * kMaxAlpha;
  int32_t *code = d.code + ((size_t)b * kMaxGroups + t) * kMaxAlpha;
  uint32_t *both = d.len_code + (size_t)b * kLenCode + t * kMaxAlpha;  // for the payload
  int lv[kCodeSlots];
  int mn = 32, mx = 0;
#pragma unroll
  for (int q = 0; q < kCodeSlots; q++) {
    const int v = 32 * q + ln;
    lv[q] = v < alpha ? (int)len[v] : -1;
    if (v < alpha) {
      mn = min(mn, lv[q]);
      mx = max(mx, lv[q]);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  const unsigned below = (1u << ln) - 1u;
  int vec = 0;
  for (int l = mn; l <= mx; l++) {
#pragma unroll
    for (int q = 0; q < kCodeSlots; q++) {
      const bool hit = lv[q] == l;
      const unsigned bal = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int c = vec + __popc(bal & below);
        code[32 * q + ln] = c;
        both[32 * q + ln] = (uint32_t)l << 24 | (uint32_t)c;
      }
      vec += __popc(bal);
    }
    vec <<= 1;
  }
}

}  // namespace

namespace {
void select_pass(const SlabDev &d, int which, int round, cudaStream_t st) {
  BZ_CUDA(cudaMemsetAsync(d.rfreq, 0, sizeof(int32_t) * kMaxGroups * kMaxAlpha * d.nblocks, st));
  const int nlive = live_group_tiles(d, st);
  const int grid = nlive >= 0 ? nlive : d.n_group_tiles;
  if (grid <= 0) return;
  k_huff_select<<<grid, kGroupTile, 0, st>>>(d, which, round, nlive >= 0 ? d.vg_list : nullptr);
  BZ_LAUNCH_CHECK();
}
void lengths_pass(const SlabDev &d, int which, int round, cudaStream_t st) {
  k_huff_lengths<<<d.nblocks, 32, 0, st>>>(d, which, round, 0);
  BZ_LAUNCH_CHECK();
}
}  // namespace

// Plain form (the reference's): initial tables, then 4 passes of selection
// and code lengths.
// Learned form, blocks with six tables: the MLP's choice gives the first
// tables, one exact selection pass and code lengths follow.  Beside them the
// plain selector runs its first two passes (initial tables, then its
// first-pass tables); that is the judge: a block whose learned tables predict
// a larger size takes the plain two-pass selection.  The judge thus costs no
// launch of its own, and the stage runs two rounds of selection and code
// lengths where the plain form runs four.  Blocks with fewer tables run the
// plain passes in the same launches (launches that serve none of a slab's
// blocks return at once).
void stage_huffman(const SlabDev &d, cudaStream_t st, const uint8_t *learned, int plain_passes,
                   uint8_t *mlp_sel_out, size_t mlp_sel_bytes) {
  k_huff_init<<<d.nblocks, 32, 0, st>>>(d, learned ? 1 : 0);
  BZ_LAUNCH_CHECK();
  if (!learned) {
    for (int it = 0; it < plain_passes; it++) {
      select_pass(d, kAll, 0, st);
      lengths_pass(d, kAll, 0, st);
    }
  } else {
    const size_t rf_bytes = sizeof(int32_t) * kMaxGroups * kMaxAlpha * d.nblocks;
    BZ_CUDA(cudaMemsetAsync(d.rfreq_m, 0, rf_bytes, st));
    select_pass(d, kAll, 0, st);  // the plain selector's first pass, every block
    mlp::launch_select(d, learned, nullptr, nullptr, d.rfreq_m, st);
    if (mlp_sel_out)
      BZ_CUDA(cudaMemcpyAsync(mlp_sel_out, d.sel, mlp_sel_bytes, cudaMemcpyDeviceToDevice, st));
    k_huff_lengths<<<dim3(d.nblocks, 2), 32, 0, st>>>(d, kAll, 0, 1);
    BZ_LAUNCH_CHECK();
    // second passes, side by side: every block over its tables (the plain
    // blocks' second pass, the learned tables' exact pass) and, for learned
    // blocks, the plain selector's second pass over its first-pass tables
    BZ_CUDA(cudaMemsetAsync(d.rfreq, 0, rf_bytes, st));
    BZ_CUDA(cudaMemsetAsync(d.rfreq2, 0, rf_bytes, st));
    {
      const int nlive = live_group_tiles(d, st);
      const int grid = nlive >= 0 ? nlive : d.n_group_tiles;
      if (grid > 0) {
        k_huff_select<<<dim3(grid, 2), kGroupTile, 0, st>>>(d, kAll, 0,
                                                          nlive >= 0 ? d.vg_list : nullptr);
        BZ_LAUNCH_CHECK();
      }
    }
    k_huff_lengths<<<dim3(d.nblocks, 2), 32, 0, st>>>(d, kAll, 0, 2);
    BZ_LAUNCH_CHECK();
    k_huff_judge<<<d.nblocks, 256, 0, st>>>(d);
    BZ_LAUNCH_CHECK();
    // plain blocks (fewer than six tables) finish their four passes
    for (int r = 0; r < kIters - 2; r++) {
      select_pass(d, kPlainRound, r, st);
      lengths_pass(d, kPlainRound, r, st);
    }
  }
  k_huff_codes<<<d.nblocks, kMaxGroups * 32, 0, st>>>(d);
  BZ_LAUNCH_CHECK();
}

}  // namespace bz2g
