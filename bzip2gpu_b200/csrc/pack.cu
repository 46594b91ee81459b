// Block headers, payload bit packing and stream placement, for a slab.
//
// Reference: src/compression/huffman_encode.cu:15-143 (per-symbol code from
// the group's table, exclusive scan of code lengths to bit offsets, MSB-first
// placement) and src/compression/compress.cu:119-137,284-375 (selector MTF
// and the block header fields).  Here the block header and payload are written
// straight to their final bit position in the .bz2 stream: the output is an
// array of big-endian 32-bit words (so memory order is stream byte order),
// zeroed first and OR-ed into, since neighbouring blocks share edge words.
#include "engine.h"

namespace bz2g {

namespace {

__device__ __forceinline__ uint32_t bswap32(uint32_t w) { return __byte_perm(w, 0, 0x0123); }

// MSB-first bit writer into zeroed big-endian words.
struct BitSink {
  uint32_t *out;
  int64_t word;
  uint64_t acc;
  int n;
  __device__ void init(uint32_t *o, int64_t bit) {
    out = o;
    word = bit >> 5;
    acc = 0;
    n = (int)(bit & 31);
  }
  __device__ __forceinline__ void put(uint32_t v, int nb) {
    acc = (acc << nb) | v;
    n += nb;
    if (n >= 32) {
      uint32_t w = (uint32_t)(acc >> (n - 32));
      atomicOr(out + word, bswap32(w));
      word++;
      n -= 32;
    }
  }
  __device__ void flush() {
    if (n > 0) atomicOr(out + word, bswap32((uint32_t)(acc << (32 - n))));
    n = 0;
  }
};

// Per block: selector MTF (src/compression/compress.cu:119-137) and the
// header size.  256 threads split the selectors into chunks; the MTF list at
// a chunk's start is the tables ordered by their last use before it (most
// recent first, unused ones in index order), read off a prefix max over the
// threads of each table's last position, so every chunk then runs its MTF on
// its own.
constexpr int kHdrThreads = 256;

__device__ __forceinline__ int sel_chunk(int nsel, int *a, int *e) {
  const int per = (nsel + kHdrThreads - 1) / kHdrThreads;
  *a = min(nsel, (int)threadIdx.x * per);
  *e = min(nsel, *a + per);
  return per;
}

// Bits of a table's delta-coded lengths (5-bit start, 2 bits per unit of
// change, 1 terminator bit per symbol), by one warp.
__device__ int table_bits(const uint8_t *len, int alpha) {
  int e = 0;
  for (int v = lane_id(); v < alpha; v += 32) {
    const int l = len[v];
    e += 2 * abs(l - (v ? (int)len[v - 1] : l)) + 1;
  }
  return 5 + __reduce_add_sync(0xffffffffu, e);
}

__device__ int used_ranges(const uint32_t *pres) {
  int r = 0;
  for (int q = 0; q < 16; q++) r += ((pres[q >> 1] >> ((q & 1) * 16)) & 0xffffu) != 0;
  return r;
}

__global__ void __launch_bounds__(kHdrThreads) k_sel_mtf_hdr(SlabDev d) {
  __shared__ int scratch[40];
  __shared__ int tbits[kMaxGroups];
  __shared__ int wl[kHdrThreads / 32][kMaxGroups];
  const int b = blockIdx.x;
  const int ngrp = d.n_groups[b];
  const int nsel = d.n_sel[b];
  const int alpha = d.n_in_use[b] + 2;
  const uint8_t *sel = d.sel + d.off[b] / 32;
  uint8_t *smtf = d.sel_mtf + d.off[b] / 32;
  int a, e;
  sel_chunk(nsel, &a, &e);
  int last[kMaxGroups];
#pragma unroll
  for (int t = 0; t < kMaxGroups; t++) last[t] = -1;
  for (int i = a; i < e; i++) {
    const int v = sel[i];
#pragma unroll
    for (int t = 0; t < kMaxGroups; t++)
      if (v == t) last[t] = i;
  }
  // the tables' last uses before this thread's chunk
  int prev[kMaxGroups];
#pragma unroll
  for (int t = 0; t < kMaxGroups; t++) {
    const int inc = warp_incl_max(last[t]);
    prev[t] = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane_id() == 0) prev[t] = -1;
    if (lane_id() == 31) wl[warp_id()][t] = inc;
  }
  if ((int)warp_id() < ngrp) {
    const int tb = table_bits(d.len + ((size_t)b * kMaxGroups + warp_id()) * kMaxAlpha, alpha);
    if (lane_id() == 0) tbits[warp_id()] = tb;
  }
  __syncthreads();
  for (int w = 0; w < (int)warp_id(); w++) {
#pragma unroll
    for (int t = 0; t < kMaxGroups; t++) prev[t] = max(prev[t], wl[w][t]);
  }
  // starting list, nibble r = table at position r: used tables by last use
  // (latest first), then unused ones
  uint32_t lst = 0;
#pragma unroll
  for (int t = 0; t < kMaxGroups; t++) {
    const int key = prev[t] >= 0 ? prev[t] : -1 - t;
    int r = 0;
#pragma unroll
    for (int u = 0; u < kMaxGroups; u++) {
      const int ku = prev[u] >= 0 ? prev[u] : -1 - u;
      r += u < ngrp && ku > key;
    }
    if (t < ngrp) lst |= (uint32_t)t << (4 * r);
  }
  // positions past the last table hold a value no selector has
  for (int r = ngrp; r < 8; r++) lst |= 15u << (4 * r);
  int unary = 0;
  for (int i = a; i < e; i++) {
    const uint32_t v = sel[i];
    // the lowest zero nibble of x is v's position
    const uint32_t x = lst ^ (v * 0x11111111u);
    const int j = (__ffs((x - 0x11111111u) & ~x & 0x88888888u) - 1) >> 2;
    const uint32_t low = (1u << (4 * j)) - 1u;
    lst = (lst & ~((low << 4) | 0xFu)) | ((lst & low) << 4) | v;
    smtf[i] = (uint8_t)j;
    unary += j + 1;
  }
  int total_unary;
  block_excl_sum(unary, scratch, &total_unary);
  if (threadIdx.x == 0) {
    int64_t tb = 0;
    for (int t = 0; t < ngrp; t++) tb += tbits[t];
    const int ranges = used_ranges(d.present + b * 8);
    d.hdr_bits[b] = 48 + 32 + 1 + 24 + 16 + 16 * ranges + 3 + 15 + (int64_t)total_unary + tb;
  }
}

// A group tile's symbols, two per word, by 16-byte loads (a tile starts on a
// 16-byte boundary: off is a multiple of kTile, 128 groups are 12,800 bytes;
// the buffer has slack past a block's end).  Group g's are at 25 g: threads
// reading their own groups meet on no bank.
constexpr int kSymWords = kGroupSize / 2;
__device__ __forceinline__ void load_groups(const SlabDev &d, int64_t off, int g0, int s,
                                            uint32_t *sy) {
  const int sym0 = g0 * kGroupSize;
  const int n = min(s - sym0, kGroupTile * kGroupSize);
  const uint4 *src = reinterpret_cast<const uint4 *>(d.rle2 + off + sym0);
  for (int i = threadIdx.x; i < (n + 7) / 8; i += kGroupTile)
    reinterpret_cast<uint4 *>(sy)[i] = src[i];
}

// Payload bits per 50-symbol group; exclusive offsets within the group tile.
__global__ void __launch_bounds__(kGroupTile) k_pay_bits(SlabDev d, const int32_t *list) {
  __shared__ uint32_t scratch[8];
  __shared__ __align__(16) uint32_t sy[kGroupTile * kSymWords];
  __shared__ __align__(4) uint8_t len[kMaxGroups * kMaxAlpha];
  const int gt = list ? list[blockIdx.x] : (int)blockIdx.x;
  const int b = d.gt_block[gt];
  const int g0 = d.gt_first[gt];
  const int nsel = d.n_sel[b];
  if (g0 >= nsel) {
    if (threadIdx.x == 0) d.gt_bits[gt] = 0;
    return;
  }
  const int s = d.s[b];
  const int64_t off = d.off[b];
  load_groups(d, off, g0, s, sy);
  static_assert(kMaxGroups * kMaxAlpha % 4 == 0, "a block's lengths are whole words");
  for (int i = threadIdx.x; i < kMaxGroups * kMaxAlpha / 4; i += kGroupTile)
    reinterpret_cast<uint32_t *>(len)[i] =
        reinterpret_cast<const uint32_t *>(d.len + (size_t)b * kMaxGroups * kMaxAlpha)[i];
  __syncthreads();
  const int g = g0 + threadIdx.x;
  uint32_t bits = 0;
  if (g < nsel) {
    const uint8_t *lt = len + d.sel[off / 32 + g] * kMaxAlpha;
    const uint32_t *my = sy + threadIdx.x * kSymWords;
    const int n = min(kGroupSize, s - g * kGroupSize);
    for (int i = 0; i < n / 2; i++) {
      const uint32_t v = my[i];
      bits += lt[v & 0xffffu] + lt[v >> 16];
    }
    if (n & 1) bits += lt[my[n / 2] & 0xffffu];
  }
  uint32_t tot;
  uint32_t ex = block_excl_sum(bits, scratch, &tot);
  if (g < nsel) d.grp_bits[off / 32 + g] = ex;
  if (threadIdx.x == 0) d.gt_bits[gt] = tot;
}

// Per block: exclusive sum over its group tiles; payload bits.
__global__ void __launch_bounds__(256) k_pay_block(SlabDev d) {
  __shared__ uint32_t scratch[40];
  const int b = blockIdx.x;
  // the group tiles that hold groups (the others are not run)
  const int nsel = d.n_sel[b];
  const int t0 = d.gt_begin[b];
  const int nt = min(d.gt_begin[b + 1] - t0, (nsel + kGroupTile - 1) / kGroupTile);
  int64_t carry = 0;
  for (int base = 0; base < nt; base += 256) {
    int k = base + threadIdx.x;
    uint32_t v = k < nt ? d.gt_bits[t0 + k] : 0;
    uint32_t tot;
    uint32_t ex = block_excl_sum(v, scratch, &tot);
    if (k < nt) d.gt_bits[t0 + k] = (uint32_t)(carry + ex);
    carry += tot;
  }
  if (threadIdx.x == 0) d.pay_bits[b] = carry;
}

__global__ void __launch_bounds__(256) k_block_starts(SlabDev d, int64_t slab_start) {
  __shared__ int64_t scratch[40];
  int64_t run = slab_start;
  for (int b0 = 0; b0 < d.nblocks; b0 += 256) {
    const int b = b0 + threadIdx.x;
    const int64_t bits = b < d.nblocks ? d.hdr_bits[b] + d.pay_bits[b] : 0;
    int64_t tot;
    const int64_t at = run + block_excl_sum(bits, scratch, &tot);
    if (b < d.nblocks) d.blk_start[b] = at;
    run += tot;
  }
}

// Block header at its stream position (src/compression/compress.cu:290-353).
// Thread 0 writes the fixed fields; every thread writes the unary selector
// codes of its chunk at an offset from a block scan; warp t < nGroups writes
// table t's delta-coded lengths, a symbol per lane at offsets from warp scans
// (a thread per table took 60 us).
__global__ void __launch_bounds__(kHdrThreads) k_write_header(SlabDev d, int64_t w0) {
  __shared__ int scratch[40];
  __shared__ int tbits[kMaxGroups];
  const int b = blockIdx.x;
  const int ngrp = d.n_groups[b];
  const int nsel = d.n_sel[b];
  const int alpha = d.n_in_use[b] + 2;
  const uint32_t *pres = d.present + b * 8;
  const uint8_t *smtf = d.sel_mtf + d.off[b] / 32;
  const int ranges = used_ranges(pres);
  const int64_t fixed = 48 + 32 + 1 + 24 + 16 + 16 * ranges + 3 + 15;
  const int64_t base = d.blk_start[b] - w0 * 32;
  if (threadIdx.x == 0) {
    BitSink w;
    w.init(d.out, base);
    w.put(0x314159u, 24);
    w.put(0x265359u, 24);
    w.put(d.crc[b], 32);
    w.put(0, 1);
    w.put((uint32_t)d.orig_ptr[b], 24);
    uint32_t l1 = 0;
    for (int r = 0; r < 16; r++)
      if ((pres[r >> 1] >> ((r & 1) * 16)) & 0xffffu) l1 |= 1u << (15 - r);
    w.put(l1, 16);
    for (int r = 0; r < 16; r++) {
      uint32_t half = (pres[r >> 1] >> ((r & 1) * 16)) & 0xffffu;
      if (!half) continue;
      uint32_t l2 = 0;
      for (int q = 0; q < 16; q++)
        if ((half >> q) & 1u) l2 |= 1u << (15 - q);
      w.put(l2, 16);
    }
    w.put((uint32_t)ngrp, 3);
    w.put((uint32_t)nsel, 15);
    w.flush();
  }
  int a, e;
  sel_chunk(nsel, &a, &e);
  int mine = 0;
  for (int i = a; i < e; i++) mine += smtf[i] + 1;
  int total;
  const int off = block_excl_sum(mine, scratch, &total);
  if (e > a) {
    BitSink w;
    w.init(d.out, base + fixed + off);
    for (int i = a; i < e; i++) {
      const int j = smtf[i];
      w.put(((1u << j) - 1u) << 1, j + 1);
    }
    w.flush();
  }
  const int t = warp_id(), ln = lane_id();
  if (t < ngrp) {
    const int tb = table_bits(d.len + ((size_t)b * kMaxGroups + t) * kMaxAlpha, alpha);
    if (ln == 0) tbits[t] = tb;
  }
  __syncthreads();
  if (t < ngrp) {
    int64_t at = base + fixed + total;
    for (int u = 0; u < t; u++) at += tbits[u];
    const uint8_t *len = d.len + ((size_t)b * kMaxGroups + t) * kMaxAlpha;
    // nb <= 33 bits at stream bit p: at most two words
    auto place = [&](int64_t p, uint64_t v, int nb) {
      const uint64_t x = v << (64 - (int)(p & 31) - nb);
      const uint32_t hi = (uint32_t)(x >> 32), lo = (uint32_t)x;
      if (hi) atomicOr(d.out + (p >> 5), bswap32(hi));
      if (lo) atomicOr(d.out + (p >> 5) + 1, bswap32(lo));
    };
    if (ln == 0) place(at, len[0], 5);
    at += 5;
    for (int v0 = 0; v0 < alpha; v0 += 32) {
      const int v = v0 + ln;
      int nb = 0;
      uint64_t code = 0;
      if (v < alpha) {
        const int l = len[v], k = l - (v ? (int)len[v - 1] : l);
        // |k| steps of 10 (longer) or 11 (shorter), then a 0
        const int n2 = 2 * abs(k);
        const uint64_t ones = (1ull << n2) - 1ull;
        code = (k > 0 ? ones & 0xAAAAAAAAAAAAAAAAull : ones) << 1;
        nb = n2 + 1;
      }
      const int inc = warp_incl_sum(nb);
      if (code) place(at + inc - nb, code, nb);
      at += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

// Payload: one thread per 50-symbol group.  The tile's bits are assembled in
// shared memory (a thread's first and last word shared with its neighbours,
// the ones between its own) and copied out by whole words; only a tile's first
// and last word meet other tiles' bits (1 GiB: 0.88 ms with every word or-ed
// into device memory).
constexpr int kTileWords = kGroupTile * kGroupSize * kMaxCodeLen / 32 + 2;

__global__ void __launch_bounds__(kGroupTile) k_write_payload(SlabDev d, int64_t w0, const int32_t *list) {
  __shared__ __align__(16) uint32_t sy[kGroupTile * kSymWords];
  __shared__ __align__(16) uint32_t tab[kLenCode];  // len << 24 | code
  __shared__ uint32_t ob[kTileWords];
  __shared__ uint32_t s_bits;
  const int gt = list ? list[blockIdx.x] : (int)blockIdx.x;
  const int b = d.gt_block[gt];
  const int g0 = d.gt_first[gt];
  const int nsel = d.n_sel[b];
  if (g0 >= nsel) return;
  const int s = d.s[b];
  const int64_t off = d.off[b];
  const int ng = min(kGroupTile, nsel - g0);
  const int64_t start = d.blk_start[b] + d.hdr_bits[b] + d.gt_bits[gt] - w0 * 32;
  const uint32_t lead = (uint32_t)(start & 31);
  load_groups(d, off, g0, s, sy);
  for (int i = threadIdx.x; i < kLenCode / 4; i += kGroupTile)
    reinterpret_cast<uint4 *>(tab)[i] =
        reinterpret_cast<const uint4 *>(d.len_code + (size_t)b * kLenCode)[i];
  // the last group's offset bounds the words
  const uint32_t most = lead + d.grp_bits[off / 32 + g0 + ng - 1] + kGroupSize * kMaxCodeLen;
  for (int i = threadIdx.x; i < min((int)(most / 32 + 1), kTileWords); i += kGroupTile) ob[i] = 0;
  __syncthreads();
  const int g = g0 + threadIdx.x;
  if (g < nsel) {
    const uint32_t *tt = tab + d.sel[off / 32 + g] * kMaxAlpha;
    const uint32_t *my = sy + threadIdx.x * kSymWords;
    const int ns = min(kGroupSize, s - g * kGroupSize);
    uint32_t bit = lead + d.grp_bits[off / 32 + g];
    uint32_t word = bit >> 5;
    int n = (int)(bit & 31);
    bool mine = n == 0;  // no other thread's bits in this word
    uint64_t acc = 0;
    auto put = [&](uint32_t sym) {
      const uint32_t e = tt[sym];
      const int nb = (int)(e >> 24);
      acc = (acc << nb) | (e & 0xffffffu);
      n += nb;
      bit += nb;
      if (n >= 32) {
        const uint32_t w = (uint32_t)(acc >> (n - 32));
        if (mine) ob[word] = w;
        else atomicOr(&ob[word], w);
        mine = true;
        word++;
        n -= 32;
      }
    };
    for (int i = 0; i < ns / 2; i++) {
      const uint32_t v = my[i];
      put(v & 0xffffu);
      put(v >> 16);
    }
    if (ns & 1) put(my[ns / 2] & 0xffffu);
    if (n > 0) atomicOr(&ob[word], (uint32_t)(acc << (32 - n)));
    if ((int)threadIdx.x == ng - 1) s_bits = bit;
  }
  __syncthreads();
  const int nw = (int)((s_bits + 31) / 32);
  uint32_t *out = d.out + (start >> 5);
  for (int i = threadIdx.x; i < nw; i += kGroupTile) {
    const uint32_t v = bswap32(ob[i]);
    if (i == 0 || i == nw - 1) atomicOr(out + i, v);
    else out[i] = v;
  }
}

// Payload only, in the reference's word layout (word w = stream bits
// [32w, 32w+32), first bit in the MSB, host byte order), for one block.
__global__ void __launch_bounds__(kGroupTile) k_pack_words(SlabDev d, uint32_t *words, const int32_t *list) {
  const int gt = list ? list[blockIdx.x] : (int)blockIdx.x;
  const int b = d.gt_block[gt];
  const int g0 = d.gt_first[gt];
  const int nsel = d.n_sel[b];
  const int g = g0 + threadIdx.x;
  if (g >= nsel) return;
  const int s = d.s[b];
  const int64_t off = d.off[b];
  const int t = d.sel[off / 32 + g];
  const uint8_t *len = d.len + ((size_t)b * kMaxGroups + t) * kMaxAlpha;
  const int32_t *code = d.code + ((size_t)b * kMaxGroups + t) * kMaxAlpha;
  int64_t bit = (int64_t)d.gt_bits[gt] + d.grp_bits[off / 32 + g];
  int64_t word = bit >> 5;
  int n = (int)(bit & 31);
  uint64_t acc = 0;
  const int a = g * kGroupSize, e = min(a + kGroupSize, s);
  for (int i = a; i < e; i++) {
    int v = d.rle2[off + i];
    int nb = len[v];
    acc = (acc << nb) | (uint32_t)code[v];
    n += nb;
    if (n >= 32) {
      atomicOr(words + word, (uint32_t)(acc >> (n - 32)));
      word++;
      n -= 32;
    }
  }
  if (n > 0) atomicOr(words + word, (uint32_t)(acc << (32 - n)));
}

}  // namespace

// A group-tile kernel over the tiles that hold groups (every tile when the
// slab has no list).
template <typename F>
void launch_groups(const SlabDev &d, cudaStream_t st, F &&launch) {
  const int nlive = live_group_tiles(d, st);
  const int grid = nlive >= 0 ? nlive : d.n_group_tiles;
  if (grid <= 0) return;
  launch(grid, nlive >= 0 ? d.vg_list : nullptr);
}

void stage_sizes(const SlabDev &d, cudaStream_t st) {
  k_sel_mtf_hdr<<<d.nblocks, kHdrThreads, 0, st>>>(d);
  BZ_LAUNCH_CHECK();
  launch_groups(d, st, [&](int grid, const int32_t *list) {
    k_pay_bits<<<grid, kGroupTile, 0, st>>>(d, list);
  });
  BZ_LAUNCH_CHECK();
  k_pay_block<<<d.nblocks, 256, 0, st>>>(d);
  BZ_LAUNCH_CHECK();
}

void stage_sizes_payload_only(const SlabDev &d, cudaStream_t st) {
  launch_groups(d, st, [&](int grid, const int32_t *list) {
    k_pay_bits<<<grid, kGroupTile, 0, st>>>(d, list);
  });
  BZ_LAUNCH_CHECK();
  k_pay_block<<<d.nblocks, 256, 0, st>>>(d);
  BZ_LAUNCH_CHECK();
}

void stage_place(const SlabDev &d, int64_t slab_start_bit, int64_t w0, int64_t nwords,
                 cudaStream_t st) {
  BZ_CUDA(cudaMemsetAsync(d.out, 0, sizeof(uint32_t) * nwords, st));
  k_block_starts<<<1, 256, 0, st>>>(d, slab_start_bit);
  BZ_LAUNCH_CHECK();
  k_write_header<<<d.nblocks, kHdrThreads, 0, st>>>(d, w0);
  BZ_LAUNCH_CHECK();
  launch_groups(d, st, [&](int grid, const int32_t *list) {
    k_write_payload<<<grid, kGroupTile, 0, st>>>(d, w0, list);
  });
  BZ_LAUNCH_CHECK();
}

// Blocks at word-aligned places of their own in `arena` (d.blk_start already
// holds each block's first bit); zeroes arena words [w0, w0 + nwords) first.
void stage_place_arena(const SlabDev &d, uint32_t *arena, int64_t w0, int64_t nwords,
                       cudaStream_t st) {
  BZ_CUDA(cudaMemsetAsync(arena + w0, 0, sizeof(uint32_t) * nwords, st));
  SlabDev a = d;
  a.out = arena;
  k_write_header<<<a.nblocks, kHdrThreads, 0, st>>>(a, 0);
  BZ_LAUNCH_CHECK();
  launch_groups(a, st, [&](int grid, const int32_t *list) {
    k_write_payload<<<grid, kGroupTile, 0, st>>>(a, 0, list);
  });
  BZ_LAUNCH_CHECK();
}

// Copy each block's bits (word-aligned in the arena) to its bit position in
// the output streams; the output is zeroed, and the first and last word of a
// block are OR-ed in because neighbours share them.  kSpliceParts CTAs share a
// block's words (one CTA per block left the longest blocks to run alone).
constexpr int kSpliceParts = 8;
__global__ void __launch_bounds__(256) k_splice(const int64_t *src_addr, const int64_t *dst_bit,
                                                const int64_t *nbits, uint32_t *out) {
  const int b = blockIdx.x;
  const int64_t L = nbits[b];
  if (L <= 0) return;
  const int64_t D = dst_bit[b];
  const uint32_t *src = reinterpret_cast<const uint32_t *>(src_addr[b]);
  const int64_t srcw = (L + 31) >> 5;
  const int64_t w_first = D >> 5, w_last = (D + L - 1) >> 5;
  for (int64_t w = w_first + blockIdx.y * 256 + threadIdx.x; w <= w_last; w += 256 * kSpliceParts) {
    const int64_t s = w * 32 - D;  // source bit of this word's first bit
    const int64_t a = s >= 0 ? s >> 5 : -1;
    const int sh = (int)(s - a * 32);
    const uint32_t x0 = (a >= 0 && a < srcw) ? bswap32(src[a]) : 0u;
    const uint32_t x1 = (a + 1 >= 0 && a + 1 < srcw) ? bswap32(src[a + 1]) : 0u;
    const uint32_t v = sh == 0 ? x0 : ((x0 << sh) | (x1 >> (32 - sh)));
    if (w == w_first || w == w_last) {
      if (v) atomicOr(out + w, bswap32(v));
    } else {
      out[w] = bswap32(v);
    }
  }
}

void launch_splice(const int64_t *src_addr, const int64_t *dst_bit, const int64_t *nbits,
                   int nblocks, uint32_t *out, cudaStream_t st) {
  if (nblocks <= 0) return;
  k_splice<<<dim3(nblocks, kSpliceParts), 256, 0, st>>>(src_addr, dst_bit, nbits, out);
  BZ_LAUNCH_CHECK();
}

void launch_pack_words(const SlabDev &d, uint32_t *words, cudaStream_t st) {
  launch_groups(d, st, [&](int grid, const int32_t *list) {
    k_pack_words<<<grid, kGroupTile, 0, st>>>(d, words, list);
  });
  BZ_LAUNCH_CHECK();
}

}  // namespace bz2g
