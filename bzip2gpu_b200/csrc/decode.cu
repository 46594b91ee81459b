// GPU decompressor for .bz2 streams (no counterpart in the reference, whose
// TODO.md:28-34 lists decompression as missing).
//
// Blocks are decoded in parallel:
//   1. k_dec_magic: every bit offset of the stream is tested for the 48-bit
//      block magic 0x314159265359 and the end-of-stream magic 0x177245385090;
//      the host then follows the chain (a block starts where the previous one
//      ended), so a magic that happens to appear inside a payload is ignored.
//   2. k_dec_head / _groups / _syms / _mscan / _emit: header and tables, the
//      bit position of every 50-symbol group (the one serial chain, hopped 8
//      codes at a time; for few blocks a group at a time, from the jumps of
//      k_dec_lens / _jumps / _starts), the groups' symbols and the inverse
//      move-to-front in parallel over chunks of 32 groups.  Out: the BWT last column L.
//   3. k_dec_lf_hist / _scan / _rank: LF vector
//      tt[C[L[i]] + rank(i)] = i << 8 | L[i] by a stable counting sort.
//   4. k_dec_walk / k_dec_chain / k_dec_gather: per block, the chain from
//      origPtr gives the RLE1 bytes, cut at every 64th or 128th position; the
//      segments are walked in parallel and copied to their places.
//   5. k_dec_unrle1_count / _scan / _write expand the RLE1 runs (4 equal bytes
//      then a count byte) from 32-byte segments at once; k_dec_crc
//      computes each block's CRC over its output (4096-byte chunks combined
//      over GF(2)), checked against the header.
// Batches of blocks go through steps 2-5 while the previous batch's bytes are
// copied out on a second stream; within a batch the largest compressed blocks
// start first, since a launch lasts as long as its slowest blocks.
// Every field read from the stream is range-checked and every loop is bounded,
// so a malformed stream gives an error status, not a fault.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/bz2g.h"
#include "common.cuh"
#include "compressor.h"
#include "crc.cuh"
#include "decode_plan.h"
#include "grow_buf.h"

namespace bz2g {

void set_last_error(const std::string &msg);

namespace {

constexpr int kDecMaxGroups = 6;
constexpr int kDecMaxAlpha = 258;
constexpr int kDecMaxCode = 20;
constexpr int kLutBits = 8;
static_assert(kDecGroupSyms == kGroupSize, "symbols per group");

enum DecStatus {
  kDecOk = 0,
  kDecBadHeader = 1,
  kDecBadTables = 2,
  kDecBadSymbol = 3,
  kDecTooLong = 4,
  kDecBadOrigPtr = 5,
  kDecBadCrc = 6,
};

__device__ __forceinline__ uint32_t bswap32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

// Sequential big-endian bit reader over the stream's words (reads past the end
// return zeros).  A three-word window w0:w1:w2 (already byte-swapped) and the
// bit offset in w0: peek32 is one funnel shift, and the word after the
// window is loaded when the offset passes a word, well before it is needed.
struct BitReader {
  const uint32_t *w;
  int64_t nwords, wnext;  // wnext: index of the word after the window
  uint32_t w0, w1, w2;
  int bo;
  __device__ __forceinline__ uint32_t ld(int64_t i) const {
    return i < nwords ? bswap32(w[i]) : 0u;
  }
  __device__ void init(const uint32_t *words, int64_t nw, int64_t bitpos) {
    w = words;
    nwords = nw;
    const int64_t i = bitpos >> 5;
    w0 = ld(i);
    w1 = ld(i + 1);
    w2 = ld(i + 2);
    wnext = i + 3;
    bo = (int)(bitpos & 31);
  }
  // the 32 bits from the current position
  __device__ __forceinline__ uint32_t peek32() const { return __funnelshift_l(w1, w0, bo); }
  __device__ __forceinline__ uint32_t peek(int n) const { return peek32() >> (32 - n); }
  // n <= 32
  __device__ __forceinline__ void skip(int n) {
    bo += n;
    if (bo >= 32) {
      bo -= 32;
      w0 = w1;
      w1 = w2;
      w2 = ld(wnext++);
    }
  }
  __device__ __forceinline__ uint32_t get(int n) {
    if (n == 0) return 0;
    const uint32_t v = peek(n);
    skip(n);
    return v;
  }
  __device__ __forceinline__ int64_t pos() const { return (wnext - 3) * 32 + bo; }
};

// A thread tests the 32 bit positions of a word: the first 32 bits of both
// magics by one funnel shift and two compares, the other 16 on a match (64-bit
// shifts and compares of all 48 bits took 8 times the instructions).
__global__ void k_dec_magic(const uint32_t *words, int64_t nwords, int64_t nbits,
                            int64_t *blk, int *nblk, int64_t *eos, int *neos, int cap) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nwords) return;
  const uint32_t a = bswap32(words[i]);
  const uint32_t b = i + 1 < nwords ? bswap32(words[i + 1]) : 0u;
  uint32_t hits = 0;
#pragma unroll
  for (int s = 0; s < 32; s++) {
    const uint32_t v = __funnelshift_l(b, a, s);
    if (v == 0x31415926u || v == 0x17724538u) hits |= 1u << s;
  }
  while (hits) {
    const int s = __ffs(hits) - 1;
    hits &= hits - 1u;
    const int64_t p = i * 32 + s;
    if (p + 48 > nbits) break;
    const uint32_t c = i + 2 < nwords ? bswap32(words[i + 2]) : 0u;
    const uint32_t v = __funnelshift_l(b, a, s), low = __funnelshift_l(c, b, s) >> 16;
    if (v == 0x31415926u && low == 0x5359u) {
      const int k = atomicAdd(nblk, 1);
      if (k < cap) blk[k] = p;
    } else if (v == 0x17724538u && low == 0x5090u) {
      const int k = atomicAdd(neos, 1);
      if (k < cap) eos[k] = p;
    }
  }
}

// Per-block results of the entropy decode.
struct DecBlock {
  int64_t start;    // bit position of the block magic
  int64_t end;      // bit position after the payload
  int32_t m;        // last-column length
  int32_t orig_ptr;
  uint32_t crc;     // from the header
  int32_t status;
  int32_t nchunks;  // chunks of symbols up to the end of the block
};

// Entropy decode of one block, split so that only the group starts are a
// serial chain (a code's length is known only once its start is):
//   k_dec_head    header, selectors, code tables           (a CTA per block)
//   k_dec_groups  bit position of every 50-symbol group    (a CTA per block), or
//   k_dec_lens, _jumps, _starts the same, for few blocks
//   k_dec_syms    the groups' symbols, a thread each, and the inverse
//                 move-to-front of 32 groups (a chunk) from an unknown
//                 starting list                            (a warp per chunk)
//   k_dec_mscan   the chunks' starting lists and offsets   (a CTA per block)
//   k_dec_emit    the last column                          (a warp per chunk)
constexpr int kHeadThreads = 256;
constexpr int kChunkSyms = kChunkGroups * kGroupSize;  // 1600

// Per-block tables.  lj[t][n]: the largest 32-bit window (the stream's next
// bits, left-justified) that starts with a code of at most n bits, for n in
// [mn, mx]; a window's code length is the smallest such n.
struct DecTab {
  int64_t pay;  // bit position of the first symbol
  int32_t status, nuse, ng, nsel, orig_ptr;
  uint32_t crc;
  int32_t ngv;  // groups whose start is known (-1: not yet looked for)
  uint8_t mn[kDecMaxGroups], mx[kDecMaxGroups];
  uint32_t lj[kDecMaxGroups][kDecMaxCode + 4];
  int32_t base[kDecMaxGroups][kDecMaxCode + 4];  // code - base = index into perm
  uint16_t lut[kDecMaxGroups][1 << kLutBits];    // (len << 9) | symbol; 0 = longer code
  uint16_t perm[kDecMaxGroups][kDecMaxAlpha + 6];
  uint8_t seq2unseq[256];
};
static_assert(sizeof(DecTab) % 8 == 0, "DecTab rows in an array");

// What a chunk's symbols amount to, before the run digits carried into it and
// its starting list are known.
struct ChunkInfo {
  int32_t nsym;   // symbols before the end of block, a bad code or the chunk's end
  int32_t eob;    // 1: the end-of-block symbol follows them
  int32_t bad;    // 1: a bad code follows them
  int32_t lead;   // run digits before the first other symbol
  int32_t trail;  // run digits after the last other symbol (nsym if there is none)
  uint32_t end;   // eob: bits from the block's magic to the end of its payload
  int64_t lead_sum, rest_sum;  // bytes of the leading run digits (counted from digit 0) and of the rest
  int64_t off;    // offset of the chunk's bytes in the last column
  int32_t q0;     // run digits just before the chunk
  int32_t pad;
};

// A block's scratch until its LF vector is built, in that vector's memory.
struct SymScratch {
  uint16_t rec[kMaxChunks * kChunkSyms];
  uint8_t list[kMaxChunks][256];  // end permutation, then starting list, of each chunk
  ChunkInfo info[kMaxChunks];
};
static_assert(sizeof(SymScratch) <= (size_t)kDecCap * 4, "symbols fit the LF vector's memory");
__device__ __forceinline__ SymScratch &sym_scratch(uint32_t *tt, int bi, int cap) {
  return *reinterpret_cast<SymScratch *>(tt + (size_t)bi * cap);
}
// A record: the symbol's position in the chunk's starting list (bits 0-7);
// a run digit has bit 15, its value in bit 13 and its place in bits 8-12.
constexpr uint32_t kRecRun = 0x8000u;

// c copies of byte v at d (word stores between unaligned ends).
__device__ __forceinline__ void fill_bytes(uint8_t *d, int c, uint8_t v) {
  while (c > 0 && (reinterpret_cast<uintptr_t>(d) & 3u)) {
    *d++ = v;
    c--;
  }
  const uint32_t wv = 0x01010101u * v;
  for (; c >= 4; c -= 4, d += 4) *reinterpret_cast<uint32_t *>(d) = wv;
  while (c-- > 0) *d++ = v;
}

// 32 stream bits from bit position p (zeros past the end).
__device__ __forceinline__ uint32_t bits_at(const uint32_t *words, int64_t nwords, int64_t p) {
  const int64_t i = p >> 5;
  const uint32_t a = i < nwords ? bswap32(words[i]) : 0u;
  const uint32_t b = i + 1 < nwords ? bswap32(words[i + 1]) : 0u;
  return __funnelshift_l(b, a, (int)(p & 31));
}

// Selector lists as six nibbles, nibble k = table at list position k.
__device__ __forceinline__ uint32_t sel_front(uint32_t lst, int j) {
  const uint32_t t = (lst >> (4 * j)) & 0xFu;
  const uint32_t low = (1u << (4 * j)) - 1u;
  return (lst & ~((low << 4) | 0xFu)) | ((lst & low) << 4) | t;
}
// The list a after the moves that take the identity list to b.
__device__ __forceinline__ uint32_t sel_then(uint32_t a, uint32_t b) {
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < kDecMaxGroups; k++)
    r |= ((a >> (4 * ((b >> (4 * k)) & 0xFu))) & 0xFu) << (4 * k);
  return r;
}

// A table's code lengths by one warp: a 5-bit start, then per symbol steps 1x
// (x = 0: +1, x = 1: -1) and a 0.  A lane takes 32 bits; whether it starts
// inside a step follows from the bits before it (a 0 always ends what it is
// in; after ones only, their number decides), then scans over the lanes give
// each one's symbol and length so far.  Every length on the way must lie in
// 1 .. kDecMaxCode, and a symbol takes at most 63 steps.  p: the table's
// first bit; moved past it.  (One thread bit by bit: 150 us for six tables.)
__device__ int code_lengths(const uint32_t *words, int64_t nwords, int64_t &p, int alpha,
                            uint8_t *len) {
  const unsigned full = 0xffffffffu;
  const int ln = lane_id();
  int cur0 = (int)(bits_at(words, nwords, p) >> 27);
  p += 5;
  int64_t last_end = p;  // where the symbol being read began
  int done = 0;
  uint32_t inside = 0;   // the round starts inside a step
  for (;;) {
    const uint32_t x = bits_at(words, nwords, p + 32 * ln);
    const int ones = x == full ? 32 : __ffs(~x) - 1;  // at the word's end
    const unsigned broken = __ballot_sync(full, x != full);
    const unsigned odd = __ballot_sync(full, ones & 1);
    const unsigned below = broken & ((1u << ln) - 1u);
    const uint32_t in = below ? (odd >> (31 - __clz(below))) & 1u : inside;
    uint32_t s = in;
    int ends = 0, sum = 0, end_at = -1;
#pragma unroll
    for (int i = 0; i < 32; i++) {
      const bool one = (x >> (31 - i)) & 1u;
      if (s) {
        sum += one ? -1 : 1;
        s = 0;
      } else if (one) {
        s = 1;
      } else {
        ends++;
        end_at = i;
      }
    }
    const int esum = warp_incl_sum(ends), dsum = warp_incl_sum(sum);
    const unsigned has = __ballot_sync(full, ends > 0);
    const unsigned hb = has & ((1u << ln) - 1u);
    const int pe = __shfl_sync(full, 32 * ln + end_at + 1, hb ? 31 - __clz(hb) : 0);
    int64_t began = hb ? p + pe : last_end;
    int sym = done + esum - ends;
    int cur = cur0 + dsum - sum;
    bool bad = sym < alpha && (cur < 1 || cur > kDecMaxCode);
    int fin = -1;
    s = in;
#pragma unroll
    for (int i = 0; i < 32; i++) {
      const bool one = (x >> (31 - i)) & 1u;
      if (s) {
        cur += one ? -1 : 1;
        s = 0;
        if (sym < alpha) bad |= cur < 1 || cur > kDecMaxCode;
      } else if (one) {
        s = 1;
      } else {
        if (sym < alpha) {
          const int64_t at = p + 32 * ln + i;
          bad |= at - began > 2 * 63;
          began = at + 1;
          len[sym] = (uint8_t)cur;
          if (sym == alpha - 1) fin = i;
        }
        sym++;
      }
    }
    if (__any_sync(full, bad) || !has) return kDecBadTables;
    const unsigned fm = __ballot_sync(full, fin >= 0);
    if (fm) {
      p += __shfl_sync(full, 32 * ln + fin + 1, __ffs(fm) - 1);
      return kDecOk;
    }
    done += __shfl_sync(full, esum, 31);
    cur0 += __shfl_sync(full, dsum, 31);
    last_end = p + __shfl_sync(full, 32 * ln + end_at + 1, 31 - __clz(has));
    inside = __shfl_sync(full, s, 31);
    p += 1024;
  }
}

// Header, selectors and tables of a candidate block.
// Selectors are unary codes: selector k ends at the k-th zero bit, so each
// thread takes 32 bits, a scan of zero counts says which selectors end in
// them, and the ones before a zero are its move-to-front index.  The index
// sequence moves a six-entry list; each thread runs its share from the
// identity list, a scan of those permutations gives every share's starting
// list.  The delta-coded lengths are one warp's (code_lengths).
__global__ void __launch_bounds__(kHeadThreads) k_dec_head(const uint32_t *words, int64_t nwords,
                                                           const int64_t *cand, DecTab *tabs,
                                                           uint8_t *selbuf) {
  __shared__ uint8_t sj[kDecMaxSel + 2];
  __shared__ uint8_t len[kDecMaxGroups][kDecMaxAlpha + 6];
  __shared__ int scratch[40];
  __shared__ uint32_t wperm[kHeadThreads / 32];
  __shared__ int64_t s_end;
  __shared__ int s_status;
  const int bi = blockIdx.x;
  const int ln = lane_id(), w = warp_id();
  DecTab &tab = tabs[bi];
  uint8_t *sel = selbuf + (size_t)bi * kDecMaxSel;
  int status = kDecOk;
  BitReader br;
  br.init(words, nwords, cand[bi] + 48);
  const uint32_t crc = br.get(32);
  const uint32_t randomised = br.get(1);
  const int orig_ptr = (int)br.get(24);
  const uint32_t used16 = br.get(16);
  int nuse = 0;
  for (int i = 0; i < 16; i++) {
    if ((used16 >> (15 - i)) & 1u) {
      const uint32_t bits = br.get(16);
      if (threadIdx.x < 16 && ((bits >> (15 - threadIdx.x)) & 1u))
        tab.seq2unseq[nuse + __popc(bits >> (16 - threadIdx.x))] = (uint8_t)(i * 16 + threadIdx.x);
      nuse += __popc(bits);
    }
  }
  const int alpha = nuse + 2;
  const int ng = (int)br.get(3);
  const int nsel = (int)br.get(15);
  if (randomised || nuse == 0 || ng < 2 || ng > 6 || nsel < 1 || nsel > kDecMaxSel)
    status = kDecBadHeader;
  if (threadIdx.x == 0) {
    s_status = status;
    s_end = 0;
  }
  __syncthreads();
  if (status == kDecOk) {
    const int64_t p0 = br.pos();
    int done = 0;  // selectors ended so far
    // a valid code has at most ng bits; a longer one ends the search
    for (int r = 0; done < nsel && r < kDecMaxGroups * nsel; r += 32 * kHeadThreads) {
      const int64_t p = p0 + r + 32 * (int64_t)threadIdx.x;
      const uint32_t x = bits_at(words, nwords, p);
      // the ones just before this thread's bits (none before the selectors)
      const uint32_t before = p > p0 ? bits_at(words, nwords, p - 32) : 0u;
      int ones = __ffs(~before) - 1;
      if (ones < 0) ones = 32;
      int tot;
      int k = done + block_excl_sum(__popc(~x), scratch, &tot);
      uint32_t z = ~x;
      int at = -ones;  // where the current unary code began
      while (z && k < nsel) {
        const int q = __clz(z);
        const int j = q - at;
        if (j >= ng) s_status = kDecBadHeader;
        sj[k] = (uint8_t)j;
        if (k == nsel - 1) s_end = p + q + 1;
        k++;
        at = q + 1;
        z &= ~(0x80000000u >> q);
      }
      done += tot;
    }
    if (done < nsel) s_status = kDecBadHeader;
    __syncthreads();
    status = s_status;
  }
  if (status == kDecOk) {
    const int per = (nsel + kHeadThreads - 1) / kHeadThreads;
    const int a = min(nsel, (int)threadIdx.x * per), e = min(nsel, a + per);
    uint32_t mine = 0x543210u;
    for (int i = a; i < e; i++) mine = sel_front(mine, sj[i]);
    uint32_t inc = mine;  // moves of this and the earlier lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
      if (ln >= d) inc = sel_then(o, inc);
    }
    if (ln == 31) wperm[w] = inc;
    uint32_t lst = __shfl_up_sync(0xffffffffu, inc, 1);
    if (ln == 0) lst = 0x543210u;
    __syncthreads();
    uint32_t pre = 0x543210u;
    for (int q = 0; q < w; q++) pre = sel_then(pre, wperm[q]);
    lst = sel_then(pre, lst);
    for (int i = a; i < e; i++) {
      lst = sel_front(lst, sj[i]);
      sel[i] = (uint8_t)(lst & 0xFu);
    }
    if (w == 0) {
      int64_t p = s_end;
      int st = kDecOk;
      for (int t = 0; t < ng && st == kDecOk; t++) st = code_lengths(words, nwords, p, alpha, len[t]);
      if (ln == 0) {
        s_status = st;
        tab.pay = p;
      }
    }
    __syncthreads();
    status = s_status;
  }
  if (status == kDecOk && w < ng) {
    // canonical codes, a warp per table: the symbols of each length in symbol
    // order take consecutive codes (lane l holds symbols l, l + 32, ...)
    constexpr int kSlots = (kDecMaxAlpha + 31) / 32;
    int lv[kSlots];
    int mn = 32, mx = 0;
#pragma unroll
    for (int q = 0; q < kSlots; q++) {
      const int v = 32 * q + ln;
      lv[q] = v < alpha ? (int)len[w][v] : -1;
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
    int idx = 0;
    uint32_t code = 0;
    for (int l = mn; l <= mx; l++) {
      const int first = idx;
#pragma unroll
      for (int q = 0; q < kSlots; q++) {
        const bool hit = lv[q] == l;
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (hit) tab.perm[w][idx + __popc(bal & below)] = (uint16_t)(32 * q + ln);
        idx += __popc(bal);
      }
      // codes of length l: [code, code + idx - first)
      const uint64_t end = (uint64_t)code + (uint32_t)(idx - first);
      if (ln == 0) {
        tab.base[w][l] = (int32_t)code - first;
        tab.lj[w][l] = (end << (32 - l)) > 0xFFFFFFFFull ? 0xFFFFFFFFu
                                                         : (uint32_t)(end << (32 - l)) - 1u;
      }
      code = (uint32_t)end << 1;
    }
    if (ln == 0) {
      tab.mn[w] = (uint8_t)mn;
      tab.mx[w] = (uint8_t)mx;
    }
    __syncwarp();
    for (int p = ln; p < (1 << kLutBits); p += 32) {
      const uint32_t x = (uint32_t)p << (32 - kLutBits);
      uint16_t e = 0;
      for (int l = mn; l <= min(mx, kLutBits); l++) {
        if (x <= tab.lj[w][l]) {
          const int i = (int)(x >> (32 - l)) - tab.base[w][l];
          if (i >= 0 && i < alpha) e = (uint16_t)((l << 9) | tab.perm[w][i]);
          break;
        }
      }
      tab.lut[w][p] = e;
    }
  }
  if (threadIdx.x == 0) {
    tab.status = status;
    tab.nuse = nuse;
    tab.ng = ng;
    tab.nsel = nsel;
    tab.orig_ptr = orig_ptr;
    tab.crc = crc;
    tab.ngv = -1;
  }
}

// Bit position of every group, one CTA of NW warps per block.  The chain over
// a group's 50 codes is cut short: for a window of bit positions from the
// group's start all code lengths are looked up at once, the map "position ->
// position after one code" is squared three times in shared memory (after 2,
// 4, 8 codes), and the group is six 8-code hops and one 2-code hop.  The
// window is as wide as the table's last group was, plus a quarter; a group
// that leaves it goes on in another.  Positions are table indices, and three
// kinds of entries map to themselves or out, so that hops need no tests:
// kPadAt .. the 32 positions past the window (a hop that ends there is good,
// a further one is not), kNoHop (the map leaves the window on its way) and
// kDeadCode (no code starts here).
// The latency of this chain bounds a call of few blocks.
constexpr int kWin = 512;
constexpr int kLenBits = 12;
constexpr int kRing = 256;
constexpr int kRingLoad = 128;  // words per refill
constexpr uint32_t kNoHop = kWin + 32;
constexpr uint32_t kDeadCode = kWin + 33;
constexpr int kHops = kWin + 34;

template <int NW>
__global__ void __launch_bounds__(32 * NW)
    k_dec_groups(const uint32_t *words, int64_t nwords, const int64_t *cand, DecTab *tabs,
                 const uint8_t *selbuf, uint32_t *gstart, const int32_t *order) {
  constexpr int NT = 32 * NW;
  constexpr int kPer = kWin / NT;  // window positions per thread
  static_assert(NT >= kRingLoad && kPer >= 1, "warps per block");
  __shared__ uint8_t llen[kDecMaxGroups][1 << kLenBits];
  __shared__ uint32_t lj[kDecMaxGroups][kDecMaxCode + 4];
  __shared__ uint8_t mn_s[kDecMaxGroups + 2], mx_s[kDecMaxGroups + 2];
  // two sets used in turn: a warp may still hop in one while others fill the next
  __shared__ uint16_t s1[2][kHops], s2[2][kHops], s4[2][kHops], s8[2][kHops];
  __shared__ uint32_t ring[kRing];
  const unsigned full = 0xffffffffu;
  const int bi = order[blockIdx.x];  // largest compressed blocks first
  const int tid = threadIdx.x, ln = lane_id();
  DecTab &tab = tabs[bi];
  if (tab.status != kDecOk || tab.ngv >= 0) return;  // bad header, or done by k_dec_starts
  const int ng = tab.ng, nsel = tab.nsel;
  for (int i = tid; i < ng * (kDecMaxCode + 4); i += NT) (&lj[0][0])[i] = (&tab.lj[0][0])[i];
  if (tid < ng) {
    mn_s[tid] = tab.mn[tid];
    mx_s[tid] = tab.mx[tid];
  }
  if (tid < 2) {
    for (uint32_t q : {kNoHop, kDeadCode})
      s1[tid][q] = s2[tid][q] = s4[tid][q] = s8[tid][q] = (uint16_t)q;
  }
  __syncthreads();
  for (int i = tid; i < ng << kLenBits; i += NT) {
    const int t = i >> kLenBits;
    const uint32_t x = (uint32_t)(i & ((1 << kLenBits) - 1)) << (32 - kLenBits);
    const int mn = mn_s[t], mx = min((int)mx_s[t], kLenBits);
    int n = mn;
    while (n <= mx && x > lj[t][n]) n++;
    llen[t][i & ((1 << kLenBits) - 1)] = (uint8_t)(n <= mx ? n : 0);
  }
  const uint8_t *sel = selbuf + (size_t)bi * kDecMaxSel;
  uint32_t *gs = gstart + (size_t)bi * kDecMaxSel;
  const int64_t start = cand[bi];
  const int64_t wbase = start >> 5;  // word indices below are relative to it
  const uint32_t *W = words + wbase;
  const int64_t navail = nwords - wbase;
  uint32_t p = (uint32_t)(tab.pay - (wbase << 5));
  const uint32_t bias = (uint32_t)(start & 31);
  // ring of byte-swapped words: [hi - kRing, hi) present, the next ones in pf
  uint32_t hi = p >> 5;
  uint32_t pf = 0;
  auto fetch = [&]() {
    const int64_t i = (int64_t)hi + tid;
    if (tid < kRingLoad) pf = i < navail ? W[i] : 0u;
  };
  fetch();
  int last_bits = kWin;  // lane t: bits of table t's last group
  uint32_t my_start = 0;
  int my_sel = 0, next_sel = ln < nsel ? sel[ln] : 0;
  int g = 0, set = 0;
  bool dead = false;
  for (; g < nsel && !dead; g++) {
    if ((g & 31) == 0) {
      my_sel = next_sel;
      next_sel = g + 32 + ln < nsel ? sel[g + 32 + ln] : 0;
    }
    if (ln == (g & 31)) my_start = p - bias;
    const int t = __shfl_sync(full, my_sel, g & 31);
    const int lb = __shfl_sync(full, last_bits, t);
    const uint8_t *lt = llen[t];
    const uint32_t p_begin = p;
    int rem = kGroupSize;
    const int ew = min(kWin, ((lb + (lb >> 2) + 63) >> 5) << 5);  // window width
    while (rem > 0 && !dead) {
      const uint32_t i0 = p >> 5;
      if (hi < i0 + kWin / 32 + 4) {  // i0 advances by less than kRingLoad words
        do {
          if (tid < kRingLoad) ring[(hi + tid) & (kRing - 1)] = bswap32(pf);
          hi += kRingLoad;
          fetch();
        } while (hi < i0 + kWin / 32 + 4);
        __syncthreads();
      }
      set ^= 1;
      uint16_t *a1 = s1[set], *a2 = s2[set], *a4 = s4[set], *a8 = s8[set];
      if (tid < 32) a1[ew + tid] = a2[ew + tid] = a4[ew + tid] = a8[ew + tid] = (uint16_t)kNoHop;
      const int o0 = (int)(p & 31) + tid;
      const uint32_t c = i0 + (o0 >> 5);
      const int sh = o0 & 31;
      uint32_t cur[kPer];
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const int o = NT * j + tid;
        if (o < ew) {
          const uint32_t x = __funnelshift_l(ring[(c + NW * j + 1) & (kRing - 1)],
                                             ring[(c + NW * j) & (kRing - 1)], sh);
          int n = lt[x >> (32 - kLenBits)];
          if (n == 0) {
            const int mx = mx_s[t];
            n = max((int)mn_s[t], kLenBits + 1);
            while (n <= mx && x > lj[t][n]) n++;
            if (n > mx) n = 0;
          }
          cur[j] = n ? (uint32_t)(o + n) : kDeadCode;
          a1[o] = (uint16_t)cur[j];
        }
      }
      __syncthreads();
      auto square = [&](const uint16_t *from, uint16_t *to) {
#pragma unroll
        for (int j = 0; j < kPer; j++) {
          if (NT * j + tid < ew) {
            cur[j] = from[cur[j]];
            to[NT * j + tid] = (uint16_t)cur[j];
          }
        }
        __syncthreads();
      };
      square(a1, a2);
      square(a2, a4);
      square(a4, a8);
      uint32_t at = kNoHop;
      if (rem == kGroupSize) {
        at = 0;
#pragma unroll
        for (int q = 0; q < kGroupSize / 8; q++) at = a8[at];
        at = a2[at];
      }
      if (at < kNoHop) {
        rem = 0;
      } else {  // out of the window on the way: as far as the window goes
        at = 0;
        while (rem >= 8 && a8[at] < kNoHop) {
          at = a8[at];
          rem -= 8;
        }
        while (rem >= 2 && a2[at] < kNoHop) {
          at = a2[at];
          rem -= 2;
        }
        while (rem >= 1 && at < (uint32_t)ew && !dead) {
          const uint32_t v = a1[at];
          if (v == kDeadCode) {
            dead = true;
          } else {
            at = v;
            rem--;
          }
        }
      }
      p += at;
    }
    if (ln == t) last_bits = (int)(p - p_begin);
    if (tid < 32 && ((g & 31) == 31 || g + 1 == nsel || dead)) {
      const int gb = g & ~31;
      if (gb + ln <= g) gs[gb + ln] = my_start;
    }
  }
  if (tid == 0) tab.ngv = g;
}

// Few blocks (jumps_pay): the jump over a whole group (50 codes) from every bit
// position with every table, then the chain of group starts is one lookup per
// group.
// k_dec_jumps covers kJumpTile positions of a block per CTA: code lengths of
// the tile and a halo (50 codes take at most 1000 bits), the map squared five
// times in shared memory, composed to 32 + 16 + 2 codes.  k_dec_starts streams
// a block's tiles through four buffers and hops.  This takes about 36
// instructions per position and table, a hundred times what the chain of
// k_dec_groups needs, but nothing of it waits: 0.1 ms and 0.3 ms for one block,
// where k_dec_groups takes 3.4 ms.  Positions are relative to the block's magic.
constexpr int kJumpHalo = 1024;
constexpr int kJumpAll = kJumpTile + kJumpHalo;
constexpr int kJumpPer = kJumpAll / 256;             // positions per thread
constexpr uint32_t kJumpOut = kJumpAll + 32;         // leaves the tile and halo
constexpr uint32_t kJumpDead = kJumpAll + 33;        // no code starts here
constexpr int kJumpSlots = kJumpAll + 34;
constexpr uint32_t kDeadJump = 0xFFFFu;
constexpr int kLensBytes = kDecMaxGroups << kLenBits;
constexpr size_t kJumpSmem = (size_t)3 * kJumpSlots * 2 + (1 << kLenBits) + 64;
constexpr int kStartStages = 4;  // tiles in flight: 48 KB each
constexpr size_t kStartStage = (size_t)kDecMaxGroups * kJumpTile * 2;
static_assert(kStartStage == kJumpTileBytes, "a tile's jumps");
constexpr size_t kStartsSmem = kStartStages * kStartStage;

// Code length (0: longer than kLenBits, or none) by the next kLenBits bits.
// grid: (table, block)
__global__ void __launch_bounds__(256) k_dec_lens(const DecTab *tabs, uint8_t *lens) {
  const int bi = blockIdx.y, t = blockIdx.x;
  const DecTab &tab = tabs[bi];
  if (tab.status != kDecOk || t >= tab.ng) return;
  uint8_t *out = lens + (size_t)bi * kLensBytes + ((size_t)t << kLenBits);
  const int mn = tab.mn[t], mx = min((int)tab.mx[t], kLenBits);
  for (int p = threadIdx.x; p < (1 << kLenBits); p += 256) {
    const uint32_t x = (uint32_t)p << (32 - kLenBits);
    int n = mn;
    while (n <= mx && x > tab.lj[t][n]) n++;
    out[p] = (uint8_t)(n <= mx ? n : 0);
  }
}

// A CTA per tile: jt0 holds the first tile of each of the nc blocks, and the
// last one's end.
// jumps: per tile, per table, kJumpTile advances, twice the bits (table bytes;
// kDeadJump: none).
__global__ void __launch_bounds__(256) k_dec_jumps(const uint32_t *words, int64_t nwords,
                                                   const int64_t *cand, const DecTab *tabs,
                                                   const uint8_t *lens, const int32_t *jt0,
                                                   int nc, uint16_t *jumps) {
  extern __shared__ __align__(16) uint8_t jsm[];
  uint16_t *A = reinterpret_cast<uint16_t *>(jsm), *B = A + kJumpSlots, *C = B + kJumpSlots;
  uint8_t *llen = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(C + kJumpSlots) + 15) & ~(uintptr_t)15);
  __shared__ uint32_t bits[kJumpAll / 32 + 2];
  __shared__ uint32_t lj[kDecMaxCode + 4];
  const int tile = jt0[0] + blockIdx.x;
  int bi = 0;  // jt0[bi] <= tile < jt0[end]
  for (int end = nc; end - bi > 1;) {
    const int mid = (bi + end) >> 1;
    if (jt0[mid] <= tile) bi = mid;
    else end = mid;
  }
  const DecTab &tab = tabs[bi];
  if (tab.status != kDecOk) return;
  const int tid = threadIdx.x;
  const int64_t p0 = cand[bi] + (int64_t)(tile - jt0[bi]) * kJumpTile;
  for (int q = tid; q < kJumpAll / 32 + 2; q += 256) bits[q] = bits_at(words, nwords, p0 + 32 * q);
  if (tid < 34) {  // positions past the halo, and the two states, in all buffers
    const uint32_t q = kJumpAll + tid;
    const uint16_t v = (uint16_t)(q == kJumpDead ? kJumpDead : kJumpOut);
    A[q] = B[q] = C[q] = v;
  }
  for (int t = 0; t < tab.ng; t++) {
    __syncthreads();  // the previous table's gathers are done
    const uint8_t *src = lens + (size_t)bi * kLensBytes + ((size_t)t << kLenBits);
    reinterpret_cast<uint4 *>(llen)[tid] = reinterpret_cast<const uint4 *>(src)[tid];
    if (tid < kDecMaxCode + 4) lj[tid] = tab.lj[t][tid];
    const int mn = tab.mn[t], mx = tab.mx[t];
    __syncthreads();
    uint32_t cur[kJumpPer];
#pragma unroll
    for (int j = 0; j < kJumpPer; j++) {
      const int o = 256 * j + tid;
      const uint32_t x = __funnelshift_l(bits[(o >> 5) + 1], bits[o >> 5], o & 31);
      int n = llen[x >> (32 - kLenBits)];
      if (n == 0) {
        n = max(mn, kLenBits + 1);
        while (n <= mx && x > lj[n]) n++;
        if (n > mx) n = 0;
      }
      cur[j] = n ? (uint32_t)(o + n) : kJumpDead;
      A[o] = (uint16_t)cur[j];
    }
    __syncthreads();
    auto square = [&](const uint16_t *from, uint16_t *to) {
#pragma unroll
      for (int j = 0; j < kJumpPer; j++) {
        cur[j] = from[cur[j]];
        to[256 * j + tid] = (uint16_t)cur[j];
      }
      __syncthreads();
    };
    square(A, B);  // 2 codes, kept
    square(B, C);  // 4
    square(C, A);  // 8
    square(A, C);  // 16, kept
    square(C, A);  // 32
    uint16_t *out = jumps + ((size_t)blockIdx.x * kDecMaxGroups + t) * kJumpTile;
#pragma unroll
    for (int j = 0; j < kJumpTile / 256; j++) {
      const uint32_t v = B[C[cur[j]]];  // 50
      const int o = 256 * j + tid;
      out[o] = (uint16_t)(v < kJumpOut ? 2 * (v - o) : kDeadJump);
    }
  }
}

// Group starts of one block by its jumps: the tiles come through
// kStartStages buffers, one thread hops.  A chain that leaves the tiles (a magic inside a payload cuts
// a block's tiles short) leaves ngv -1: k_dec_groups then walks that block.
__global__ void __launch_bounds__(256) k_dec_starts(DecTab *tabs, const uint8_t *selbuf,
                                                    uint32_t *gstart, const int64_t *cand,
                                                    const int32_t *jt0, const uint16_t *jumps) {
  extern __shared__ __align__(16) uint8_t ssm[];
  __shared__ uint8_t sel[kDecMaxSel + 6];
  const int bi = blockIdx.x, tid = threadIdx.x;
  DecTab &tab = tabs[bi];
  if (tab.status != kDecOk) return;
  const int ng = tab.ng, nsel = tab.nsel;
  const int t0 = jt0[bi] - jt0[0], nt = jt0[bi + 1] - jt0[bi];
  for (int q = tid; q < nsel; q += 256) sel[q] = selbuf[(size_t)bi * kDecMaxSel + q];
  uint32_t *gs = gstart + (size_t)bi * kDecMaxSel;
  const uint32_t first = (uint32_t)(tab.pay - cand[bi]);
  const int vec = ng * kJumpTile * 2 / 16;  // 16-byte pieces of a tile's tables
  auto load = [&](int k) {
    if (k < nt) {
      const uint4 *src = reinterpret_cast<const uint4 *>(
          jumps + (size_t)(t0 + k) * kDecMaxGroups * kJumpTile);
      uint4 *dst = reinterpret_cast<uint4 *>(ssm + (size_t)(k % kStartStages) * kStartStage);
      for (int q = tid; q < vec; q += 256) {
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + q);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src + q));
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  const int k0 = (int)(first / kJumpTile);
  for (int k = k0; k < k0 + kStartStages - 1; k++) load(k);
  int g = 0;             // thread 0's place in the chain
  uint32_t p = first;
  bool done = false;     // thread 0: the chain has ended
  for (int k = k0; k < nt; k++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStartStages - 2));
    // tile k is here for all threads, the tile before it is done with, and all
    // leave together (a flag in shared memory could be set by the next hop while
    // a slower warp still reads it)
    if (__syncthreads_or(done)) break;
    load(k + kStartStages - 1);
    if (tid == 0) {
      // bytes of the tile's tables: a jump is one load and one add
      const uint8_t *J = ssm + (size_t)(k % kStartStages) * kStartStage;
      const uint32_t base = (uint32_t)k * kJumpTile;
      uint32_t q = 2 * (p - base), at = sel[g] * (uint32_t)(2 * kJumpTile), v = 0;
      while (q < 2 * kJumpTile && g < nsel) {
        gs[g] = base + (q >> 1);
        g++;
        v = *reinterpret_cast<const uint16_t *>(J + at + q);
        at = sel[g] * (uint32_t)(2 * kJumpTile);  // one byte past nsel is there, not used
        q += v;
      }
      p = base + (q >> 1);
      if (g >= nsel || v == kDeadJump) {
        tab.ngv = g;  // a dead jump's group is the last with a known start
        done = true;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;");
}

// How group starts are found: by the rules below, or (BZ2G_DECODE_STARTS =
// jumps, chains8, chains4) always by the jumps where their scratch fits, or by
// k_dec_groups with 8 or 4 warps per block.  The decoded bytes are the same.
enum class Starts { kByRule, kJumps, kChains8, kChains4 };
Starts starts_choice() {
  const char *e = std::getenv("BZ2G_DECODE_STARTS");
  if (!e) return Starts::kByRule;
  if (!std::strcmp(e, "jumps")) return Starts::kJumps;
  if (!std::strcmp(e, "chains8")) return Starts::kChains8;
  if (!std::strcmp(e, "chains4")) return Starts::kChains4;
  return Starts::kByRule;
}

// Warps per block: eight where the blocks leave the GPU room (the chain's
// latency is what counts), four where there are enough blocks to fill it.
using GroupsKernel = decltype(&k_dec_groups<8>);
inline GroupsKernel groups_kernel(int nblocks, int sms, Starts how, int *threads) {
  const bool few = how == Starts::kChains8 || (how != Starts::kChains4 && nblocks <= 6 * sms);
  *threads = few ? 256 : 128;
  return few ? k_dec_groups<8> : k_dec_groups<4>;
}

// Symbols and local move-to-front of a chunk of 32 groups, one warp each.
// Lane l decodes group l's codes into shared memory.  The inverse
// move-to-front then runs over the chunk from the identity list (so a
// symbol's value is a position in the chunk's starting list), 32 symbols at
// a time across the warp:
//  * lane t walks its index back through the batch's earlier steps s: a
//    step moved the entry at v_s to the front, so position p after it was
//    p - 1 before it when 1 <= p <= v_s, and p == 0 is step s's own output
//    (a run digit repeats the front entry: index 0, no move; 5 instructions
//    per step and 32 symbols);
//  * lanes that reach position 0 point at that step's lane, the others read
//    the list as it was before the batch; pointer jumping settles pointers;
//  * the new list: the batch's distinct outputs, most recent first, then
//    the untouched entries in their old order (equal outputs found by
//    ballots).
__global__ void __launch_bounds__(32 * kSymWarps)
    k_dec_syms(const uint32_t *words, int64_t nwords, const int64_t *cand, const DecTab *tabs,
               const uint8_t *selbuf, const uint32_t *gstart, uint32_t *tt, int cap) {
  __shared__ uint16_t lut[kDecMaxGroups][1 << kLutBits];
  __shared__ uint32_t lj[kDecMaxGroups][kDecMaxCode + 4];
  __shared__ int32_t base[kDecMaxGroups][kDecMaxCode + 4];
  __shared__ uint16_t perm[kDecMaxGroups][kDecMaxAlpha + 6];
  __shared__ uint16_t sy[kSymWarps][kChunkSyms];
  __shared__ __align__(4) uint8_t lists[kSymWarps][2][256];
  __shared__ uint32_t used_s[kSymWarps][8];
  const unsigned full = 0xffffffffu;
  const int bi = blockIdx.y;
  const DecTab &tab = tabs[bi];
  if (tab.status != kDecOk) return;
  const int ngv = tab.ngv;
  if ((int)blockIdx.x * kSymWarps * kChunkGroups >= ngv) return;
  const int ng = tab.ng, nuse = tab.nuse;
  for (int i = threadIdx.x; i < ng * (1 << kLutBits); i += blockDim.x)
    (&lut[0][0])[i] = (&tab.lut[0][0])[i];
  for (int i = threadIdx.x; i < ng * (kDecMaxCode + 4); i += blockDim.x) {
    (&lj[0][0])[i] = (&tab.lj[0][0])[i];
    (&base[0][0])[i] = (&tab.base[0][0])[i];
  }
  for (int i = threadIdx.x; i < ng * (kDecMaxAlpha + 6); i += blockDim.x)
    (&perm[0][0])[i] = (&tab.perm[0][0])[i];
  __syncthreads();
  const int ln = lane_id(), w = warp_id();
  SymScratch &out = sym_scratch(tt, bi, cap);
  const int64_t start = cand[bi];
  const int alpha = nuse + 2, eob = nuse + 1;
  const int stride = gridDim.x * kSymWarps;
  for (int c = (int)blockIdx.x * kSymWarps + w; c * kChunkGroups < ngv; c += stride) {
    const int ngc = min(kChunkGroups, ngv - c * kChunkGroups);
    int e_at = INT32_MAX, b_at = INT32_MAX;  // chunk index of this lane's end-of-block, bad code
    uint32_t e_end = 0;
    if (ln < ngc) {
      const int g = c * kChunkGroups + ln;
      const int t = selbuf[(size_t)bi * kDecMaxSel + g];
      const int mn = tab.mn[t], mx = tab.mx[t];
      BitReader br;
      br.init(words, nwords, start + gstart[(size_t)bi * kDecMaxSel + g]);
      uint16_t *dst = sy[w] + ln * kGroupSize;
      for (int i = 0; i < kGroupSize; i++) {
        const uint32_t x = br.peek32();
        const uint32_t e = lut[t][x >> (32 - kLutBits)];
        int sym;
        if (e) {
          br.skip((int)(e >> 9));
          sym = (int)(e & 511u);
        } else {
          int n = max(mn, kLutBits + 1);
          while (n <= mx && x > lj[t][n]) n++;
          const int idx = n <= mx ? (int)(x >> (32 - n)) - base[t][n] : -1;
          if (idx < 0 || idx >= alpha) {
            b_at = ln * kGroupSize + i;
            break;
          }
          br.skip(n);
          sym = perm[t][idx];
        }
        if (sym == eob) {
          e_at = ln * kGroupSize + i;
          e_end = (uint32_t)(br.pos() - start);
          break;
        }
        dst[i] = (uint16_t)sym;
      }
    }
    const int eob_at = __reduce_min_sync(full, e_at), bad_at = __reduce_min_sync(full, b_at);
    const int n = min(min(eob_at, bad_at), ngc * kGroupSize);
    __syncwarp();
    uint8_t *lb = lists[w][0];
    uint32_t *used = used_s[w];
    for (int q = ln; q < 256; q += 32) lb[q] = (uint8_t)q;
    __syncwarp();
    int cur = 0;
    int run = 0;        // run digits just before the batch
    bool lead = true;   // only run digits so far
    int lead_cnt = 0;
    int64_t lead_sum = 0, rest_sum = 0;
    uint16_t *rec = out.rec + (size_t)c * kChunkSyms;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int nb = min(32, n - i0);
      const bool act = ln < nb;
      const int sym = act ? sy[w][i0 + ln] : 0;
      const bool dgt = act && sym <= 1;
      const unsigned runs = __ballot_sync(full, dgt);
      const unsigned others = __ballot_sync(full, act && !dgt);
      const uint8_t *lst = lb + 256 * cur;
      int rv;  // the symbol's position in the chunk's starting list
      if (others == 0u) {
        rv = lst[0];
      } else {
        const int my_v = act && !dgt ? sym - 1 : 0;
        // p: the position before step ln - d of what this step puts out.  Once
        // at 0 it stays there; it then is the output of the step before the one
        // that last moved it (a run digit: of the step before itself).
        int p = my_v, moved = 0;
  #pragma unroll
        for (int d = 1; d < 32; d++) {
          uint32_t vs;
          int in;
          asm volatile("{ .reg .pred q; shfl.sync.up.b32 %0|q, %2, %3, 0, 0xffffffff; selp.s32 %1, 1, 0, q; }"
              : "=r"(vs), "=r"(in)
              : "r"(my_v), "r"(d));
          if (in && (uint32_t)(p - 1) < vs) {
            p--;
            moved = d;
          }
        }
        int ptr = p == 0 ? ln - moved - 1 : -1;  // below 0: no step before, the list's front
        const bool from_list = act && ptr < 0;
        int val = from_list ? (int)lst[p] : -1;
  #pragma unroll
        for (int r2 = 0; r2 < 5; r2++) {
          const int src = ptr >= 0 ? ptr : ln;
          const int tv = __shfl_sync(full, val, src);
          const int tp = __shfl_sync(full, ptr, src);
          if (val < 0 && ptr >= 0) {
            if (tv >= 0) val = tv;
            else ptr = tp;
          }
        }
        // active lanes with the same output: one ballot per bit of it
        unsigned peers = __ballot_sync(full, act);
  #pragma unroll
        for (int bit = 0; bit < 8; bit++) {
          const bool on = act && ((val >> bit) & 1);
          const unsigned bb = __ballot_sync(full, on);
          peers &= on ? bb : ~bb;
        }
        const unsigned above = ~((2u << ln) - 1u);  // lanes after this one
        const bool last = act && (peers & above) == 0u;
        const unsigned lastm = __ballot_sync(full, last);
        const int D = __popc(lastm);
        if (ln < 8) used[ln] = 0u;
        __syncwarp();
        if (from_list) atomicOr(&used[p >> 5], 1u << (p & 31));
        __syncwarp();
        uint8_t *nx = lb + 256 * (cur ^ 1);
        if (last) nx[__popc(lastm & above)] = (uint8_t)val;
        const int q0 = 8 * ln;
        int below = 0;
        for (int x = 0; x < (q0 >> 5); x++) below += __popc(used[x]);
        const uint32_t uw = used[q0 >> 5];
        for (int j = 0; j < 8; j++) {
          const int q = q0 + j;
          if (q >= nuse) break;
          const uint32_t bit = 1u << (q & 31);
          if (!(uw & bit)) nx[D + q - below - __popc(uw & (bit - 1u))] = lst[q];
        }
        cur ^= 1;
        rv = val;
        __syncwarp();
      }
      // a run digit's place: the digits just before it
      const unsigned bm = others & ((1u << ln) - 1u);
      const int q = bm ? ln - 32 + __clz(bm) : ln + run;
      const int qc = min(q, 31);
      if (act) rec[i0 + ln] = (uint16_t)(dgt ? kRecRun | (sym << 13) | (qc << 8) | rv : rv);
      if (act) {
        const int64_t bytes = dgt ? (int64_t)(sym + 1) << min(q, 40) : 1;
        if (lead && bm == 0u && dgt) lead_sum += bytes;
        else rest_sum += bytes;
      }
      if (lead) lead_cnt += others ? __ffs(others) - 1 : nb;
      if (others) {
        lead = false;
        run = nb - 32 + __clz(others);
      } else {
        run += nb;
      }
    }
    for (int o = 16; o; o >>= 1) {
      lead_sum += __shfl_xor_sync(full, lead_sum, o);
      rest_sum += __shfl_xor_sync(full, rest_sum, o);
    }
    const uint8_t *lst = lb + 256 * cur;
    for (int q = ln; q < 64; q += 32)
      reinterpret_cast<uint32_t *>(out.list[c])[q] = reinterpret_cast<const uint32_t *>(lst)[q];
    ChunkInfo &ci = out.info[c];
    if (e_at == eob_at && e_at != INT32_MAX) ci.end = e_end;
    if (ln == 0) {
      ci.nsym = n;
      ci.eob = eob_at != INT32_MAX && eob_at < bad_at;
      ci.bad = bad_at < eob_at;
      ci.lead = lead_cnt;
      ci.trail = run;
      ci.lead_sum = lead_sum;
      ci.rest_sum = rest_sum;
    }
    __syncwarp();  // the warp's shared memory is free for the next chunk
  }
}

// Per block: chunk offsets, starting lists, and the block's result.
__global__ void __launch_bounds__(256) k_dec_mscan(const int64_t *cand, const DecTab *tabs,
                                                   uint32_t *tt, int cap, DecBlock *res) {
  __shared__ int64_t scratch[40];
  __shared__ int s_last;
  __shared__ uint8_t lst[2][256];
  const int bi = blockIdx.x;
  const DecTab &tab = tabs[bi];
  DecBlock r;
  r.start = cand[bi];
  r.end = r.start;
  r.m = 0;
  r.orig_ptr = tab.orig_ptr;
  r.crc = tab.crc;
  r.status = tab.status;
  r.nchunks = 0;
  if (r.status != kDecOk) {
    if (threadIdx.x == 0) res[bi] = r;
    return;
  }
  SymScratch &sc = sym_scratch(tt, bi, cap);
  const int nch = (tab.ngv + kChunkGroups - 1) / kChunkGroups;
  if (threadIdx.x == 0) s_last = nch;
  __syncthreads();
  for (int c = threadIdx.x; c < nch; c += 256)
    if (sc.info[c].eob || sc.info[c].bad) atomicMin(&s_last, c);
  __syncthreads();
  const int last = s_last;  // the chunk holding the end of the block (nch: none does)
  if (last == nch || sc.info[last].bad) r.status = kDecBadSymbol;
  const int nc = min(last + 1, nch);
  // bytes per chunk and their offsets
  int64_t total = 0;
  for (int c0 = 0; c0 < nc; c0 += 256) {
    const int c = c0 + threadIdx.x;
    int64_t bytes = 0;
    if (c < nc) {
      // digits just before the chunk (a chunk of nothing else is an overlong run by itself)
      const int q0 = c > 0 ? min(sc.info[c - 1].trail, 40) : 0;
      sc.info[c].q0 = q0;
      // more than 2^30 bytes, or a digit past place 20, is too long in any case
      constexpr int64_t kHuge = (int64_t)1 << 30;
      const int64_t ls = sc.info[c].lead_sum;
      bytes = ls > 0 && (ls > kHuge || q0 > 20) ? kHuge : ls << min(q0, 20);
      bytes = min(kHuge, bytes) + min(kHuge, sc.info[c].rest_sum);
    }
    int64_t tot;
    const int64_t off = total + block_excl_sum(bytes, scratch, &tot);
    if (c < nc) sc.info[c].off = off;
    total += tot;
  }
  if (r.status == kDecOk && total > cap) r.status = kDecTooLong;
  if (r.status == kDecOk) {
    r.m = (int)total;
    r.nchunks = nc;
    r.end = r.start + sc.info[last].end;
    if (r.orig_ptr < 0 || r.orig_ptr >= r.m) r.status = kDecBadOrigPtr;
  }
  if (threadIdx.x == 0) res[bi] = r;
  if (r.status != kDecOk) return;
  // starting lists, in bytes: chunk c + 1's entry k is chunk c's entry P_c[k]
  const int k = threadIdx.x;
  lst[0][k] = k < tab.nuse ? tab.seq2unseq[k] : 0;
  __syncthreads();
  int cur = 0;
  constexpr int kAhead = 8;
  for (int c0 = 0; c0 < nc; c0 += kAhead) {
    uint8_t P[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; q++) P[q] = c0 + q < nc ? sc.list[c0 + q][k] : 0;
#pragma unroll
    for (int q = 0; q < kAhead; q++) {
      if (c0 + q < nc) {
        sc.list[c0 + q][k] = lst[cur][k];
        lst[cur ^ 1][k] = lst[cur][P[q]];
        __syncthreads();
        cur ^= 1;
      }
    }
  }
}

// The last column: a warp per chunk writes its symbols' bytes, long runs by
// all its lanes.
__global__ void __launch_bounds__(32 * kSymWarps)
    k_dec_emit(const DecBlock *res, uint32_t *tt, uint8_t *Lbuf, int cap) {
  __shared__ __align__(4) uint8_t lists[kSymWarps][256];
  const unsigned full = 0xffffffffu;
  const int bi = blockIdx.y;
  if (res[bi].status != kDecOk) return;
  const int ln = lane_id(), w = warp_id();
  const int nch = res[bi].nchunks;
  SymScratch &sc = sym_scratch(tt, bi, cap);
  uint8_t *L = Lbuf + (size_t)bi * cap;
  for (int c = (int)blockIdx.x * kSymWarps + w; c < nch; c += gridDim.x * kSymWarps) {
    const ChunkInfo ci = sc.info[c];
    int64_t off = ci.off;
    for (int q = ln; q < 64; q += 32)
      reinterpret_cast<uint32_t *>(lists[w])[q] = reinterpret_cast<const uint32_t *>(sc.list[c])[q];
    __syncwarp();
    const uint16_t *rec = sc.rec + (size_t)c * kChunkSyms;
    for (int i0 = 0; i0 < ci.nsym; i0 += 32) {
      const int i = i0 + ln;
      const uint32_t r = i < ci.nsym ? rec[i] : 0u;
      int nb = i < ci.nsym ? 1 : 0;
      if (r & kRecRun) {
        const int q = (int)((r >> 8) & 31u) + (i < ci.lead ? ci.q0 : 0);
        nb = (int)(((r >> 13) & 1u) + 1u) << min(q, 28);
      }
      const uint8_t v = lists[w][r & 0xFFu];
      const int inc = warp_incl_sum(nb);
      const int64_t at = off + inc - nb;
      if (nb == 1) L[at] = v;
      else if (nb > 1 && nb <= 64) fill_bytes(L + at, nb, v);
      unsigned big = __ballot_sync(full, nb > 64);
      while (big) {
        const int s = __ffs(big) - 1;
        big &= big - 1u;
        const int bn = __shfl_sync(full, nb, s);
        const int64_t ba = __shfl_sync(full, at, s);
        const uint32_t bv = 0x01010101u * __shfl_sync(full, (uint32_t)v, s);
        uint8_t *d = L + ba;
        const int head = min(bn, (int)((0u - (uint32_t)reinterpret_cast<uintptr_t>(d)) & 15u));
        const int body = (bn - head) / 16;
        if (ln < head) d[ln] = (uint8_t)bv;
        for (int q = ln; q < body; q += 32)
          reinterpret_cast<uint4 *>(d + head)[q] = make_uint4(bv, bv, bv, bv);
        const int done = head + 16 * body;
        if (done + ln < bn) d[done + ln] = (uint8_t)bv;
      }
      off += __shfl_sync(full, inc, 31);
    }
    __syncwarp();  // the list is free for the next chunk
  }
}

// The RLE1 bytes of each block follow tt from origPtr:
// T[j] = psi(j) << 8 | F[j], psi = LF^-1, and the text is F[origPtr],
// F[psi(origPtr)], ...  One dependent load per byte, so the chain is cut at
// every walk_step(m)-th position and at origPtr: a walker per cut follows the
// chain to the next one, the segments are ordered along the chain from origPtr
// by pointer jumping, and their bytes are copied to their place.  Segment
// lengths are close to exponential, so the longest is about ln(walkers) times
// the step.  A walker keeps its bytes in 64-byte chunks of a pool (its own
// first one, then the block's next free ones), so the chain is walked once.
// The step is as small as the ordering's shared memory allows: the walk is
// bound by the latency of its longest segments, and the more walkers a block
// has, the fewer blocks' T (4 bytes per RLE1 byte) are in use at a time, which
// keeps them in L2.  Two walks of steps of 512 took 0.67 ms each for one block
// and 4.7 ms each for 600 blocks.
constexpr int kMaxWalkers = (kDecCap + 127) / 128 + 2;
constexpr int kMaxWalkChunks = kMaxWalkers + kDecCap / kWalkChunk + 1;
constexpr int kChainThreads = 1024;
constexpr int kChainPer = (kMaxWalkers + kChainThreads - 1) / kChainThreads;
constexpr int kNoWalker = 0xFFFF;
static_assert(kMaxWalkers < (1 << 14) && kDecCap / kWalkChunk < (1 << 18), "chunk owner packing");

// The walker that starts at a cut.
__device__ __forceinline__ int walker_at(int p, int m, int orig) {
  const int s = walk_step(m);
  return p % s == 0 ? p / s : (m + s - 1) / s;
}

struct WalkCtl {
  int32_t cycle;     // bytes of the chain from origPtr before it closes (m if it does not)
  int32_t nchunks;   // pool chunks taken
  int32_t len[kMaxWalkers];     // segment length (steps to the next cut)
  uint16_t next[kMaxWalkers];   // the walker there
  int32_t off[kMaxWalkers];     // output offset, -1 when off the chain
  uint32_t owner[kMaxWalkChunks];  // chunk: walker | its place among the walker's << 14
};

// LF vector without serial ranks: T[C[L[i]] + rank(i)] = i << 8 | L[i], with
// rank(i) = #{j < i : L[j] == L[i]} (then for j = LF(i), psi(j) = i and
// F[j] = L[i]).  A stable counting sort by the byte: per 4096-entry chunk a
// histogram, per block a scan over chunks (each chunk's start per byte value,
// C included), then per chunk the ranks of 256 entries at a time: equal bytes
// in a warp by ballots, earlier warps by shared counts.
constexpr int kLfChunks = (kDecCap + kLfChunk - 1) / kLfChunk;

__global__ void __launch_bounds__(256) k_dec_lf_hist(const int32_t *idx, const DecBlock *db,
                                                     const uint8_t *Lbuf, int32_t *H, int cap) {
  __shared__ int cnt[256];
  const int k = blockIdx.y, ch = blockIdx.x;
  const int bi = idx[k];
  const int m = db[bi].m;
  const int c0 = ch * kLfChunk;
  if (c0 >= m) return;
  const uint8_t *L = Lbuf + (size_t)bi * cap;
  cnt[threadIdx.x] = 0;
  __syncthreads();
  const int c1 = min(m, c0 + kLfChunk);
  for (int i = c0 + threadIdx.x; i < c1; i += 256) atomicAdd(&cnt[L[i]], 1);
  __syncthreads();
  H[((size_t)k * kLfChunks + ch) * 256 + threadIdx.x] = cnt[threadIdx.x];
}

// Per block (thread = byte value): H[chunk][c] becomes the position of the
// chunk's first c in F order.
__global__ void __launch_bounds__(256) k_dec_lf_scan(const int32_t *idx, const DecBlock *db,
                                                     int32_t *H, WalkCtl *ctl) {
  __shared__ int scratch[40];
  const int k = blockIdx.x;
  const int m = db[idx[k]].m;
  // every walker owns the pool chunk of its number; the next ones are free
  if (threadIdx.x == 0) ctl[k].nchunks = walker_count(m, db[idx[k]].orig_ptr);
  const int nch = (m + kLfChunk - 1) / kLfChunk;
  int32_t *h = H + (size_t)k * kLfChunks * 256 + threadIdx.x;
  int tot = 0;
  for (int ch = 0; ch < nch; ch++) tot += h[(size_t)ch * 256];
  int all;
  int run = block_excl_sum(tot, scratch, &all);  // C[c]
  for (int ch = 0; ch < nch; ch++) {
    const int v = h[(size_t)ch * 256];
    h[(size_t)ch * 256] = run;
    run += v;
  }
}

__global__ void __launch_bounds__(256) k_dec_lf_rank(const int32_t *idx, const DecBlock *db,
                                                     const uint8_t *Lbuf, const int32_t *H,
                                                     uint32_t *tt, int cap) {
  __shared__ int run[256];
  __shared__ int wc[8][256];
  const int k = blockIdx.y, ch = blockIdx.x;
  const int bi = idx[k];
  const int m = db[bi].m;
  const int c0 = ch * kLfChunk;
  if (c0 >= m) return;
  const uint8_t *L = Lbuf + (size_t)bi * cap;
  uint32_t *T = tt + (size_t)k * cap;
  const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
  run[threadIdx.x] = H[((size_t)k * kLfChunks + ch) * 256 + threadIdx.x];
  for (int sub = 0; sub < kLfChunk / 256; sub++) {
    const int i = c0 + sub * 256 + threadIdx.x;
    if (c0 + sub * 256 >= m) break;  // uniform
    const bool valid = i < m;
    const int c = valid ? (int)L[i] : 256 + ln;
    for (int q = threadIdx.x; q < 8 * 256; q += 256) (&wc[0][0])[q] = 0;
    __syncthreads();
    // lanes with the same byte: one ballot per bit (cheaper than match_any)
    unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int bit = 0; bit < 8; bit++) {
      const bool on = (c >> bit) & 1;
      const unsigned bb = __ballot_sync(0xffffffffu, on);
      peers &= on ? bb : ~bb;
    }
    const int wr = __popc(peers & ((1u << ln) - 1u));
    if (valid && wr == 0) wc[w][c] = __popc(peers);
    __syncthreads();
    if (valid) {
      int j = run[c] + wr;
      for (int q = 0; q < w; q++) j += wc[q][c];
      if (j >= 0 && j < m) T[j] = ((uint32_t)i << 8) | (uint32_t)c;
    }
    __syncthreads();
    if (valid && wr == 0) atomicAdd(&run[c], __popc(peers));
  }
}

__global__ void __launch_bounds__(kWalkThreads) k_dec_walk(const int32_t *idx, const DecBlock *db,
                                                           const uint32_t *tt, WalkCtl *ctl,
                                                           uint8_t *pool, int cap) {
  const int k = blockIdx.y;
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  WalkCtl &c = ctl[k];
  const DecBlock b = db[idx[k]];
  const int m = b.m, orig = b.orig_ptr;
  if (w >= walker_count(m, orig)) return;
  const uint32_t *T = tt + (size_t)k * cap;
  uint8_t *P = pool + (size_t)k * kMaxWalkChunks * kWalkChunk;
  const int step = walk_step(m);  // a power of two
  int p = w * step < m ? w * step : orig;
  uint32_t *chunk = reinterpret_cast<uint32_t *>(P + (size_t)w * kWalkChunk);
  c.owner[w] = (uint32_t)w;
  int n = 0;
  uint32_t acc = 0;
  // T is a permutation, so segments are disjoint and a walk ends within m steps
  for (;;) {
    const uint32_t e = T[p];
    acc |= (e & 0xFFu) << (8 * (n & 3));
    n++;
    p = (int)(e >> 8);
    const bool end = (p & (step - 1)) == 0 || p == orig || n >= m;
    if ((n & 3) == 0 || end) {
      chunk[((n - 1) & (kWalkChunk - 1)) >> 2] = acc;
      acc = 0;
    }
    if (end) break;
    if ((n & (kWalkChunk - 1)) == 0) {
      const int q = atomicAdd(&c.nchunks, 1);
      c.owner[q] = (uint32_t)w | (uint32_t)(n / kWalkChunk) << 14;
      chunk = reinterpret_cast<uint32_t *>(P + (size_t)q * kWalkChunk);
    }
  }
  c.len[w] = n;
  c.next[w] = (uint16_t)walker_at(p, m, orig);
}

// Per block: segment offsets along the chain from origPtr.  The chain is
// opened before origPtr's walker; pointer jumping sums the lengths from each
// walker to the end (walkers of other cycles never reach it).
constexpr size_t kChainSmem = (size_t)kMaxWalkers * 6 + 16;

__global__ void __launch_bounds__(kChainThreads) k_dec_chain(const int32_t *idx,
                                                             const DecBlock *db, WalkCtl *ctl,
                                                             int *bad) {
  extern __shared__ uint32_t chain_smem[];
  uint32_t *sum = chain_smem;
  uint16_t *nxt = reinterpret_cast<uint16_t *>(sum + kMaxWalkers);
  const int k = blockIdx.x;
  const DecBlock b = db[idx[k]];
  WalkCtl &c = ctl[k];
  const int nw = walker_count(b.m, b.orig_ptr);
  const int w0 = walker_at(b.orig_ptr, b.m, b.orig_ptr);
  for (int q = threadIdx.x; q < nw; q += kChainThreads) {
    sum[q] = (uint32_t)c.len[q];
    const int x = c.next[q];
    nxt[q] = (uint16_t)(x == w0 ? kNoWalker : x);
  }
  __syncthreads();
  for (int span = 1; span < nw; span <<= 1) {
    uint32_t s[kChainPer];
    uint16_t x[kChainPer];
#pragma unroll
    for (int j = 0; j < kChainPer; j++) {
      const int q = threadIdx.x + j * kChainThreads;
      if (q < nw) {
        x[j] = nxt[q];
        s[j] = sum[q];
        if (x[j] != kNoWalker) {
          s[j] += sum[x[j]];
          x[j] = nxt[x[j]];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kChainPer; j++) {
      const int q = threadIdx.x + j * kChainThreads;
      if (q < nw) {
        sum[q] = s[j];
        nxt[q] = x[j];
      }
    }
    __syncthreads();
  }
  const uint32_t total = sum[w0];
  for (int q = threadIdx.x; q < nw; q += kChainThreads)
    c.off[q] = nxt[q] == kNoWalker ? (int32_t)(total - sum[q]) : -1;
  if (threadIdx.x == 0) {
    const int cyc = (int)min(total, (uint32_t)b.m);
    c.cycle = cyc;
    if (cyc <= 0 || b.m % cyc != 0 || total > (uint32_t)b.m) atomicOr(bad, 1);
  }
}

// The walkers' chunks to their places: 16 threads per chunk, 4 bytes each.
__global__ void __launch_bounds__(256) k_dec_gather(const int32_t *idx, const DecBlock *db,
                                                    const WalkCtl *ctl, const uint8_t *pool,
                                                    uint8_t *rle, int cap) {
  const int k = blockIdx.y;
  const WalkCtl &c = ctl[k];
  const int bi = idx[k];
  const int m = db[bi].m;
  const int nq = min(c.nchunks, kMaxWalkChunks);
  const uint8_t *P = pool + (size_t)k * kMaxWalkChunks * kWalkChunk;
  uint8_t *R = rle + (size_t)bi * cap;
  const int l = 4 * (threadIdx.x & 15);
  const int q1 = min(nq, ((int)blockIdx.x + 1) * kGatherChunks);
  for (int q = blockIdx.x * kGatherChunks + (threadIdx.x >> 4); q < q1; q += 16) {
    const uint32_t ow = c.owner[q];
    const int w = (int)(ow & 0x3FFFu), at = (int)(ow >> 14) * kWalkChunk + l;
    const int off = c.off[w], n = c.len[w] - at;
    if (off < 0 || n <= 0) continue;
    const uint32_t v = *reinterpret_cast<const uint32_t *>(P + (size_t)q * kWalkChunk + l);
#pragma unroll
    for (int z = 0; z < 4; z++)
      if (z < n && off + at + z < m) R[off + at + z] = (uint8_t)(v >> (8 * z));
  }
}

// A periodic block: the first `cycle` bytes repeated to m.
__global__ void k_dec_repeat(const int32_t *idx, const DecBlock *db, const WalkCtl *ctl,
                             uint8_t *rle, int cap) {
  const int k = blockIdx.y;
  const int m = db[idx[k]].m;
  const int cyc = ctl[k].cycle;
  if (cyc <= 0 || cyc >= m) return;
  uint8_t *R = rle + (size_t)idx[k] * cap;
  for (int i = cyc + blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    R[i] = R[i % cyc];
}


// Inverse RLE1 (4 equal bytes are followed by a count of further copies).
// The block's RLE1 bytes are cut into segments of 32, one thread each, 256 to
// a tile.  What a segment produces depends only on the run state it starts
// in: 0 = no run (block start, or just after a count byte), 1..3 = the byte
// before the segment closes a run of that length, 4 = the next byte is a
// count.  A segment is followed from all five states at once until they merge
// (typically within a few bytes: at a byte that differs from the one before
// it); its map "state before -> state after, bytes written" is one of an
// associative set, so scans over a tile's segments, and over a block's tiles,
// give every segment its state and offset.  The write pass forms the maps of
// its tile again instead of reading them back (they would be 20 bytes per 32).
// One warp per block took 3.5 + 1.0 ms for a single block, the latency of
// 7,500 bytes per lane one after another.
constexpr int kSegBytes = 32;
static_assert(kUnTile == 256 * kSegBytes, "a thread per segment");
constexpr int kUnTiles = (kDecCap + kUnTile - 1) / kUnTile;
constexpr int kSegStride = kSegBytes + 4;  // in shared memory: lanes on different banks

// state after (bits 29-31) and bytes written, for each state before
struct RunMap {
  uint32_t v[5];
};
constexpr uint32_t kRunBytes = (1u << 29) - 1u;

__device__ __forceinline__ uint32_t pick5(uint32_t x, const uint32_t (&a)[5]) {
  return x == 0 ? a[0] : x == 1 ? a[1] : x == 2 ? a[2] : x == 3 ? a[3] : a[4];
}
// f, then g
__device__ __forceinline__ RunMap run_then(const RunMap &f, const RunMap &g) {
  RunMap h;
#pragma unroll
  for (int q = 0; q < 5; q++) h.v[q] = pick5(f.v[q] >> 29, g.v) + (f.v[q] & kRunBytes);
  return h;
}
__device__ __forceinline__ RunMap run_identity() {
  RunMap h;
#pragma unroll
  for (int q = 0; q < 5; q++) h.v[q] = (uint32_t)q << 29;
  return h;
}

__device__ __forceinline__ void rle1_step(int &r, int &n, int c, int p) {
  if (r == 4) {
    n += c;
    r = 0;
  } else if (r >= 1 && c == p) {
    r++;
    n++;
  } else {
    r = 1;
    n++;
  }
}

// Loads the tile's bytes (thread t's segment at t * kSegStride) and returns
// the bytes of this thread's segment; *prev: the byte before it (-1: none).
__device__ __forceinline__ int load_segments(const uint8_t *R, int m, int tile, uint8_t *sb,
                                             int *prev) {
  const int t0 = tile * kUnTile;
  const int len = min(kUnTile, m - t0);
  for (int q = threadIdx.x; q < (len + 15) / 16; q += 256) {
    const uint4 v = reinterpret_cast<const uint4 *>(R + t0)[q];  // rows are 16-byte aligned
    uint32_t *d = reinterpret_cast<uint32_t *>(sb + (q >> 1) * kSegStride + (q & 1) * 16);
    d[0] = v.x;
    d[1] = v.y;
    d[2] = v.z;
    d[3] = v.w;
  }
  __syncthreads();
  const int s0 = threadIdx.x * kSegBytes;
  *prev = -1;
  if (threadIdx.x > 0) *prev = sb[(threadIdx.x - 1) * kSegStride + kSegBytes - 1];
  else if (t0 > 0) *prev = R[t0 - 1];
  return max(0, min(kSegBytes, len - s0));
}

__device__ __forceinline__ RunMap segment_map(const uint8_t *seg, int n, int p) {
  int r0 = 0, r1 = 1, r2 = 2, r3 = 3, r4 = 4;
  int n0 = 0, n1 = 0, n2 = 0, n3 = 0, n4 = 0;
  int i = 0;
  bool merged = false;
  while (i < n && !merged) {
    const int c = seg[i++];
    rle1_step(r0, n0, c, p);
    rle1_step(r1, n1, c, p);
    rle1_step(r2, n2, c, p);
    rle1_step(r3, n3, c, p);
    rle1_step(r4, n4, c, p);
    p = c;
    merged = r0 == r1 && r0 == r2 && r0 == r3 && r0 == r4;
  }
  if (merged) {
    int r = r0, nb = 0;
    while (i < n) {
      const int c = seg[i++];
      rle1_step(r, nb, c, p);
      p = c;
    }
    r0 = r1 = r2 = r3 = r4 = r;
    n0 += nb;
    n1 += nb;
    n2 += nb;
    n3 += nb;
    n4 += nb;
  }
  RunMap h;
  h.v[0] = ((uint32_t)r0 << 29) | (uint32_t)n0;
  h.v[1] = ((uint32_t)r1 << 29) | (uint32_t)n1;
  h.v[2] = ((uint32_t)r2 << 29) | (uint32_t)n2;
  h.v[3] = ((uint32_t)r3 << 29) | (uint32_t)n3;
  h.v[4] = ((uint32_t)r4 << 29) | (uint32_t)n4;
  return h;
}

// Exclusive scan of the tile's maps (256 threads); *total: the tile's map.
__device__ __forceinline__ RunMap scan_maps(RunMap mine, RunMap (&wm)[8], RunMap *total) {
  const int ln = lane_id(), w = warp_id();
  RunMap inc = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    RunMap o;
#pragma unroll
    for (int q = 0; q < 5; q++) o.v[q] = __shfl_up_sync(0xffffffffu, inc.v[q], d);
    if (ln >= d) inc = run_then(o, inc);
  }
  if (ln == 31) wm[w] = inc;
  RunMap ex;
#pragma unroll
  for (int q = 0; q < 5; q++) ex.v[q] = __shfl_up_sync(0xffffffffu, inc.v[q], 1);
  if (ln == 0) ex = run_identity();
  __syncthreads();
  RunMap pre = run_identity();
  for (int q = 0; q < w; q++) pre = run_then(pre, wm[q]);
  if (total) *total = run_then(pre, wm[7]);  // meaningful in the last warp
  return run_then(pre, ex);
}

// grid: (tile, block)
__global__ void __launch_bounds__(256) k_dec_unrle1_count(const int32_t *idx, const DecBlock *db,
                                                          const uint8_t *rle, int cap,
                                                          RunMap *maps) {
  __shared__ __align__(16) uint8_t sb[256 * kSegStride];
  __shared__ RunMap wm[8];
  const int k = blockIdx.y, tile = blockIdx.x;
  const int bi = idx[k];
  const int m = db[bi].m;
  if (tile * kUnTile >= m) return;
  int prev;
  const int n = load_segments(rle + (size_t)bi * cap, m, tile, sb, &prev);
  RunMap total;
  scan_maps(segment_map(sb + threadIdx.x * kSegStride, n, prev), wm, &total);
  if (threadIdx.x == 255) maps[(size_t)k * kUnTiles + tile] = total;
}

// Per block: every tile's state and offset (map v[0] = state, v[1..2] = its
// 64-bit offset) and the block's length.
__global__ void __launch_bounds__(256) k_dec_unrle1_scan(const int32_t *idx, const DecBlock *db,
                                                         RunMap *maps, int64_t *lens) {
  __shared__ RunMap tm[kUnTiles];
  const int k = blockIdx.x;
  const int nt = (db[idx[k]].m + kUnTile - 1) / kUnTile;
  RunMap *mp = maps + (size_t)k * kUnTiles;
  for (int q = threadIdx.x; q < nt; q += 256) tm[q] = mp[q];
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t state = 0;
    int64_t off = 0;
    for (int q = 0; q < nt; q++) {
      const uint32_t e = pick5(state, tm[q].v);
      tm[q].v[0] = state;
      tm[q].v[1] = (uint32_t)off;
      tm[q].v[2] = (uint32_t)(off >> 32);
      state = e >> 29;
      off += e & kRunBytes;
    }
    lens[k] = off;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nt; q += 256) mp[q] = tm[q];
}

// Sequential byte writer: whole words where the thread owns them, bytes at
// its two ends.
struct ByteWriter {
  uint8_t *o;     // next byte
  uint8_t *lo;    // first byte
  uint32_t acc;
  __device__ __forceinline__ void init(uint8_t *p) {
    o = lo = p;
    acc = 0;
  }
  __device__ __forceinline__ void store_part(uint8_t *from) {  // bytes [from, o) of one word
    for (uint8_t *q = from; q < o; q++)
      *q = (uint8_t)(acc >> (8 * (int)(reinterpret_cast<uintptr_t>(q) & 3u)));
  }
  __device__ __forceinline__ void put(uint32_t c) {
    const int sh = 8 * (int)(reinterpret_cast<uintptr_t>(o) & 3u);
    acc = (sh ? acc : 0u) | (c << sh);
    o++;
    if (sh == 24) {
      if (o - lo >= 4) *reinterpret_cast<uint32_t *>(o - 4) = acc;
      else store_part(lo);
    }
  }
  __device__ __forceinline__ void fill(uint32_t c, int n) {
    while (n > 0 && (reinterpret_cast<uintptr_t>(o) & 3u)) {
      put(c);
      n--;
    }
    const uint32_t wv = 0x01010101u * c;
    while (n >= 4 && (reinterpret_cast<uintptr_t>(o) & 15u)) {
      *reinterpret_cast<uint32_t *>(o) = wv;
      o += 4;
      n -= 4;
    }
    for (; n >= 16; n -= 16, o += 16) *reinterpret_cast<uint4 *>(o) = make_uint4(wv, wv, wv, wv);
    for (; n >= 4; n -= 4, o += 4) *reinterpret_cast<uint32_t *>(o) = wv;
    while (n-- > 0) put(c);
  }
  __device__ __forceinline__ void finish() {
    const int k = (int)(reinterpret_cast<uintptr_t>(o) & 3u);
    if (k && o > lo) store_part(o - k > lo ? o - k : lo);
  }
};

__global__ void __launch_bounds__(256) k_dec_unrle1_write(const int32_t *idx, const DecBlock *db,
                                                          const uint8_t *rle, int cap,
                                                          const RunMap *maps, const int64_t *off,
                                                          uint8_t *out) {
  __shared__ __align__(16) uint8_t sb[256 * kSegStride];
  __shared__ RunMap wm[8];
  const int k = blockIdx.y, tile = blockIdx.x;
  const int bi = idx[k];
  const int m = db[bi].m;
  if (tile * kUnTile >= m) return;
  int p;
  const int n = load_segments(rle + (size_t)bi * cap, m, tile, sb, &p);
  const uint8_t *seg = sb + threadIdx.x * kSegStride;
  const RunMap ex = scan_maps(segment_map(seg, n, p), wm, nullptr);
  const RunMap &tm = maps[(size_t)k * kUnTiles + tile];
  const uint32_t e = pick5(tm.v[0], ex.v);
  int r = (int)(e >> 29);
  ByteWriter bw;
  bw.init(out + off[k] + (((int64_t)tm.v[2] << 32) | tm.v[1]) + (e & kRunBytes));
  for (int i = 0; i < n; i++) {
    const int c = seg[i];
    if (r == 4) {
      bw.fill((uint32_t)p, c);
      r = 0;
    } else {
      r = (r >= 1 && c == p) ? r + 1 : 1;
      bw.put((uint32_t)c);
    }
    p = c;
  }
  bw.finish();
}

// Block CRCs of the expanded output.  gridDim.x CTAs share a block's
// 4096-byte chunks; in a chunk thread l's 16 bytes give crc0 *
// x^(8*16*(255-l)) (the chunk right-aligned in 4096 bytes when shorter), the
// XOR is the chunk's crc0, a CTA's crc0 accumulates chunk by chunk and is
// shifted past the bytes after its part.  crcs: all ones before (the format's
// complement); the initial value's term comes with part 0.
__global__ void __launch_bounds__(256) k_dec_crc(const int64_t *lens, const int64_t *off,
                                                 const uint8_t *out, uint32_t *crcs) {
  __shared__ uint32_t tbl[256];
  __shared__ uint32_t red4[16];
  __shared__ uint32_t part[2][8];
  const int k = blockIdx.y;
  const int64_t n = lens[k];
  const int64_t nch = (n + kCrcChunk - 1) / kCrcChunk;
  const int64_t per = (nch + gridDim.x - 1) / gridDim.x;
  const int64_t b0 = (int64_t)blockIdx.x * per * 4096;
  const int64_t b1 = b0 + per * 4096 < n ? b0 + per * 4096 : n;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    atomicXor(&crcs[k], gf_mul(0xFFFFFFFFu, xpow8((uint64_t)n)));
  if (b0 >= b1) return;
  crc_table_fill(tbl);
  red4_fill(red4);
  __syncthreads();
  const uint8_t *src = out + off[k];
  uint32_t acc = 0;  // thread 0
  int it = 0;
  for (int64_t base = b0; base < b1; base += 4096, it++) {
    const int len = b1 - base < 4096 ? (int)(b1 - base) : 4096;
    const int at = 16 * (int)threadIdx.x - (4096 - len);  // this thread's first byte in the chunk
    uint32_t r = 0;
    if (at >= 0) {
      // 16 bytes from any address: five aligned words (the buffer has slack)
      const uintptr_t a = reinterpret_cast<uintptr_t>(src + base + at);
      const uint32_t *wp = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
      const int sh = 8 * (int)(a & 3u);
      uint32_t lo = wp[0];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t hi = wp[q + 1];
        const uint32_t x = __funnelshift_r(lo, hi, sh);
        lo = hi;
#pragma unroll
        for (int z = 0; z < 4; z++) r = crc_byte(r, (x >> (8 * z)) & 0xFFu, tbl);
      }
    } else {
      for (int q = -at; q < 16; q++) r = crc_byte(r, src[base + at + q], tbl);
    }
    r = gf_mul_lane(r, threadIdx.x, red4);
    for (int o = 16; o; o >>= 1) r ^= __shfl_xor_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0) part[it & 1][threadIdx.x >> 5] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t c = 0;
      for (int q = 0; q < 8; q++) c ^= part[it & 1][q];
      // acc * x^(8 len) ^ c
      acc = (acc ? gf_mul(acc, len == 4096 ? c_xpow[12] : xpow8((uint64_t)len)) : 0u) ^ c;
    }
  }
  if (threadIdx.x == 0) atomicXor(&crcs[k], gf_mul(acc, xpow8((uint64_t)(n - b1))));
}

struct DevMem {
  static void *alloc(size_t bytes) {
    void *p = nullptr;
    const cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      return nullptr;
    }
    BZ_CUDA(e);
    return p;
  }
  static void free(void *p) { BZ_CUDA(cudaFree(p)); }  // waits for kernels that use it
};
using DevBuf = GrowBuf<DevMem>;

// Where decoded bytes go, batch by batch, in stream order.
struct DecSink {
  size_t size = 0;
  virtual ~DecSink() = default;
  // Queue the copy of n device bytes to the end of the output on stream cs.
  virtual void put(const uint8_t *d_src, size_t n, cudaStream_t cs) = 0;
};

// A caller's buffer of cap bytes (host or device memory).
struct BufferSink : DecSink {
  uint8_t *dst;
  size_t cap;
  BufferSink(uint8_t *d, size_t c) : dst(d), cap(c) {}
  void put(const uint8_t *d_src, size_t n, cudaStream_t cs) override {
    BZ_REQUIRE(n <= cap - size, kErrTooLarge,
               "decoded data larger than the output buffer (" + std::to_string(cap) + " bytes)");
    if (n) BZ_CUDA(cudaMemcpyAsync(dst + size, d_src, n, cudaMemcpyDefault, cs));
    size += n;
  }
};

// A malloc'ed host buffer grown by realloc (large blocks are remapped, not
// copied, and pages are touched only by the copies into them).
struct MallocSink : DecSink {
  uint8_t *buf = nullptr;
  size_t cap = 0;
  ~MallocSink() override { std::free(buf); }
  void put(const uint8_t *d_src, size_t n, cudaStream_t cs) override {
    if (n > cap - size) {
      BZ_CUDA(cudaStreamSynchronize(cs));  // no copy into the old buffer in flight
      const size_t nc = std::max(size + n, 2 * cap);
      void *q = std::realloc(buf, nc);
      BZ_REQUIRE(q != nullptr, kErrAlloc, "host allocation failed");
      buf = static_cast<uint8_t *>(q);
      cap = nc;
    }
    if (n) BZ_CUDA(cudaMemcpyAsync(buf + size, d_src, n, cudaMemcpyDefault, cs));
    size += n;
  }
  uint8_t *release() {
    uint8_t *p = buf;
    if (!p) p = static_cast<uint8_t *>(std::malloc(1));
    else if (size && size < cap) p = static_cast<uint8_t *>(std::realloc(buf, size));
    BZ_REQUIRE(p != nullptr, kErrAlloc, "host allocation failed");
    buf = nullptr;
    cap = 0;
    return p;
  }
};

// The decoder's device scratch, one per device, grown on demand and kept
// between calls.  Output batches alternate between two device buffers: the
// copy of one batch to the sink (stream cs) overlaps the decoding of the next
// (stream st).
struct DecWork {
  std::mutex mu;
  DevBuf words, blk, eos, cnt, cand, order, db, tab, gstart, L, hist, sel, idx, tt, lens, off, crc,
      ctl, pool, bad, maps, jumps, jt0, lutlen;
  DevBuf out[2];
  cudaStream_t st = nullptr, cs = nullptr;
  cudaEvent_t written[2] = {nullptr, nullptr}, copied[2] = {nullptr, nullptr};
  bool used[2] = {false, false};
  uint32_t *h_crc = nullptr;  // pinned
  size_t h_crc_cap = 0;
  int sms = 0;
  int resident = 0;  // k_dec_groups blocks resident on the whole device

  void init() {
    if (st) return;
    BZ_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    BZ_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    for (int q = 0; q < 2; q++) {
      BZ_CUDA(cudaEventCreateWithFlags(&written[q], cudaEventDisableTiming));
      BZ_CUDA(cudaEventCreateWithFlags(&copied[q], cudaEventDisableTiming));
    }
    int dev = 0, per_sm = 0;
    BZ_CUDA(cudaGetDevice(&dev));
    BZ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    BZ_CUDA(cudaFuncSetAttribute(k_dec_jumps, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kJumpSmem));
    BZ_CUDA(cudaFuncSetAttribute(k_dec_starts, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kStartsSmem));
    BZ_CUDA(cudaFuncSetAttribute(k_dec_chain, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kChainSmem));
    BZ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_dec_groups<4>, 128, 0));
    resident = std::max(1, sms * per_sm);
  }
  // The jumps' scratch (up to 2.5 GB) is the one that a call can do without:
  // it is given up where any other is refused.
  void reserve(DevBuf &b, size_t bytes) {
    BZ_REQUIRE(reserve_or_free(b, bytes, jumps), kErrCuda,
               "decoder: device allocation of " + std::to_string(bytes) + " bytes failed");
  }
  // What a batch's size counts on: all that is kept and grows with it.
  size_t held() const {
    size_t s = 0;
    for (const DevBuf *b : {&L, &hist, &tt, &sel, &tab, &gstart, &ctl, &pool, &maps, &lutlen,
                            &jumps, &out[0], &out[1]})
      s += b->cap;
    return s;
  }
};

DecWork &dec_work() {
  static std::mutex mu;
  static std::vector<DecWork *> per_device;  // kept for the process lifetime
  int dev = 0;
  BZ_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  if ((int)per_device.size() <= dev) per_device.resize(dev + 1, nullptr);
  if (!per_device[dev]) per_device[dev] = new DecWork();
  return *per_device[dev];
}

// Device bytes of one candidate slot: last column (later the RLE1 bytes), LF
// vector (before it the symbols), chunk histograms, selectors and group
// starts, tables, walk control and pool.
constexpr size_t kSlotBytes = (size_t)kDecCap * 5 + (size_t)kLfChunks * 256 * 4 + kDecMaxSel * 5 +
                              sizeof(DecTab) + sizeof(WalkCtl) + sizeof(DecBlock) +
                              (size_t)kMaxWalkChunks * kWalkChunk +
                              sizeof(RunMap) * kUnTiles + kLensBytes + 64;
static_assert(kSlotBytes / 100000 == 84, "8.4 MB, as documented");
constexpr int kMaxBatch = 4096;

bool is_header(const uint8_t *h) {
  return h[0] == 'B' && h[1] == 'Z' && h[2] == 'h' && h[3] >= '1' && h[3] <= '9';
}

// The decoder proper.  w.words holds the n stream bytes, zero-padded to whole
// words plus two.
void decode_words(DecWork &w, size_t n, DecSink &sink) {
  cudaStream_t st = w.st, cs = w.cs;
  // on every exit no kernel or copy is left in flight (the sink's memory may
  // be released by the caller)
  struct Drain {
    cudaStream_t a, b;
    ~Drain() {
      cudaStreamSynchronize(a);
      cudaStreamSynchronize(b);
    }
  } drain{st, cs};
  const uint8_t *bytes = w.words.get<uint8_t>();
  const int64_t nwords = (int64_t)(n + 3) / 4 + 2;
  uint8_t head[4];
  BZ_CUDA(cudaMemcpyAsync(head, bytes, 4, cudaMemcpyDeviceToHost, st));
  BZ_CUDA(cudaStreamSynchronize(st));
  BZ_REQUIRE(is_header(head), kErrArg, "not a bzip2 stream (bad header)");
  const int64_t nbits = (int64_t)n * 8;
  // candidates
  const int ccap = (int)std::min<int64_t>((int64_t)n / 8 + 64, 1 << 26);
  w.reserve(w.blk, 8 * (size_t)ccap);
  w.reserve(w.eos, 8 * (size_t)ccap);
  w.reserve(w.cnt, 8);
  BZ_CUDA(cudaMemsetAsync(w.cnt.p, 0, 8, st));
  k_dec_magic<<<(unsigned)((nwords + 255) / 256), 256, 0, st>>>(
      w.words.get<uint32_t>(), nwords, nbits, w.blk.get<int64_t>(), w.cnt.get<int>(),
      w.eos.get<int64_t>(), w.cnt.get<int>() + 1, ccap);
  BZ_LAUNCH_CHECK();
  int hcnt[2];
  BZ_CUDA(cudaMemcpyAsync(hcnt, w.cnt.p, 8, cudaMemcpyDeviceToHost, st));
  BZ_CUDA(cudaStreamSynchronize(st));
  BZ_REQUIRE(hcnt[0] <= ccap && hcnt[1] <= ccap, kErrTooLarge, "too many block candidates");
  std::vector<int64_t> cands(hcnt[0]), eoss(hcnt[1]);
  if (hcnt[0])
    BZ_CUDA(cudaMemcpyAsync(cands.data(), w.blk.p, 8 * hcnt[0], cudaMemcpyDeviceToHost, st));
  if (hcnt[1])
    BZ_CUDA(cudaMemcpyAsync(eoss.data(), w.eos.p, 8 * hcnt[1], cudaMemcpyDeviceToHost, st));
  BZ_CUDA(cudaStreamSynchronize(st));
  std::sort(cands.begin(), cands.end());
  std::sort(eoss.begin(), eoss.end());
  // batch: whole waves of resident k_dec_groups blocks where memory allows
  size_t freeb = 0, totb = 0;
  BZ_CUDA(cudaMemGetInfo(&freeb, &totb));
  int bmax = (int)std::min<size_t>(kMaxBatch, (freeb + w.held()) / 3 / kSlotBytes);
  bmax = std::max(bmax, 32);
  if (bmax >= w.resident) bmax = bmax / w.resident * w.resident;
  // BZ2G_DECODE_BATCH caps the blocks per batch (smaller batches, less memory)
  if (const char *e = std::getenv("BZ2G_DECODE_BATCH")) {
    const int v = std::atoi(e);
    if (v > 0) bmax = std::min(bmax, v);
  }
  const Starts starts = starts_choice();
  const int batch = (int)std::min<size_t>(bmax, std::max<size_t>(cands.size(), 1));
  const int cap = kDecCap;
  w.reserve(w.cand, 8 * (size_t)batch);
  w.reserve(w.order, 4 * (size_t)batch);
  w.reserve(w.db, sizeof(DecBlock) * (size_t)batch);
  w.reserve(w.L, (size_t)batch * cap);
  w.reserve(w.hist, (size_t)batch * kLfChunks * 256 * 4);
  w.reserve(w.sel, (size_t)batch * kDecMaxSel);
  w.reserve(w.gstart, (size_t)batch * kDecMaxSel * 4);
  w.reserve(w.tab, (size_t)batch * sizeof(DecTab));
  w.reserve(w.idx, 4 * (size_t)batch);
  w.reserve(w.tt, (size_t)batch * cap * 4);
  w.reserve(w.lens, 8 * (size_t)batch);
  w.reserve(w.off, 8 * (size_t)batch);
  w.reserve(w.crc, 4 * (size_t)batch);
  w.reserve(w.ctl, sizeof(WalkCtl) * (size_t)batch);
  w.reserve(w.pool, (size_t)kMaxWalkChunks * kWalkChunk * (size_t)batch);
  w.reserve(w.bad, 16);
  w.reserve(w.maps, sizeof(RunMap) * kUnTiles * (size_t)batch);
  if (w.h_crc_cap < (size_t)batch) {
    if (w.h_crc) BZ_CUDA(cudaFreeHost(w.h_crc));
    w.h_crc = nullptr;
    w.h_crc_cap = 0;
    BZ_CUDA(cudaMallocHost((void **)&w.h_crc, 4 * (size_t)batch));
    w.h_crc_cap = batch;
  }
  uint8_t *L = w.L.get<uint8_t>();  // the RLE1 bytes overwrite the last column
  int64_t expect = 32;              // next block or end-of-stream marker
  uint32_t stream_crc = 0;
  bool stream_done = false;
  size_t ci = 0;
  int nbatch = 0;
  std::vector<DecBlock> hdb(batch);
  std::vector<int32_t> order;
  // block CRCs of the last batch, checked once st has caught up
  std::vector<uint32_t> want;
  auto settle = [&]() {
    if (want.empty()) return;
    BZ_CUDA(cudaStreamSynchronize(st));
    for (size_t q = 0; q < want.size(); q++) {
      BZ_REQUIRE(w.h_crc[q] == want[q], kErrArg, "bzip2 stream: block CRC mismatch");
      stream_crc = ((stream_crc << 1) | (stream_crc >> 31)) ^ w.h_crc[q];
    }
    want.clear();
  };
  for (;;) {
    if (stream_done) {
      // another stream may follow, from the next byte boundary
      const int64_t nb = (expect + 7) / 8;
      if (nb + 14 > (int64_t)n) break;
      uint8_t h[4];
      BZ_CUDA(cudaMemcpyAsync(h, bytes + nb, 4, cudaMemcpyDeviceToHost, st));
      BZ_CUDA(cudaStreamSynchronize(st));
      if (!is_header(h)) break;
      expect = nb * 8 + 32;
      stream_crc = 0;
      stream_done = false;
    }
    // the end-of-stream marker at `expect`?
    if (std::binary_search(eoss.begin(), eoss.end(), expect)) {
      settle();
      // combined CRC after the 48-bit marker
      const int64_t p = expect + 48;
      uint8_t tail[8] = {0};
      const int64_t b0 = p / 8;
      const size_t nb = (size_t)std::min<int64_t>(8, (int64_t)n - b0);
      BZ_CUDA(cudaMemcpyAsync(tail, bytes + b0, nb, cudaMemcpyDeviceToHost, st));
      BZ_CUDA(cudaStreamSynchronize(st));
      uint64_t win = 0;
      for (int q = 0; q < 8; q++) win = (win << 8) | tail[q];
      const uint32_t got = (uint32_t)((win << (p % 8)) >> 32);
      BZ_REQUIRE(got == stream_crc, kErrArg, "bzip2 stream CRC mismatch");
      expect = p + 32;
      stream_done = true;
      continue;
    }
    // next candidates from `expect` on
    while (ci < cands.size() && cands[ci] < expect) ci++;
    BZ_REQUIRE(ci < cands.size() && cands[ci] == expect, kErrArg,
               "bzip2 stream: no block or end-of-stream marker where one must start");
    const int nc = (int)std::min<size_t>(batch, cands.size() - ci);
    BZ_CUDA(cudaMemcpyAsync(w.cand.p, cands.data() + ci, 8 * nc, cudaMemcpyHostToDevice, st));
    // A launch lasts as long as its slowest blocks: start the largest ones
    // first.
    std::vector<int64_t> bits(nc);  // to the next block or end-of-stream magic
    auto eos = std::upper_bound(eoss.begin(), eoss.end(), cands[ci]);
    for (int q = 0; q < nc; q++) {
      const size_t k = ci + (size_t)q;
      while (eos != eoss.end() && *eos < cands[k]) ++eos;
      bits[q] = std::min(k + 1 < cands.size() ? cands[k + 1] : nbits,
                         eos != eoss.end() ? *eos : nbits) -
                cands[k];
    }
    order.resize(nc);
    for (int q = 0; q < nc; q++) order[q] = q;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return bits[a] > bits[b]; });
    BZ_CUDA(cudaMemcpyAsync(w.order.p, order.data(), 4 * nc, cudaMemcpyHostToDevice, st));
    const uint32_t *wd = w.words.get<uint32_t>();
    const int64_t *dcand = w.cand.get<int64_t>();
    DecTab *dtab = w.tab.get<DecTab>();
    const dim3 cgrid(chunk_grid(bits[order[0]]), nc);
    k_dec_head<<<nc, kHeadThreads, 0, st>>>(wd, nwords, dcand, dtab, w.sel.get<uint8_t>());
    BZ_LAUNCH_CHECK();
    // group starts by jumps where that is the shorter way; k_dec_groups walks the
    // blocks that have none yet
    const std::vector<int32_t> jt0 = jump_tiles(bits);
    const int64_t room = std::max<int64_t>(w.jumps.cap, freeb / 4) / kJumpTileBytes;
    const std::vector<int> pieces = jump_pieces(jt0, std::min<int64_t>(room, kJumpMaxTiles));
    int64_t most = 0;
    for (size_t k = 0; k + 1 < pieces.size(); k++)
      most = std::max<int64_t>(most, jt0[pieces[k + 1]] - jt0[pieces[k]]);
    if (!pieces.empty() &&
        (starts == Starts::kJumps ||
         (starts == Starts::kByRule && jumps_pay(jt0, (int)pieces.size() - 1))) &&
        w.jt0.try_reserve(4 * (size_t)(nc + 1)) && w.lutlen.try_reserve((size_t)nc * kLensBytes) &&
        w.jumps.try_reserve((size_t)(most * kJumpTileBytes))) {
      BZ_CUDA(cudaMemcpyAsync(w.jt0.p, jt0.data(), 4 * (size_t)(nc + 1), cudaMemcpyHostToDevice, st));
      uint8_t *dlens = w.lutlen.get<uint8_t>();
      k_dec_lens<<<dim3(kDecMaxGroups, nc), 256, 0, st>>>(dtab, dlens);
      BZ_LAUNCH_CHECK();
      for (size_t k = 0; k + 1 < pieces.size(); k++) {
        const int q = pieces[k], nq = pieces[k + 1] - q;
        const int32_t *djt0 = w.jt0.get<int32_t>() + q;
        k_dec_jumps<<<jt0[q + nq] - jt0[q], 256, kJumpSmem, st>>>(
            wd, nwords, dcand + q, dtab + q, dlens + (size_t)q * kLensBytes, djt0, nq,
            w.jumps.get<uint16_t>());
        BZ_LAUNCH_CHECK();
        k_dec_starts<<<nq, 256, kStartsSmem, st>>>(
            dtab + q, w.sel.get<uint8_t>() + (size_t)q * kDecMaxSel,
            w.gstart.get<uint32_t>() + (size_t)q * kDecMaxSel, dcand + q, djt0,
            w.jumps.get<uint16_t>());
        BZ_LAUNCH_CHECK();
      }
    }
    int gthreads = 0;
    const GroupsKernel groups = groups_kernel(nc, w.sms, starts, &gthreads);
    groups<<<nc, gthreads, 0, st>>>(wd, nwords, dcand, dtab, w.sel.get<uint8_t>(),
                                    w.gstart.get<uint32_t>(), w.order.get<int32_t>());
    BZ_LAUNCH_CHECK();
    k_dec_syms<<<cgrid, 32 * kSymWarps, 0, st>>>(wd, nwords, dcand, dtab, w.sel.get<uint8_t>(),
                                                 w.gstart.get<uint32_t>(), w.tt.get<uint32_t>(),
                                                 cap);
    BZ_LAUNCH_CHECK();
    k_dec_mscan<<<nc, 256, 0, st>>>(dcand, dtab, w.tt.get<uint32_t>(), cap, w.db.get<DecBlock>());
    BZ_LAUNCH_CHECK();
    k_dec_emit<<<cgrid, 32 * kSymWarps, 0, st>>>(w.db.get<DecBlock>(), w.tt.get<uint32_t>(), L,
                                                 cap);
    BZ_LAUNCH_CHECK();
    BZ_CUDA(cudaMemcpyAsync(hdb.data(), w.db.p, sizeof(DecBlock) * nc, cudaMemcpyDeviceToHost,
                            st));
    BZ_CUDA(cudaStreamSynchronize(st));
    settle();
    // accept the chain within this batch
    std::vector<int32_t> acc;
    size_t used = 0;
    for (int q = 0; q < nc; q++) {
      if (hdb[q].start != expect) continue;
      BZ_REQUIRE(hdb[q].status == kDecOk, kErrArg,
                 "bzip2 stream: corrupt block (status " + std::to_string(hdb[q].status) + ")");
      acc.push_back(q);
      expect = hdb[q].end;
      used = q + 1;
      if (std::binary_search(eoss.begin(), eoss.end(), expect)) break;
    }
    ci += std::max<size_t>(used, 1);
    const int na = (int)acc.size();
    if (na == 0) continue;
    const int32_t *didx = w.idx.get<int32_t>();
    const DecBlock *ddb = w.db.get<DecBlock>();
    BZ_CUDA(cudaMemcpyAsync(w.idx.p, acc.data(), 4 * na, cudaMemcpyHostToDevice, st));
    int max_m = 0;
    for (const int q : acc) max_m = std::max(max_m, hdb[q].m);
    const ColumnGrids grids = column_grids(max_m);
    const dim3 lgrid(grids.lf, na);
    k_dec_lf_hist<<<lgrid, 256, 0, st>>>(didx, ddb, L, w.hist.get<int32_t>(), cap);
    BZ_LAUNCH_CHECK();
    WalkCtl *dctl = w.ctl.get<WalkCtl>();
    k_dec_lf_scan<<<na, 256, 0, st>>>(didx, ddb, w.hist.get<int32_t>(), dctl);
    BZ_LAUNCH_CHECK();
    k_dec_lf_rank<<<lgrid, 256, 0, st>>>(didx, ddb, L, w.hist.get<int32_t>(),
                                         w.tt.get<uint32_t>(), cap);
    BZ_LAUNCH_CHECK();
    k_dec_walk<<<dim3(grids.walk, na), kWalkThreads, 0, st>>>(
        didx, ddb, w.tt.get<uint32_t>(), dctl, w.pool.get<uint8_t>(), cap);
    BZ_LAUNCH_CHECK();
    BZ_CUDA(cudaMemsetAsync(w.bad.p, 0, 4, st));
    k_dec_chain<<<na, kChainThreads, kChainSmem, st>>>(didx, ddb, dctl, w.bad.get<int>());
    BZ_LAUNCH_CHECK();
    k_dec_gather<<<dim3(grids.gather, na), 256, 0, st>>>(
        didx, ddb, dctl, w.pool.get<uint8_t>(), L, cap);
    BZ_LAUNCH_CHECK();
    k_dec_repeat<<<dim3(grids.repeat, na), 256, 0, st>>>(didx, ddb, w.ctl.get<WalkCtl>(), L, cap);
    BZ_LAUNCH_CHECK();
    const dim3 ugrid(grids.unrle, na);
    k_dec_unrle1_count<<<ugrid, 256, 0, st>>>(didx, ddb, L, cap, w.maps.get<RunMap>());
    BZ_LAUNCH_CHECK();
    k_dec_unrle1_scan<<<na, 256, 0, st>>>(didx, ddb, w.maps.get<RunMap>(), w.lens.get<int64_t>());
    BZ_LAUNCH_CHECK();
    std::vector<int64_t> lens(na), offs(na);
    int hbad = 0;
    BZ_CUDA(cudaMemcpyAsync(lens.data(), w.lens.p, 8 * na, cudaMemcpyDeviceToHost, st));
    BZ_CUDA(cudaMemcpyAsync(&hbad, w.bad.p, 4, cudaMemcpyDeviceToHost, st));
    BZ_CUDA(cudaStreamSynchronize(st));
    BZ_REQUIRE(hbad == 0, kErrArg, "bzip2 stream: inconsistent block (BWT chain)");
    int64_t tot = 0;
    for (int q = 0; q < na; q++) {
      offs[q] = tot;
      tot += lens[q];
    }
    const int slot = nbatch++ & 1;
    if (w.used[slot]) {
      if ((size_t)tot + 16 > w.out[slot].cap) BZ_CUDA(cudaEventSynchronize(w.copied[slot]));
      BZ_CUDA(cudaStreamWaitEvent(st, w.copied[slot], 0));
    }
    w.reserve(w.out[slot], (size_t)tot + 16);
    BZ_CUDA(cudaMemcpyAsync(w.off.p, offs.data(), 8 * na, cudaMemcpyHostToDevice, st));
    k_dec_unrle1_write<<<ugrid, 256, 0, st>>>(didx, ddb, L, cap, w.maps.get<RunMap>(),
                                              w.off.get<int64_t>(), w.out[slot].get<uint8_t>());
    BZ_LAUNCH_CHECK();
    BZ_CUDA(cudaMemsetAsync(w.crc.p, 0xFF, 4 * na, st));
    k_dec_crc<<<dim3(crc_grid(*std::max_element(lens.begin(), lens.end())), na), 256, 0, st>>>(w.lens.get<int64_t>(), w.off.get<int64_t>(),
                                                   w.out[slot].get<uint8_t>(),
                                                   w.crc.get<uint32_t>());
    BZ_LAUNCH_CHECK();
    BZ_CUDA(cudaMemcpyAsync(w.h_crc, w.crc.p, 4 * na, cudaMemcpyDeviceToHost, st));
    BZ_CUDA(cudaEventRecord(w.written[slot], st));
    BZ_CUDA(cudaStreamWaitEvent(cs, w.written[slot], 0));
    sink.put(w.out[slot].get<uint8_t>(), (size_t)tot, cs);
    BZ_CUDA(cudaEventRecord(w.copied[slot], cs));
    w.used[slot] = true;
    want.resize(na);
    for (int q = 0; q < na; q++) want[q] = hdb[acc[q]].crc;
  }
  settle();
  BZ_REQUIRE(stream_done, kErrArg, "bzip2 stream: no end-of-stream marker");
  BZ_CUDA(cudaStreamSynchronize(cs));
}

// Stages the stream (host or device memory) in the workspace and decodes it.
void decode_into_sink(const uint8_t *in, size_t n, DecSink &sink) {
  BZ_REQUIRE(n >= 14, kErrArg, "not a bzip2 stream (shorter than 14 bytes)");
  DecWork &w = dec_work();
  std::lock_guard<std::mutex> g(w.mu);
  w.init();
  const size_t nwords = (n + 3) / 4 + 2;
  w.reserve(w.words, nwords * 4);
  const size_t body = n / 4 * 4;
  BZ_CUDA(cudaMemsetAsync(w.words.get<uint8_t>() + body, 0, nwords * 4 - body, w.st));
  BZ_CUDA(cudaMemcpyAsync(w.words.p, in, n, cudaMemcpyDefault, w.st));
  decode_words(w, n, sink);
}

template <typename F>
int guarded(F f) {
  try {
    f();
    set_last_error("");
    return BZ2G_OK;
  } catch (const Error &e) {
    set_last_error(e.what());
    return e.code;
  } catch (const std::exception &e) {
    set_last_error(e.what());
    return BZ2G_ERR_INTERNAL;
  }
}

int decompress_malloc(const uint8_t *in, size_t n, uint8_t **out, size_t *out_len) {
  return guarded([&] {
    BZ_REQUIRE(out && out_len && (n == 0 || in), kErrArg, "bad arguments");
    MallocSink sink;
    decode_into_sink(in, n, sink);
    *out_len = sink.size;
    *out = sink.release();
  });
}

int decompress_buffer(const uint8_t *in, size_t n, uint8_t *out, size_t cap,
                      size_t *out_len) {
  return guarded([&] {
    BZ_REQUIRE(out_len && (n == 0 || in) && (cap == 0 || out), kErrArg, "bad arguments");
    BufferSink sink(out, cap);
    decode_into_sink(in, n, sink);
    *out_len = sink.size;
  });
}

}  // namespace
}  // namespace bz2g

using namespace bz2g;

extern "C" int bz2g_decompress(const uint8_t *in, size_t n, uint8_t **out, size_t *out_len) {
  return decompress_malloc(in, n, out, out_len);
}

extern "C" int bz2g_decompress_device(const uint8_t *d_in, size_t n, uint8_t **out,
                                      size_t *out_len) {
  return decompress_malloc(d_in, n, out, out_len);
}

extern "C" int bz2g_decompress_into(const uint8_t *in, size_t n, uint8_t *out, size_t cap,
                                    size_t *out_len) {
  return decompress_buffer(in, n, out, cap, out_len);
}

extern "C" int bz2g_decompress_device_into(const uint8_t *d_in, size_t n, uint8_t *d_out,
                                           size_t cap, size_t *out_len) {
  return decompress_buffer(d_in, n, d_out, cap, out_len);
}
