// RLE1 (runs cut at C = 259, or 255 for bzip2 1.0.8's format) and the block
// CRC-32, over every block of a slab.
//
// Reference: src/compression/rle1.cu:13-113 (RLE1), src/compression/crc32.cpp
// (CRC).  A maximal run of length L is emitted as floor(L/C) chunks
// "cccc (C-4)" followed by the remainder r = L mod C: r < 4 copies of c, or
// "cccc (r-4)".  Position j of a run (j = i - run_start) emits
//   1 byte (c)            if j mod C < 3,
//   2 bytes (c, len-4)    if j mod C == 3,  len = length of its C-chunk,
//   nothing               otherwise,
// so every output offset is an exclusive scan of a per-position count, and the
// run start / end of a position are a max-scan / min-scan of run-start flags.
//
// CRC: crc0(D) (zero init, no final complement) is linear over GF(2).  Per
// 4096-byte tile, thread l takes 16 bytes and multiplies their crc0 by
// x^(8*16*(255-l)) mod P (a compile-time table), and the XOR of the 256
// products is the tile's crc0; the per-block kernel shifts each tile's crc0
// by x^(8 * bytes after the tile) (one thread per tile) and XORs them; the
// init term ~0 * x^(8n) is added at the end.
#include "crc.cuh"
#include "engine.h"

namespace bz2g {

namespace {


// A thread's 16 bytes of a raw tile (positions p0 .. p0 + 15 of the tile, p0 =
// 16 * thread): the bytes as words, the mask of run starts among them (bit k:
// byte k lies in the tile and differs from the byte before it; a block's first
// byte is one), and how many lie in the tile.
struct RawBytes {
  uint32_t w[4];
  uint32_t starts;
  int p0, nv;
  int b, st, n, len;  // block, tile start in the block, block and tile length
  const uint8_t *base;
};

__device__ __forceinline__ RawBytes raw_bytes(const SlabDev &d, int t) {
  RawBytes r;
  r.b = d.rt_block[t];
  r.st = d.rt_start[t];
  r.n = d.raw_len[r.b];
  r.len = min(kRawTile, r.n - r.st);
  r.base = d.raw + d.raw_off[r.b] + r.st;
  r.p0 = threadIdx.x * kTileItems;
  r.nv = min(kTileItems, max(0, r.len - r.p0));
  uint4 v = make_uint4(0, 0, 0, 0);
  if (r.nv > 0) v = reinterpret_cast<const uint4 *>(r.base)[threadIdx.x];
  r.w[0] = v.x;
  r.w[1] = v.y;
  r.w[2] = v.z;
  r.w[3] = v.w;
  // the byte before: the neighbour lane's last, or for lane 0 from memory
  uint32_t prev = __shfl_up_sync(0xffffffffu, v.w, 1);
  if (lane_id() == 0 && r.nv > 0 && r.st + r.p0 > 0) prev = (uint32_t)r.base[r.p0 - 1] << 24;
  r.starts = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    // bytes that differ from the one before: the top bit of each such byte,
    // the four bits gathered by one multiplication
    const uint32_t x = r.w[i] ^ __funnelshift_l(prev, r.w[i], 8);
    const uint32_t t8 = (((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u;
    r.starts |= ((t8 * 0x00204081u) >> 28) << (4 * i);
    prev = r.w[i];
  }
  if (r.st + r.p0 == 0) r.starts |= 1u;
  r.starts &= (1u << r.nv) - 1u;
  return r;
}

// A thread's position in the run chunk of the cut (259 or 255).
__device__ __forceinline__ int mod_cut(int x, int cut) {
  return cut == 259 ? (int)((uint32_t)x % 259u) : (int)((uint32_t)x % (uint32_t)255);
}

// Last run start in the warp before this lane (-1: none) and, in *warp_last,
// of the whole warp, from the lanes' own last starts ls (-1: none).
__device__ __forceinline__ int start_before(int ls, unsigned have, int *warp_last) {
  const unsigned below = have & ((1u << lane_id()) - 1u);
  const int v = __shfl_sync(0xffffffffu, ls, below ? 31 - __clz(below) : 0);
  *warp_last = have ? __shfl_sync(0xffffffffu, ls, 31 - __clz(have)) : -1;
  return below ? v : -1;
}

// Output bytes of the positions [0, n) of a run (the per-position counts
// summed: 5 per chunk of `cut`, and 1, 1, 1, 2 for its first four).
__device__ __forceinline__ int rle1_out_upto(int n, int cut) {
  const int f = n / cut, r = n - f * cut;
  return 5 * f + (r < 4 ? r : 5);
}

// Which of a thread's 16 bytes (bit k: byte k) emit output: positions 0..3
// of a run chunk emit their byte (e), position 3 also a length byte (e3).
// sm: the run starts among the bytes; nv: bytes in the tile.  With carry,
// byte 0 continues a run at position q0 of its chunk; the chunk starts are
// then the run starts, the carried chunk's start (byte -q0) and, while the
// carried run lasts, its next chunk start (byte cut - q0; a run beginning
// among these bytes reaches no chunk end within them, as cut > 16).
// Without carry the bytes before the first run start emit nothing here.
// A byte emits when a chunk starts within the 4 bytes up to it; it emits a
// length too when that start is exactly 3 before it.
__device__ __forceinline__ void rle1_emit_masks(uint32_t sm, int q0, int nv, int cut, bool carry,
                                                uint32_t *e, uint32_t *e3) {
  uint32_t s4 = sm << 4;  // bit k + 4: byte k
  if (carry) {
    if (q0 <= 3) {
      s4 |= 1u << (4 - q0);
    } else {
      const int pw = cut - q0;
      if (pw < kTileItems && (sm & ((1u << pw) - 1u)) == 0) s4 |= 1u << (pw + 4);
    }
  }
  const uint32_t nvm = (1u << nv) - 1u;
  uint32_t em = ((s4 | (s4 << 1) | (s4 << 2) | (s4 << 3)) >> 4) & nvm;
  uint32_t em3 = (((s4 << 3) & ~(s4 << 2) & ~(s4 << 1) & ~s4) >> 4) & nvm;
  if (!carry) {
    const uint32_t keep = sm ? ~((sm & (0u - sm)) - 1u) : 0u;
    em &= keep;
    em3 &= keep;
  }
  *e = em;
  *e3 = em3;
}

// Per raw tile: its first and last run start, its crc0, and its RLE1 output
// bytes from its first run start on (the bytes before it continue a run from
// an earlier tile; the per-block kernel adds their count in closed form).
// Bound by instructions: neighbours come by shuffle, starts by word arithmetic
// and ballots, the CRC four bytes at a time.
__global__ void __launch_bounds__(256) k_rle1_scan_tiles(SlabDev d) {
  __shared__ __align__(16) uint32_t tbl[4][256];
  __shared__ uint32_t red4[16];
  __shared__ int wl[8], wf[8], wc[8];
  __shared__ uint32_t wcrc[8];
  const int t = blockIdx.x;
  const int w = warp_id(), ln = lane_id();
  crc_word_table_fill(tbl);
  red4_fill(red4);
  const RawBytes r = raw_bytes(d, t);
  const uint32_t sm = r.starts;
  const int pbase = r.st + r.p0;
  const int ls = sm ? pbase + 31 - __clz(sm) : -1;
  const int fs = sm ? pbase + __ffs(sm) - 1 : INT32_MAX;
  const unsigned have = __ballot_sync(0xffffffffu, sm != 0);
  int wlast;
  int before = start_before(ls, have, &wlast);
  const int wfirst = __shfl_sync(0xffffffffu, fs, have ? __ffs(have) - 1 : 0);
  if (ln == 0) {
    wl[w] = wlast;
    wf[w] = wfirst;
  }
  __syncthreads();
  if (before < 0)
    for (int q = 0; q < w; q++) before = max(before, wl[q]);
  // output bytes: each thread's bytes from the last run start before them in
  // this tile (positions in the run modulo the cut)
  const int cut = d.run_cut;
  uint32_t em, em3;
  rle1_emit_masks(sm, before >= 0 ? mod_cut(pbase - before, cut) : 0, r.nv, cut, before >= 0, &em,
                  &em3);
  const int cnt = __reduce_add_sync(0xffffffffu, __popc(em) + __popc(em3));
  // crc0 of the tile, right-aligned into a virtual 4096-byte tile (leading
  // zeros leave a zero-init CRC unchanged): 16 bytes per thread, each
  // thread's crc0 moved to the tile's end by one multiplication, then XOR.
  uint32_t c = 0;
  if (r.len == kRawTile) {
#pragma unroll
    for (int i = 0; i < 4; i++) c = crc_word(c, r.w[i], tbl);
  } else {
    const int pad = kRawTile - r.len;
    for (int v = max(r.p0, pad); v < r.p0 + kTileItems; v++) c = crc_byte(c, r.base[v - pad], tbl[0]);
  }
  c = __reduce_xor_sync(0xffffffffu, gf_mul_lane(c, threadIdx.x, red4));
  if (ln == 0) {
    wc[w] = cnt;
    wcrc[w] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int f = INT32_MAX, l = -1, total = 0;
    uint32_t x = 0;
    for (int q = 0; q < 8; q++) {
      f = min(f, wf[q]);
      l = max(l, wl[q]);
      total += wc[q];
      x ^= wcrc[q];
    }
    d.tile_a[t] = f;  // first run start in tile
    d.tile_b[t] = l;  // last run start in tile
    d.tile_c[t] = total;
    d.tile_d[t] = (int32_t)x;  // the tile's crc0 (shifted per block)
  }
}

// Per block: exclusive max of last-starts (run start carried into a tile) and
// exclusive min of first-starts (next run start after a tile), and the CRC.
__global__ void __launch_bounds__(256) k_rle1_block_carry(SlabDev d, const int *rt_first) {
  __shared__ int scratch[40];
  __shared__ int sx[256];
  const int b = blockIdx.x;
  const int t0 = rt_first[b], nt = rt_first[b + 1] - t0;
  const int n = d.raw_len[b];
  int carry = -1, out_carry = 0;
  const int cut = d.run_cut;
  for (int base = 0; base < nt; base += 256) {
    int k = base + threadIdx.x;
    int v = k < nt ? d.tile_b[t0 + k] : -1;
    int inc = block_incl_max(v, scratch, -1);
    sx[threadIdx.x] = inc;
    __syncthreads();
    int ex = threadIdx.x == 0 ? carry : max(carry, sx[threadIdx.x - 1]);
    int cnt = 0;
    if (k < nt) {
      d.tile_b[t0 + k] = ex;
      // the tile's output: its own count plus that of its bytes before its
      // first run start, positions j0 .. j0 + pre - 1 of the run begun at ex
      const int st = d.rt_start[t0 + k];
      const int len = min(kRawTile, n - st);
      const int fs = d.tile_a[t0 + k];
      const int pre = (fs == INT32_MAX ? st + len : fs) - st;
      const int j0 = st - ex;
      cnt = d.tile_c[t0 + k] + (pre > 0 ? rle1_out_upto(j0 + pre, cut) - rle1_out_upto(j0, cut) : 0);
    }
    int c2 = max(carry, sx[255]);
    __syncthreads();
    carry = c2;
    int tot;
    const int o = block_excl_sum(cnt, scratch, &tot);
    if (k < nt) d.tile_c[t0 + k] = out_carry + o;
    out_carry += tot;
  }
  if (threadIdx.x == 0) d.m[b] = out_carry;
  int carry_min = n;
  // walk backwards for the suffix minimum
  for (int base = ((nt - 1) / 256) * 256; base >= 0; base -= 256) {
    int k = base + threadIdx.x;
    int v = k < nt ? d.tile_a[t0 + k] : INT32_MAX;
    int inc = block_suffix_min(v, scratch, INT32_MAX);
    sx[threadIdx.x] = inc;
    __syncthreads();
    int ex = threadIdx.x == 255 ? carry_min : min(carry_min, sx[threadIdx.x + 1]);
    if (k < nt) d.tile_a[t0 + k] = ex;
    int c2 = min(carry_min, sx[0]);
    __syncthreads();
    carry_min = c2;
  }
  // block CRC: each tile's crc0 shifted by x^(8 * bytes after it), XOR-ed
  uint32_t acc = 0;
  for (int k = threadIdx.x; k < nt; k += blockDim.x) {
    const int st = d.rt_start[t0 + k];
    const int len = min(kRawTile, n - st);
    const uint32_t c = (uint32_t)d.tile_d[t0 + k];
    if (c) acc ^= gf_mul(c, xpow8((uint64_t)(n - (st + len))));
  }
  for (int o = 16; o > 0; o >>= 1) acc ^= __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane_id() == 0) scratch[warp_id()] = (int)acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t a = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) a ^= (uint32_t)scratch[w];
    d.crc[b] = ~(gf_mul(0xFFFFFFFFu, xpow8((uint64_t)n)) ^ a);
  }
}

// Bound by instructions like the scan: a byte of output costs a test, a byte
// store and an add, the copy out goes by words.
__global__ void __launch_bounds__(256) k_rle1_write(SlabDev d) {
  // the tile's output, at the alignment it has in the block
  __shared__ __align__(16) uint8_t so[kRawTile + kRawTile / 4 + 16];
  __shared__ int wl[8], wf[8], wc[8];
  const int t = blockIdx.x;
  const int w = warp_id(), ln = lane_id();
  const RawBytes r = raw_bytes(d, t);
  const uint32_t sm = r.starts;
  const int pbase = r.st + r.p0;  // block-local position of byte 0
  const int ls = sm ? pbase + 31 - __clz(sm) : -1;
  const int fs = sm ? pbase + __ffs(sm) - 1 : INT32_MAX;
  const unsigned have = __ballot_sync(0xffffffffu, sm != 0);
  int wlast;
  int before = start_before(ls, have, &wlast);
  // first start after this lane in the warp, and in the whole warp
  const unsigned above = have & ~((2u << ln) - 1u);
  int after = __shfl_sync(0xffffffffu, fs, above ? __ffs(above) - 1 : 0);
  if (!above) after = INT32_MAX;
  const int wfirst = __shfl_sync(0xffffffffu, fs, have ? __ffs(have) - 1 : 0);
  if (ln == 0) {
    wl[w] = wlast;
    wf[w] = wfirst;
  }
  __syncthreads();
  if (before < 0) {
    before = d.tile_b[t];  // the last start before the tile
    for (int q = 0; q < w; q++) before = max(before, wl[q]);
  }
  if (after == INT32_MAX) {
    after = d.tile_a[t];  // next start after the tile (or n)
    for (int q = w + 1; q < 8; q++) after = min(after, wf[q]);
  }
  // each byte's emits: its position in its chunk from the run start before
  // the thread (one division per thread), then bit masks
  const int cut = d.run_cut;
  uint32_t em = 0, em3 = 0;
  if (r.nv > 0)
    rle1_emit_masks(sm, before >= 0 ? mod_cut(pbase - before, cut) : 0, r.nv, cut, before >= 0, &em,
                    &em3);
  const int cnt = __popc(em) + __popc(em3);
  const int inc = warp_incl_sum(cnt);
  if (ln == 31) wc[w] = inc;
  __syncthreads();
  int o = inc - cnt, tot = 0;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int c = wc[q];
    if (q < w) o += c;
    tot += c;
  }
  uint8_t *dst = d.rle1 + d.off[r.b] + d.tile_c[t];
  const int lead = (int)(reinterpret_cast<uintptr_t>(dst) & 3u);
  if (__any_sync(0xffffffffu, em)) {
    uint8_t *out = so + lead + o;
#pragma unroll
    for (int k = 0; k < kTileItems; k++) {
      if ((em >> k) & 1u) {
        *out++ = (uint8_t)(r.w[k >> 2] >> (8 * (k & 3)));
        if ((em3 >> k) & 1u) {
          // the chunk's length: from its start (3 bytes back) to the run's end
          // or the cut, whichever comes first
          const uint32_t rest = k + 1 < kTileItems ? sm >> (k + 1) : 0u;
          const int run_end = rest ? pbase + k + __ffs(rest) : after;
          *out++ = (uint8_t)(min(cut, run_end - (pbase + k - 3)) - 4);
        }
      }
    }
  }
  __syncthreads();
  // the tile's output to its place in the block, by words where they are whole
  dst -= lead;
  const int end = lead + tot;
  for (int i = 4 * threadIdx.x; i < end; i += 4 * 256) {
    if (i >= lead && i + 4 <= end) {
      *reinterpret_cast<uint32_t *>(dst + i) = *reinterpret_cast<const uint32_t *>(so + i);
    } else {
      for (int q = max(i, lead); q < min(i + 4, end); q++) dst[q] = so[q];
    }
  }
}

}  // namespace

void stage_rle1_crc(const SlabDev &d, cudaStream_t st) {
  const int *rt_first = d.rt_first;
  if (d.n_raw_tiles > 0) {
    k_rle1_scan_tiles<<<d.n_raw_tiles, 256, 0, st>>>(d);
    BZ_LAUNCH_CHECK();
  }
  k_rle1_block_carry<<<d.nblocks, 256, 0, st>>>(d, rt_first);
  BZ_LAUNCH_CHECK();
  if (d.n_raw_tiles > 0) {
    k_rle1_write<<<d.n_raw_tiles, 256, 0, st>>>(d);
    BZ_LAUNCH_CHECK();
  }
}

void launch_crc_only(const SlabDev &d, cudaStream_t st) {
  const int *rt_first = d.rt_first;
  if (d.n_raw_tiles > 0) {
    k_rle1_scan_tiles<<<d.n_raw_tiles, 256, 0, st>>>(d);
    BZ_LAUNCH_CHECK();
  }
  k_rle1_block_carry<<<d.nblocks, 256, 0, st>>>(d, rt_first);
  BZ_LAUNCH_CHECK();
}

}  // namespace bz2g
