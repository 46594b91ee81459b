// RLE2: MTF values to bzip2 symbols, with the per-block symbol histogram.
//
// Reference: src/compression/rle2.cu:11-158 (and its oracle
// tests/compression/rle2.cu:9-33).  A value v > 0 becomes v + 1; a run of k
// zeros becomes the bijective base-2 digits of k, least significant first,
// RUNA (0) for digit 1 and RUNB (1) for digit 2 -- floor(log2(k+1)) symbols;
// EOB = nInUse + 1 ends the block.  Position q of a zero run emits digit q if
// q < floor(log2(k+1)), so output offsets are a scan of 0/1 counts and the
// run bounds are a max-scan / min-scan of non-zero positions.
#include "engine.h"

namespace bz2g {

namespace {

__device__ __forceinline__ int tile_len(const SlabDev &d, int t, int *b, int *lt, int64_t *off,
                                        int *m) {
  *b = d.tile_block[t];
  *off = d.off[*b];
  *lt = (int)((int64_t)t * kTile - *off);
  *m = d.m[*b];
  return min(kTile, *m - *lt);
}

__device__ __forceinline__ int n_digits(int k) { return 31 - __clz(k + 1); }

// A thread's 16 MTF values (one 16-byte load; the buffer has slack past a
// block's end): the mask of non-zero ones, how many lie in the tile, and the
// non-zeros nearest before and after them in the tile (block positions; -1 and
// INT32_MAX when there are none).
struct Values16 {
  uint32_t w[4];
  uint32_t nz;
  int nv, pos;  // pos: block position of value 0
  int before, after;
  int wlast, wfirst;  // the warp's last and first non-zero
};

__device__ __forceinline__ Values16 values16(const uint8_t *V, int lt, int valid) {
  Values16 v;
  const int p0 = threadIdx.x * kTileItems;
  v.nv = min(kTileItems, max(0, valid - p0));
  v.pos = lt + p0;
  uint4 x = make_uint4(0, 0, 0, 0);
  if (v.nv > 0) x = *reinterpret_cast<const uint4 *>(V + lt + p0);
  v.w[0] = x.x;
  v.w[1] = x.y;
  v.w[2] = x.z;
  v.w[3] = x.w;
  v.nz = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    // the top bit of each non-zero byte, gathered by one multiplication
    const uint32_t t8 = (((v.w[i] & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v.w[i]) & 0x80808080u;
    v.nz |= ((t8 * 0x00204081u) >> 28) << (4 * i);
  }
  v.nz &= (1u << v.nv) - 1u;
  return v;
}

// The non-zeros around each thread's values, within the tile (256 threads).
__device__ __forceinline__ void zero_bounds(Values16 &v, int *wl, int *wf) {
  const unsigned full = 0xffffffffu;
  const int ln = lane_id(), w = warp_id();
  const int ls = v.nz ? v.pos + 31 - __clz(v.nz) : -1;
  const int fs = v.nz ? v.pos + __ffs(v.nz) - 1 : INT32_MAX;
  const unsigned have = __ballot_sync(full, v.nz != 0);
  const unsigned below = have & ((1u << ln) - 1u), above = have & ~((2u << ln) - 1u);
  v.before = __shfl_sync(full, ls, below ? 31 - __clz(below) : 0);
  v.after = __shfl_sync(full, fs, above ? __ffs(above) - 1 : 0);
  if (!below) v.before = -1;
  if (!above) v.after = INT32_MAX;
  v.wlast = have ? __shfl_sync(full, ls, 31 - __clz(have)) : -1;
  v.wfirst = have ? __shfl_sync(full, fs, __ffs(have) - 1) : INT32_MAX;
  if (ln == 0) {
    wl[w] = v.wlast;
    wf[w] = v.wfirst;
  }
  __syncthreads();
  if (v.before < 0)
    for (int q = 0; q < w; q++) v.before = max(v.before, wl[q]);
  if (v.after == INT32_MAX)
    for (int q = w + 1; q < 8; q++) v.after = min(v.after, wf[q]);
}

// The run digits among a thread's values, zero run by zero run: which zeros
// emit one (bit mask), and the digits (bit mask).  A run of k zeros from zs on
// emits digit q at zs + q for q < n_digits(k); digit q is bit q of k + 1.
// kTileOnly: v's bounds are the tile's, and runs that may start before it
// (before < 0) or end after it (after INT32_MAX) are left out.
template <bool kTileOnly>
__device__ __forceinline__ void run_digits(const Values16 &v, uint32_t *emit, uint32_t *digits) {
  uint32_t z = ~v.nz & ((1u << v.nv) - 1u);
  uint32_t em = 0, dg = 0;
  while (z) {
    const int a = __ffs(z) - 1;
    const int n = __ffs(~(z >> a)) - 1;
    const uint32_t span = ((1u << n) - 1u) << a;
    z &= ~span;
    const int end = a + n >= v.nv ? v.after : v.pos + a + n;
    if (kTileOnly && ((a == 0 && v.before < 0) || end == INT32_MAX)) continue;
    const int q = a == 0 ? v.pos - v.before - 1 : 0;  // the run's zeros before position a
    const int k = end - (v.pos + a - q);
    const int c = min(n_digits(k) - q, n);
    if (c > 0) {
      const uint32_t m = (1u << c) - 1u;
      em |= m << a;
      dg |= (((uint32_t)(k + 1) >> q) & m) << a;
    }
  }
  *emit = em;
  *digits = dg;
}

// Per tile: first and last non-zero (tile_a, tile_b, and the first again in
// tile_d), and the output symbols of its non-zeros and of the zero runs
// between two of its non-zeros (tile_c); the zero runs at its ends are
// counted by the per-block kernel, which knows where they start and end.
__global__ void __launch_bounds__(256) k_rle2_scan_tiles(SlabDev d, const int32_t *list) {
  const int t = list ? list[blockIdx.x] : (int)blockIdx.x;
  __shared__ int wl[8], wf[8], wc[8];
  int b, lt, m;
  int64_t off;
  int valid = tile_len(d, t, &b, &lt, &off, &m);
  if (valid <= 0) return;
  Values16 v = values16(d.mtf + off, lt, valid);
  zero_bounds(v, wl, wf);
  uint32_t em, dg;
  run_digits<true>(v, &em, &dg);
  const int cnt = __reduce_add_sync(0xffffffffu, __popc(v.nz) + __popc(em));
  if (lane_id() == 0) wc[warp_id()] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    int f = INT32_MAX, l = -1, tot = 0;
    for (int w = 0; w < 8; w++) {
      f = min(f, wf[w]);
      l = max(l, wl[w]);
      tot += wc[w];
    }
    d.tile_a[t] = f;
    d.tile_b[t] = l;
    d.tile_d[t] = f;
    d.tile_c[t] = tot;
  }
}

// Per block: previous non-zero before each tile (tile_b) and next non-zero
// after each tile (tile_a, m if none); tile output offsets (tile_c), the
// symbol count s with the EOB written and counted.
__global__ void __launch_bounds__(256) k_rle2_block_carry(SlabDev d) {
  __shared__ int scratch[40];
  __shared__ int sx[256];
  const int b = blockIdx.x;
  const int m = d.m[b];
  if (m <= 0) {
    if (threadIdx.x == 0) {
      const int eob = d.n_in_use[b] + 1;
      d.rle2[d.off[b]] = (uint16_t)eob;
      d.s[b] = 1;
      atomicAdd(&d.freq[b * kMaxAlpha + eob], 1);
    }
    return;
  }
  const int nt = (m + kTile - 1) / kTile;
  const int t0 = (int)(d.off[b] / kTile);
  int carry = -1;
  for (int base = 0; base < nt; base += 256) {
    int k = base + threadIdx.x;
    int v = k < nt ? d.tile_b[t0 + k] : -1;
    int inc = block_incl_max(v, scratch, -1);
    sx[threadIdx.x] = inc;
    __syncthreads();
    int ex = threadIdx.x == 0 ? carry : max(carry, sx[threadIdx.x - 1]);
    if (k < nt) d.tile_b[t0 + k] = ex;
    int c2 = max(carry, sx[255]);
    __syncthreads();
    carry = c2;
  }
  int carry_min = m;
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
  // Each tile's output: its own count plus the digits of the zero runs at
  // its ends that fall inside it (a zero run of length n starting at zs
  // emits its digits at positions zs .. zs + n_digits(n) - 1), then the
  // tile offsets, the block's symbol count and its EOB.
  int out_carry = 0;
  for (int base = 0; base < nt; base += 256) {
    const int k = base + threadIdx.x;
    int cnt = 0;
    if (k < nt) {
      const int t = t0 + k;
      const int lt = k * kTile;
      const int te = min(lt + kTile, m);
      const int first = d.tile_d[t];  // first non-zero in the tile
      const int prev = d.tile_b[t];   // last non-zero before the tile
      const int next = d.tile_a[t];   // first non-zero after the tile, or m
      auto digits_in = [](int zs, int end, int a, int b) {  // of run [zs, end), at [a, b)
        if (end <= zs || b <= a) return 0;
        const int nd = n_digits(end - zs);
        return min(b - zs, nd) - min(a - zs, nd);
      };
      cnt = d.tile_c[t];
      if (first == INT32_MAX) {
        cnt += digits_in(prev + 1, next, lt, te);
      } else {
        cnt += digits_in(prev + 1, first, lt, first);
        // the last non-zero of this tile is the last one before the next
        const int last = k + 1 < nt ? d.tile_b[t + 1] : carry;
        cnt += digits_in(last + 1, next, last + 1, te);
      }
    }
    int tot;
    const int o = block_excl_sum(cnt, scratch, &tot);
    if (k < nt) d.tile_c[t0 + k] = out_carry + o;
    out_carry += tot;
  }
  if (threadIdx.x == 0) {
    const int eob = d.n_in_use[b] + 1;
    d.rle2[d.off[b] + out_carry] = (uint16_t)eob;
    d.s[b] = out_carry + 1;
    atomicAdd(&d.freq[b * kMaxAlpha + eob], 1);
  }
}

// The tile's symbols are assembled in shared memory, at the alignment they have
// in the block, and copied out by words.
__global__ void __launch_bounds__(256) k_rle2_write(SlabDev d, const int32_t *list) {
  const int t = list ? list[blockIdx.x] : (int)blockIdx.x;
  __shared__ int wl[8], wf[8], wc[8];
  __shared__ int hist[kMaxAlpha];
  __shared__ __align__(16) uint16_t so[kTile + 8];
  int b, lt, m;
  int64_t off;
  int valid = tile_len(d, t, &b, &lt, &off, &m);
  if (valid <= 0) return;
  for (int i = threadIdx.x; i < kMaxAlpha; i += blockDim.x) hist[i] = 0;
  Values16 v = values16(d.mtf + off, lt, valid);
  zero_bounds(v, wl, wf);
  v.before = max(v.before, d.tile_b[t]);
  v.after = min(v.after, d.tile_a[t]);
  uint32_t em, dg;
  run_digits<false>(v, &em, &dg);
  const int cnt = __popc(v.nz) + __popc(em);
  const int inc = warp_incl_sum(cnt);
  if (lane_id() == 31) wc[warp_id()] = inc;
  __syncthreads();
  int o = inc - cnt, tot = 0;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int c = wc[q];
    if (q < (int)warp_id()) o += c;
    tot += c;
  }
  const int64_t at = off + d.tile_c[t];
  const int lead = (int)(at & 1);
  uint16_t *out = so + lead + o;
  // the frequent symbols are counted in registers (RUNA and RUNB by their
  // masks, symbols 2 .. 7 in byte fields), added to the tile's histogram once
  // per thread
  const int h1 = __popc(dg & em), h0 = __popc(em) - h1;
  uint64_t hot = 0;
  const uint32_t any = v.nz | em;
#pragma unroll
  for (int k = 0; k < kTileItems; k++) {
    if ((any >> k) & 1u) {
      const uint32_t x = (v.w[k >> 2] >> (8 * (k & 3))) & 0xffu;
      const uint32_t sym = x ? x + 1 : (dg >> k) & 1u;
      *out++ = (uint16_t)sym;
      if (sym < 8) hot += 1ull << (8 * sym);
      else atomicAdd(&hist[sym], 1);
    }
  }
  if (h0) atomicAdd(&hist[0], h0);
  if (h1) atomicAdd(&hist[1], h1);
#pragma unroll
  for (int q = 2; q < 8; q++) {
    const int c = (int)((hot >> (8 * q)) & 0xffu);
    if (c) atomicAdd(&hist[q], c);
  }
  __syncthreads();
  uint32_t *dst = reinterpret_cast<uint32_t *>(d.rle2 + at - lead);
  const int end = lead + tot;
  for (int i = threadIdx.x; 2 * i < end; i += 256) {
    if (2 * i >= lead && 2 * i + 2 <= end) {
      dst[i] = reinterpret_cast<const uint32_t *>(so)[i];
    } else {
      for (int q = max(2 * i, lead); q < min(2 * i + 2, end); q++) d.rle2[at - lead + q] = so[q];
    }
  }
  for (int i = threadIdx.x; i < kMaxAlpha; i += blockDim.x)
    if (hist[i]) atomicAdd(&d.freq[b * kMaxAlpha + i], hist[i]);
}

}  // namespace

void stage_rle2(const SlabDev &d, cudaStream_t st) {
  BZ_CUDA(cudaMemsetAsync(d.freq, 0, sizeof(int32_t) * kMaxAlpha * d.nblocks, st));
  const int nlive = live_tiles(d, st);
  const int grid = nlive >= 0 ? nlive : d.ntiles;
  const int32_t *list = nlive >= 0 ? d.vt_list : nullptr;
  if (grid > 0) {
    k_rle2_scan_tiles<<<grid, 256, 0, st>>>(d, list);
    BZ_LAUNCH_CHECK();
  }
  k_rle2_block_carry<<<d.nblocks, 256, 0, st>>>(d);
  BZ_LAUNCH_CHECK();
  if (grid > 0) {
    k_rle2_write<<<grid, 256, 0, st>>>(d, list);
    BZ_LAUNCH_CHECK();
  }
}

}  // namespace bz2g
