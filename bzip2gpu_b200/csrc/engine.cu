// Slab plan and workspace (device buffers of one slab context).
#include "engine.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <sstream>
#include <utility>

namespace bz2g {

static std::atomic<int64_t> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
int64_t launch_count() { return g_launches.load(); }

[[noreturn]] void throw_cuda(cudaError_t e, const char *expr, const char *file, int line) {
  std::ostringstream os;
  os << expr << " failed at " << file << ":" << line << ": " << cudaGetErrorName(e) << " ("
     << cudaGetErrorString(e) << ")";
  throw Error(kErrCuda, os.str());
}

static int64_t m_bound(int64_t raw_len, int64_t m_cap) {
  const int64_t b = rle1_bound(raw_len);
  return m_cap > 0 ? std::min(b, m_cap) : b;
}

static int64_t groups_bound(int64_t raw_len, int64_t m_cap = 0) {
  // symbols <= RLE1 bytes + 1 (EOB), 50 symbols per group
  return (m_bound(raw_len, m_cap) + 1 + kGroupSize - 1) / kGroupSize;
}

BlockNeeds block_needs(int64_t L, int64_t m_cap) {
  BlockNeeds r;
  r.raw = align_up(L, 16);
  r.raw_tiles = (int)((L + kRawTile - 1) / kRawTile);
  r.elems = align_up(std::max<int64_t>(m_bound(L, m_cap), 1), kTile);
  r.tiles = (int)(r.elems / kTile);
  r.group_tiles = (int)((groups_bound(L, m_cap) + kGroupTile - 1) / kGroupTile);
  return r;
}

void SlabPlan::build(const int *lens, int n, int cut, int64_t mcap) {
  nblocks = n;
  run_cut = cut;
  m_cap = mcap;
  raw_off.assign(n, 0);
  off.assign(n, 0);
  cap.assign(n, 0);
  raw_len.assign(lens, lens + n);
  rt_block.clear();
  rt_start.clear();
  rt_first.assign(n + 1, 0);
  tile_block.clear();
  gt_block.clear();
  gt_first.clear();
  gt_begin.assign(n + 1, 0);
  raw_total = 0;
  elem_total = 0;
  max_m_bound = 0;
  for (int b = 0; b < n; b++) {
    const int64_t L = lens[b];
    raw_off[b] = raw_total;
    raw_total += align_up(L, 16);
    rt_first[b] = (int)rt_block.size();
    for (int64_t st = 0; st < L; st += kRawTile) {
      rt_block.push_back(b);
      rt_start.push_back((int)st);
    }
    const int64_t c = align_up(std::max<int64_t>(m_bound(L, m_cap), 1), kTile);
    off[b] = elem_total;
    cap[b] = c;
    for (int64_t k = 0; k < c / kTile; k++) tile_block.push_back(b);
    elem_total += c;
    gt_begin[b] = (int)gt_block.size();
    const int64_t G = groups_bound(L, m_cap);
    for (int64_t g = 0; g < G; g += kGroupTile) {
      gt_block.push_back(b);
      gt_first.push_back((int)g);
    }
    max_m_bound = std::max<int>(max_m_bound, (int)m_bound(L, m_cap));
  }
  rt_first[n] = (int)rt_block.size();
  gt_begin[n] = (int)gt_block.size();
}

Workspace::Workspace(int mb, int64_t mr, int64_t me, int mt, int mrt, int mgt)
    : max_blocks(mb), max_raw(mr), max_elems(me), max_tiles(mt), max_raw_tiles(mrt),
      max_group_tiles(mgt) {
  std::memset(&dev, 0, sizeof(dev));
  // One allocation on the device and one page-locked one, shared out: the calls
  // for single stages make a workspace each, and one by one its 76 arrays cost
  // more than the stage (CRC of 20,000 bytes 1.0 ms, of 900,000 8.2; so 0.6, 0.7).
  size_t bytes = 0;
  std::vector<std::pair<void **, size_t>> parts;
  auto part = [&](auto *&p, size_t n) {
    parts.push_back({(void **)&p, bytes});
    bytes += (std::max<size_t>(n, 1) + 511) / 512 * 512;
  };
  try {
    const int64_t E = me + kTile;  // slack for vector loads past a block's end
    const int64_t B = mb + 1;
    const int64_t G = mt / kScanTiles + B;  // groups: t / kScanTiles + b of a block's tiles t
    // (these three are zeroed by the first upload_plan)
    part(dev.err, 64);
    part(dev.scan_count, G * 4);
    part(dev.blk_count, B * 4);
    to_zero_ = bytes;
    part(dev.raw, mr + 64);
    part(dev.rle1, E);
    part(dev.last, E);
    part(dev.mtf, E);
    part(dev.sa, E * 4);
    part(dev.isa, E * 4);
    part(dev.kpos[0], E * 4);
    part(dev.kpos[1], E * 4);
    part(dev.keys[0], E * 8);
    part(dev.keys[1], E * 8);
    part(dev.vals[0], E * 4);
    part(dev.vals[1], E * 4);
    part(dev.rle2, E * 2);
    part(dev.sel, E / 32 + 64);
    part(dev.sel_mtf, E / 32 + 64);
    part(dev.grp_bits, (E / 32 + 64) * 4);
    // payload: <= 17 bits per symbol; header: <= 6 bits per selector + tables
    out_words = E * kMaxCodeLen / 32 + (int64_t)mb * 8192 + 64;
    part(dev.out, out_words * 4);
    const int64_t T = std::max<int64_t>(mt, mrt) + 1;
    part(dev.tile_a, T * 4);
    part(dev.tile_b, T * 4);
    part(dev.tile_c, T * 4);
    part(dev.tile_d, T * 4);
    part(dev.tile_list, T * 4);
    part(dev.loc_list, 8 * T * 4);
    part(dev.vt_list, T * 4);
    part(dev.vg_list, ((int64_t)mgt + 1) * 4);
    part(dev.warp_last, ((int64_t)mt + 1) * (kTileThreads / 32) * 4);
    part(dev.warp_act, ((int64_t)mt + 1) * (kTileThreads / 32) * 4);
    part(dev.head_bits, ((int64_t)mt * (kTile / 32) + 1) * 4);
    part(dev.tile_hist, (int64_t)mt * kMaxRadix * 4);
    part(dev.tile_last, (int64_t)mt * 256 * 4);
    part(dev.gt_bits, ((int64_t)mgt + 1) * 4);
    part(dev.m, B * 4);
    part(dev.s, B * 4);
    part(dev.n_in_use, B * 4);
    part(dev.orig_ptr, B * 4);
    part(dev.n_groups, B * 4);
    part(dev.n_sel, B * 4);
    part(dev.crc, B * 4);
    part(dev.crc_acc, B * 4);
    part(dev.present, B * 8 * 4);
    part(dev.freq, B * kMaxAlpha * 4);
    part(dev.len, B * kMaxGroups * kMaxAlpha);
    part(dev.code, B * kMaxGroups * kMaxAlpha * 4);
    part(dev.len_code, B * kLenCode * 4);
    part(dev.rfreq, B * kMaxGroups * kMaxAlpha * 4);
    part(dev.learned, B * 4);
    part(dev.rfreq_m, B * kMaxGroups * kMaxAlpha * 4);
    part(dev.len2, B * kMaxGroups * kMaxAlpha);
    part(dev.sel2, E / 32 + 64);
    part(dev.rfreq2, B * kMaxGroups * kMaxAlpha * 4);
    part(dev.plain_left, B * 4);
    part(dev.sort_len, B * 4);
    part(dev.done, B * 4);
    part(dev.ngroups, B * 4);
    part(dev.act_len, B * 4);
    for (int32_t **a : {&dev.loc, &dev.loc_cur, &dev.loc_act, &dev.loc_heads, &dev.loc_sing,
                        &dev.gmax, &dev.loc_step})
      part(*a, B * 4);
    part(dev.active_sum, B * 8);
    part(dev.pstat, B * 8 * 4);
    part(dev.hdr_bits, B * 8);
    part(dev.pay_bits, B * 8);
    part(dev.blk_start, B * 8);
    part(dev.sort_ctl, 64);
    part(dev.scan_base, G * kMaxRadix * 4);
    part(dev.stream, 64);
    part(dev.kt_elems, 8 * kMaxTimedLaunches);
    // plan arrays: 3 int64 per block + ints
    pinned_plan_bytes = (size_t)B * 3 * 8 + ((size_t)B * 4 + mrt * 2 + mt + mgt * 2) * 4 + 1024;
    part(plan_dev_, pinned_plan_bytes);
    BZ_CUDA(cudaMalloc((void **)&device_, bytes));
    for (const auto &q : parts) *q.first = device_ + q.second;
    BZ_CUDA(cudaMallocHost((void **)&host_, 128 + pinned_plan_bytes));
    dev.h_flags = reinterpret_cast<int32_t *>(host_);
    dev.live = reinterpret_cast<int *>(host_ + 64);
    pinned_plan = host_ + 128;
    dev.live[0] = dev.live[1] = dev.live[2] = -1;
  } catch (...) {
    if (device_) cudaFree(device_);
    if (host_) cudaFreeHost(host_);
    throw;
  }
}

Workspace::~Workspace() {
  if (device_) cudaFree(device_);
  if (host_) cudaFreeHost(host_);
}

void Workspace::upload_plan(const SlabPlan &p, cudaStream_t st) {
  // on the stream whose work counts on it: a memset on the default stream may
  // still wait for the program's kernels there when that work runs
  if (to_zero_) BZ_CUDA(cudaMemsetAsync(device_, 0, to_zero_, st));
  to_zero_ = 0;
  dev.live[0] = dev.live[1] = dev.live[2] = -1;  // a new slab: its lists are built anew
  BZ_REQUIRE(p.nblocks <= max_blocks && p.raw_total <= max_raw && p.elem_total <= max_elems &&
                 (int)p.tile_block.size() <= max_tiles && (int)p.rt_block.size() <= max_raw_tiles &&
                 (int)p.gt_block.size() <= max_group_tiles,
             kErrInternal, "slab plan exceeds workspace");
  uint8_t *h = (uint8_t *)pinned_plan;
  uint8_t *dbase = (uint8_t *)plan_dev_;
  size_t pos = 0;
  auto put = [&](const void *src, size_t bytes) -> const void * {
    std::memcpy(h + pos, src, bytes);
    const void *dp = dbase + pos;
    pos += (bytes + 15) / 16 * 16;
    return dp;
  };
  const int n = p.nblocks;
  dev.raw_off = (const int64_t *)put(p.raw_off.data(), 8 * n);
  dev.off = (const int64_t *)put(p.off.data(), 8 * n);
  dev.cap = (const int64_t *)put(p.cap.data(), 8 * n);
  dev.raw_len = (const int *)put(p.raw_len.data(), 4 * n);
  dev.rt_block = (const int *)put(p.rt_block.data(), 4 * p.rt_block.size());
  dev.rt_start = (const int *)put(p.rt_start.data(), 4 * p.rt_start.size());
  dev.rt_first = (const int *)put(p.rt_first.data(), 4 * (n + 1));
  dev.tile_block = (const int *)put(p.tile_block.data(), 4 * p.tile_block.size());
  dev.gt_block = (const int *)put(p.gt_block.data(), 4 * p.gt_block.size());
  dev.gt_first = (const int *)put(p.gt_first.data(), 4 * p.gt_first.size());
  dev.gt_begin = (const int *)put(p.gt_begin.data(), 4 * (n + 1));
  BZ_REQUIRE(pos <= pinned_plan_bytes, kErrInternal, "plan staging overflow");
  BZ_CUDA(cudaMemcpyAsync(plan_dev_, pinned_plan, pos, cudaMemcpyHostToDevice, st));
  dev.nblocks = n;
  dev.run_cut = p.run_cut;
  dev.ntiles = (int)p.tile_block.size();
  dev.n_raw_tiles = (int)p.rt_block.size();
  dev.n_group_tiles = (int)p.gt_block.size();
}

Workspace *Workspace::create_for(int max_blocks, int64_t max_block_bytes, int block_slots) {
  const int64_t nb = std::max<int64_t>(max_block_bytes, 1);
  const int64_t cap = align_up(std::max<int64_t>(rle1_bound(nb), 1), kTile);
  const int64_t E = (int64_t)max_blocks * cap;
  const int64_t R = (int64_t)max_blocks * align_up(nb, 16);
  BZ_REQUIRE(E + kTile < (int64_t(1) << 32), kErrArg,
             "slab too large: its element offsets must fit 32 bits (use fewer slab blocks)");
  const int mt = (int)(E / kTile);
  const int mrt = (int)(max_blocks * ((nb + kRawTile - 1) / kRawTile));
  const int mgt = (int)(max_blocks * ((groups_bound(nb) + kGroupTile - 1) / kGroupTile));
  return new Workspace(std::max(max_blocks, block_slots), R, E, mt, mrt, mgt);
}

namespace {

// One block of threads lists, in block order, the tiles that hold data:
// element tiles (groups = 0) of the m[b] bytes from off[b], or group tiles
// (groups = 1) of the ceil(s[b] / 50) groups from gt_begin[b].  The count
// goes to sort_ctl[10 + groups].
__global__ void __launch_bounds__(256) k_live_tiles(SlabDev d, int groups) {
  __shared__ int scratch[40];
  int32_t *list = groups ? d.vg_list : d.vt_list;
  int base = 0, mmax = 0;
  for (int b0 = 0; b0 < d.nblocks; b0 += 256) {
    const int b = b0 + threadIdx.x;
    int cnt = 0, first = 0;
    if (b < d.nblocks) {
      if (groups) {
        const int s = d.s[b];
        const int nsel = s > 0 ? (s + kGroupSize - 1) / kGroupSize : 0;
        cnt = (nsel + kGroupTile - 1) / kGroupTile;
        first = d.gt_begin[b];
      } else {
        const int m = d.m[b];
        cnt = m > 0 ? (m + kTile - 1) / kTile : 0;
        first = (int)(d.off[b] / kTile);
        mmax = max(mmax, m);
      }
    }
    int tot;
    const int at = base + block_excl_sum(cnt, scratch, &tot);
    for (int k = 0; k < cnt; k++) list[at + k] = first + k;
    base += tot;
  }
  if (!groups) {
    for (int o = 16; o > 0; o >>= 1) mmax = max(mmax, __shfl_xor_sync(0xffffffffu, mmax, o));
    if (lane_id() == 0) atomicMax(&d.sort_ctl[12], mmax);
  }
  if (threadIdx.x == 0) d.sort_ctl[10 + groups] = base;
}

int live_list(const SlabDev &d, cudaStream_t st, int groups) {
  if (!d.live) return -1;
  if (d.live[groups] >= 0) return d.live[groups];
  if (!groups) BZ_CUDA(cudaMemsetAsync(d.sort_ctl + 12, 0, sizeof(int32_t), st));
  k_live_tiles<<<1, 256, 0, st>>>(d, groups);
  BZ_LAUNCH_CHECK();
  BZ_CUDA(cudaMemcpyAsync(d.live + 4, d.sort_ctl + 10, 3 * sizeof(int32_t),
                          cudaMemcpyDeviceToHost, st));
  BZ_CUDA(cudaStreamSynchronize(st));
  d.live[groups] = d.live[4 + groups];
  if (!groups) d.live[2] = d.live[6];  // the largest m of the slab
  return d.live[groups];
}

}  // namespace

int live_tiles(const SlabDev &d, cudaStream_t st) { return live_list(d, st, 0); }
int live_group_tiles(const SlabDev &d, cudaStream_t st) { return live_list(d, st, 1); }

}  // namespace bz2g
