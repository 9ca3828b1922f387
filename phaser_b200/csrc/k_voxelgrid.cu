// Voxel-grid downsampling on the GPU: preproc::VoxelGridCmd
// (phaser_pre/src/commands/voxel-grid-cmd.cc:11-22), which runs
// pcl::VoxelGrid<pcl::PointXYZI> (PCL 1.8.1, the libpcl-dev of the
// reference's Ubuntu 18.04 / ROS Melodic image; PCL is not part of the
// reference tree) with leaf --phaser_voxel_grid_leaf_size (0.25) in place.
//
// pcl::VoxelGrid::applyFilter, restated:
//   * min/max of x, y, z over the finite points (getMinMax3D);
//   * inv = 1 / leaf (float); d = int64((max - min) * inv) + 1 per axis; if
//     dx*dy*dz > INT32_MAX the output is the input (an overflow warning);
//   * min_b = int(floor(min * inv)), max_b = int(floor(max * inv)),
//     div_b = max_b - min_b + 1, multipliers (1, div_x, div_x * div_y);
//   * per finite point: ijk = int(floor(p * inv) - float(min_b)) per axis and
//     leaf index = ijk . multipliers (x fastest);
//   * sort the (leaf, point) pairs by leaf; every run of one leaf with at least
//     min_points_per_voxel points becomes one output point, the float sum of
//     x, y, z, intensity over the run divided by float(run length); leaves
//     come out in increasing leaf index.
// PCL sorts with std::sort, whose order among the points of one leaf is
// unspecified; here the sort is stable, so a leaf's points are summed in
// input order, which fixes the result bit for bit (the oracle sums in the
// same order).  Non-finite points are dropped (PCL does so for clouds flagged
// not dense and is undefined otherwise).  Leaf grids whose indices leave
// int32 (|floor(coordinate / leaf)| >= 2^31), with more than 2^30 leaves along
// an axis, or whose cell count leaves 32 bits are refused with
// PHGPU_ERR_LIMIT: PCL's int arithmetic is undefined there.
//
// GPU layout: every step is a pass over 32-bit words in HBM -- a bounds
// reduction that ends in the plan, stable 8-bit LSD radix passes over the
// leaf index's bits (a ranked scatter per tile, which also counts the tile's
// items for the next pass; the first makes the (leaf, point) pairs of the
// finite points), a compaction of the leaf heads, and the centroids: a leaf of up
// to 128 points by a warp that stages them in one batch, a longer one by its
// block, whose other warps gather the next 896 points while the first adds, one
// lane per component, in input order.
// Nothing synchronises the host until the output count is read.  Bound by the
// latency of the nine dependent launches: a 131072-point scan at 0.25 m takes
// 84 us (154 with twenty-one launches and one lane adding a leaf).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <string>

#include "../../include/phaser_gpu.h"
#include "kernels.h"

namespace phgpu {
namespace {

constexpr int kVgThreads = 256;
constexpr int kVgWarps = kVgThreads / 32;
// 4 rounds: a 131072-point scan fills 128 blocks (8 rounds: 64 of the 148 SMs busy, 130 us a call against
// 117; equal from a million points on)
constexpr int kVgRounds = 4;
constexpr int kVgTile = kVgThreads * kVgRounds;  // items per block and pass
constexpr int kBins = 256;                        // 8-bit radix digits
constexpr int kScanThreads = 1024;

enum VgStatus : int32_t { kVgOk = 0, kVgEmpty = 1, kVgOverflow = 2, kVgRange = 3 };

struct VgState {
  uint32_t lo_inv[3];  // max of ~order(x): decodes to the minimum
  uint32_t hi[3];      // max of order(x); 0 = no finite point
  int32_t status;
  int32_t min_b[3];
  uint32_t mul[3];
  uint32_t n_passes;  // 8-bit radix passes that cover every leaf index
  uint32_t ticket;    // blocks of the bounds pass that are done
  uint32_t n_valid;   // finite points
  uint32_t n_leaves;  // occupied leaves
  uint32_t n_out;     // leaves kept (>= min points)
};

__device__ __forceinline__ bool finite3(float4 p) { return isfinite(p.x) && isfinite(p.y) && isfinite(p.z); }

__device__ __forceinline__ uint32_t lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// ---------------------------------------------------------------- bounds and plan
// Per block: max of ~order(v) (decodes to the minimum) and of order(v) per
// axis over the finite points, written to part[block][6]; the block that
// finishes last reduces the blocks and plans the grid (no atomics on a few hot
// words but the ticket, and no launch of its own).
constexpr int kBoundsBlocks = 148 * 4;

__device__ void vg_plan(const uint32_t (&m)[6], VgState* st, float inv_x, float inv_y, float inv_z);

__device__ __forceinline__ void block_max6(uint32_t (&m)[6], uint32_t (*s_m)[6]) {
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    for (int off = 16; off > 0; off >>= 1) m[c] = max(m[c], __shfl_xor_sync(0xffffffffu, m[c], off));
    if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5][c] = m[c];
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    m[c] = 0;
    for (int w = 0; w < kVgWarps; ++w) m[c] = max(m[c], s_m[w][c]);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kVgThreads) k_vg_bounds(const float4* __restrict__ pts, uint32_t n, uint32_t* part,
                                                          VgState* st, float inv_x, float inv_y, float inv_z) {
  chain_begin();
  uint32_t m[6] = {0, 0, 0, 0, 0, 0};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 p = pts[i];
    if (!finite3(p)) continue;
    const float v[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t o = float_order_bits(v[a]);
      m[a] = max(m[a], ~o);
      m[3 + a] = max(m[3 + a], o);
    }
  }
  __shared__ uint32_t s_m[kVgWarps][6];
  __shared__ bool s_last;
  block_max6(m, s_m);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < 6; ++c) part[blockIdx.x * 6 + c] = m[c];
    __threadfence();
    s_last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kVgThreads)
#pragma unroll
    for (int c = 0; c < 6; ++c) m[c] = max(m[c], __ldcg(&part[b * 6 + c]));
  block_max6(m, s_m);
  if (threadIdx.x == 0) vg_plan(m, st, inv_x, inv_y, inv_z);
}

__device__ void vg_plan(const uint32_t (&m)[6], VgState* st, float inv_x, float inv_y, float inv_z) {
  for (int a = 0; a < 3; ++a) {
    st->lo_inv[a] = m[a];
    st->hi[a] = m[3 + a];
  }
  st->n_valid = st->n_leaves = st->n_out = 0;
  if (st->hi[0] == 0) {
    st->status = kVgEmpty;
    return;
  }
  const float inv[3] = {inv_x, inv_y, inv_z};
  float mn[3], mx[3];
  long long d[3], div[3];
  bool overflow = false, range = false;
  for (int a = 0; a < 3; ++a) {
    mn[a] = float_from_order_bits(~st->lo_inv[a]);
    mx[a] = float_from_order_bits(st->hi[a]);
    const float ext = __fmul_rn(__fsub_rn(mx[a], mn[a]), inv[a]);
    if (!(ext < 4.0e18f)) {  // the int64 conversion itself would overflow
      overflow = true;
      d[a] = 0;
    } else {
      d[a] = (long long)ext + 1;
    }
    const float fb_lo = floorf(__fmul_rn(mn[a], inv[a]));
    const float fb_hi = floorf(__fmul_rn(mx[a], inv[a]));
    if (!(fb_lo >= -2147483648.0f && fb_hi < 2147483648.0f)) range = true;
    st->min_b[a] = range ? 0 : (int32_t)fb_lo;
    div[a] = range ? 1 : (long long)(int32_t)fb_hi - (long long)(int32_t)fb_lo + 1;
    // ijk = float(floor) - float(min_b) must convert to int exactly
    if (div[a] > (1ll << 30)) range = true;
  }
  if (!overflow) {
    // dx * dy * dz > INT32_MAX, evaluated without int64 overflow
    if (d[0] > 2147483647ll || d[1] > 2147483647ll || d[2] > 2147483647ll) overflow = true;
    else if (d[0] * d[1] > 2147483647ll) overflow = true;
    else overflow = d[0] * d[1] * d[2] > 2147483647ll;
  }
  if (overflow) {
    st->status = kVgOverflow;
    return;
  }
  const unsigned long long cells = (unsigned long long)div[0] * (unsigned long long)div[1] * (unsigned long long)div[2];
  if (range || cells > 0xffffffffull) {
    st->status = kVgRange;
    return;
  }
  st->n_passes = cells <= 0x100ull ? 1u : (cells <= 0x10000ull ? 2u : (cells <= 0x1000000ull ? 3u : 4u));
  st->mul[0] = 1u;
  st->mul[1] = (uint32_t)div[0];
  st->mul[2] = (uint32_t)div[0] * (uint32_t)div[1];
  st->status = kVgOk;
}

// ---------------------------------------------------------------- scan
// Exclusive scan of `len` words by one block; *total gets the sum.
__global__ void __launch_bounds__(kScanThreads) k_scan_words(const uint32_t* __restrict__ in, uint32_t len,
                                                             uint32_t* __restrict__ out, uint32_t* total) {
  chain_begin();
  __shared__ uint32_t s_warp[kScanThreads / 32];
  const uint32_t chunk = (len + kScanThreads - 1) / kScanThreads;
  const uint32_t b = threadIdx.x * chunk;
  const uint32_t e = min(len, b + chunk);
  uint32_t sum = 0;
  for (uint32_t i = b; i < e; ++i) sum += in[i];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = s_warp[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += v;
    }
    s_warp[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  uint32_t run = incl - sum + (warp > 0 ? s_warp[warp - 1] : 0u);
  for (uint32_t i = b; i < e; ++i) {
    const uint32_t v = in[i];
    out[i] = run;
    run += v;
  }
  if (threadIdx.x == kScanThreads - 1 && total) *total = run;
}

// ---------------------------------------------------------------- stable compaction
// Op: __device__ uint32_t n() const; bool flag(uint32_t i) const (i < n());
//     void emit(uint32_t i, uint32_t pos) const.  Item order inside a tile
//     is (round, thread), i.e. ascending index, so ranks are stable.
template <class Op>
__global__ void __launch_bounds__(kVgThreads) k_flag_count(Op op, uint32_t* __restrict__ counts) {
  chain_begin();
  const uint32_t n = op.n();
  const uint32_t base = blockIdx.x * kVgTile;
  bool f[kVgRounds];  // all of the tile's flags first: one load latency, not one per round
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t i = base + r * kVgThreads + threadIdx.x;
    f[r] = i < n && op.flag(i);
  }
  uint32_t c = 0;
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) c += __popc(__ballot_sync(0xffffffffu, f[r]));
  __shared__ uint32_t s[kVgWarps];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kVgWarps; ++w) t += s[w];
    counts[blockIdx.x] = t;
  }
}

// offsets == nullptr: every block adds the counts of the tiles before it itself
// (the last one also writes the total), which is cheaper than a one-block scan
// and its launch for as long as it is a few coalesced loads a thread.
constexpr uint32_t kSelfScanTiles = 4096;

template <class Op>
__global__ void __launch_bounds__(kVgThreads) k_flag_scatter(Op op, const uint32_t* __restrict__ counts,
                                                             const uint32_t* __restrict__ offsets, uint32_t* total) {
  chain_begin();
  const uint32_t n = op.n();
  const uint32_t base = blockIdx.x * kVgTile;
  __shared__ uint32_t s_w[kVgWarps];
  const int warp = threadIdx.x >> 5;
  if (base >= n && (offsets || blockIdx.x != gridDim.x - 1)) return;
  uint32_t run = 0;
  if (offsets) {
    run = offsets[blockIdx.x];
  } else {
    for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kVgThreads) run += counts[i];
    run = __reduce_add_sync(0xffffffffu, run);
    if ((threadIdx.x & 31) == 0) s_w[warp] = run;
    __syncthreads();
    run = 0;
    for (int w = 0; w < kVgWarps; ++w) run += s_w[w];
    __syncthreads();
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = run + counts[blockIdx.x];
    if (base >= n) return;
  }
  bool fl[kVgRounds];
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t i = base + r * kVgThreads + threadIdx.x;
    fl[r] = i < n && op.flag(i);
  }
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t i = base + r * kVgThreads + threadIdx.x;
    const bool f = fl[r];
    const uint32_t bal = __ballot_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0) s_w[warp] = __popc(bal);
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int w = 0; w < kVgWarps; ++w) {
      const uint32_t c = s_w[w];
      before += w < warp ? c : 0u;
      all += c;
    }
    if (f) op.emit(i, run + before + __popc(bal & lanemask_lt()));
    run += all;
    __syncthreads();
  }
}

// First entry of every run of one leaf in the sorted pairs.
struct HeadOp {
  const uint32_t* keys0;
  const uint32_t* keys1;
  const VgState* st;
  uint32_t* leaf_start;
  __device__ uint32_t n() const { return st->n_valid; }
  __device__ bool flag(uint32_t i) const {
    const uint32_t* keys = st->n_passes & 1u ? keys0 : keys1;
    return i == 0 || keys[i] != keys[i - 1];
  }
  __device__ void emit(uint32_t i, uint32_t pos) const { leaf_start[pos] = i; }
};

// Leaves with at least min_points points (centroids staged per leaf).
struct KeepOp {
  const uint32_t* leaf_start;
  const VgState* st;
  uint32_t min_points;
  const float4* tmp;
  const float* tmp_refl;
  const float* tmp_amb;
  float4* out;
  float* out_refl;
  float* out_amb;
  __device__ uint32_t n() const { return st->n_leaves; }
  __device__ bool flag(uint32_t j) const {
    const uint32_t e = j + 1 < st->n_leaves ? leaf_start[j + 1] : st->n_valid;
    return e - leaf_start[j] >= min_points;
  }
  __device__ void emit(uint32_t j, uint32_t pos) const {
    out[pos] = tmp[j];
    if (out_refl) out_refl[pos] = tmp_refl[j];
    if (out_amb) out_amb[pos] = tmp_amb[j];
  }
};

// ---------------------------------------------------------------- radix passes
// Pass p writes the pairs to buffer p & 1.  The first pass makes the keys from
// the points and leaves the non-finite ones out, so no compaction runs before
// it; passes beyond the leaf indices' bits return at once (a 20 x 15 x 6 m
// room at 0.25 m has 74 k cells: three passes), and the readers behind the
// last pass pick its buffer.
struct PointKeys {
  const float4* pts;
  uint32_t n_points;
  float inv[3];
};

__device__ __forceinline__ bool point_key(const PointKeys& pk, const VgState* st, uint32_t i, uint32_t* key) {
  const float4 p = pk.pts[i];
  const float v[3] = {p.x, p.y, p.z};
  *key = 0;
  if (!finite3(p)) return false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float f = floorf(__fmul_rn(v[a], pk.inv[a]));
    const int32_t ijk = (int32_t)__fsub_rn(f, (float)st->min_b[a]);
    *key += (uint32_t)ijk * st->mul[a];
  }
  return true;
}

// Pairs the pass reads: all points of a planned grid in the first, the finite
// ones after it, none in a pass that has nothing to do.
template <bool FIRST>
__device__ __forceinline__ uint32_t pass_items(const PointKeys& pk, const VgState* st, int pass) {
  if (FIRST) return st->status == kVgOk ? pk.n_points : 0u;
  return pass < (int)st->n_passes ? st->n_valid : 0u;
}

// Digit counts of the first pass's tiles, counts[tile][digit]; the later
// passes' counts are added up by the scatter before them.
__global__ void __launch_bounds__(kVgThreads) k_radix_count(PointKeys pk, const VgState* st,
                                                            uint32_t* __restrict__ counts,
                                                            uint32_t* __restrict__ clear) {
  chain_begin();
  __shared__ uint32_t s_hist[kBins];
  const uint32_t n = pass_items<true>(pk, st, 0);
  s_hist[threadIdx.x] = 0;
  clear[blockIdx.x * kBins + threadIdx.x] = 0;
  __syncthreads();
  const uint32_t base = blockIdx.x * kVgTile;
  uint32_t dg[kVgRounds];
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t i = base + r * kVgThreads + threadIdx.x;
    uint32_t key = 0;
    dg[r] = i < n && point_key(pk, st, i, &key) ? key & 0xffu : 0x100u;
  }
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t d = dg[r];
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    if (d < kBins && (peers & lanemask_lt()) == 0) atomicAdd(&s_hist[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  counts[blockIdx.x * kBins + threadIdx.x] = s_hist[threadIdx.x];
}

// Per digit: exclusive scan of its tile counts and the digit's total, for
// clouds of more than kSelfRadixTiles tiles.  A block takes 32 digits (lane =
// digit, so every load is one coalesced row); its warps take equal chunks of
// the tiles, sum them, and run over them again from the chunks' scanned sums.
constexpr int kRadixScanThreads = 1024;
constexpr int kScanRows = 16;

__global__ void __launch_bounds__(kRadixScanThreads) k_radix_scan(const VgState* st, int pass,
                                                                  const uint32_t* __restrict__ counts, uint32_t n_tiles,
                                                                  uint32_t* __restrict__ offsets,
                                                                  uint32_t* __restrict__ digit_total) {
  chain_begin();
  if (pass > 0 && pass >= (int)st->n_passes) return;
  constexpr int kWarps = kRadixScanThreads / 32;
  __shared__ uint32_t s_sum[kWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t d = blockIdx.x * 32 + lane;
  const uint32_t chunk = (n_tiles + kWarps - 1) / kWarps;
  const uint32_t t0 = min(n_tiles, w * chunk), t1 = min(n_tiles, t0 + chunk);
  uint32_t sum = 0;
  for (uint32_t t = t0; t < t1; t += kScanRows) {
    uint32_t v[kScanRows];
#pragma unroll
    for (int q = 0; q < kScanRows; ++q) v[q] = t + q < t1 ? counts[(size_t)(t + q) * kBins + d] : 0u;
#pragma unroll
    for (int q = 0; q < kScanRows; ++q) sum += v[q];
  }
  s_sum[w][lane] = sum;
  __syncthreads();
  uint32_t run = 0, all = 0;
  for (int k = 0; k < kWarps; ++k) {
    const uint32_t v = s_sum[k][lane];
    run += k < w ? v : 0u;
    all += v;
  }
  if (w == 0) digit_total[d] = all;
  for (uint32_t t = t0; t < t1; t += kScanRows) {
    uint32_t v[kScanRows];
#pragma unroll
    for (int q = 0; q < kScanRows; ++q) v[q] = t + q < t1 ? counts[(size_t)(t + q) * kBins + d] : 0u;
#pragma unroll
    for (int q = 0; q < kScanRows; ++q) {
      if (t + q < t1) offsets[(size_t)(t + q) * kBins + d] = run;
      run += v[q];
    }
  }
}

// Stable scatter of one tile: items are ranked in tile order into a
// digit-sorted copy of the tile in shared memory, then written out in that
// order, so each digit's run of the tile lands in consecutive words.  Each item
// is also counted for the next pass, in the tile where it lands; `clear` (the
// counts read two passes from now) is zeroed on the way.  Up to
// kSelfRadixTiles tiles every block adds up the counts of all tiles itself
// (16-byte loads, 4 tiles at a time), which saves the scan's launch; the work
// grows with the square of the tiles.  A call on 128 tiles: 115 us, with the
// scan kernel 124; on 320 tiles: 198 us and 183.
constexpr uint32_t kSelfRadixTiles = 192;

template <bool FIRST>
__global__ void __launch_bounds__(kVgThreads) k_radix_scatter(const uint32_t* __restrict__ keys_in,
                                                              const uint32_t* __restrict__ vals_in,
                                                              uint32_t* __restrict__ keys_out,
                                                              uint32_t* __restrict__ vals_out, PointKeys pk,
                                                              VgState* st, int pass,
                                                              const uint32_t* __restrict__ counts,
                                                              const uint32_t* __restrict__ offsets,
                                                              const uint32_t* __restrict__ digit_total,
                                                              uint32_t* __restrict__ next_counts,
                                                              uint32_t* __restrict__ clear) {
  chain_begin();
  __shared__ uint32_t s_key[kVgTile];
  __shared__ uint32_t s_val[kVgTile];
  __shared__ uint32_t s_local[kBins];  // start of each digit in the sorted tile
  __shared__ uint32_t s_run[kBins];    // next free position of each digit
  __shared__ uint32_t s_gbase[kBins];  // global position of the tile's first item of each digit
  __shared__ __align__(16) uint32_t s_wc[kVgWarps][kBins];
  __shared__ uint32_t s_tile_n;
  const uint32_t n = pass_items<FIRST>(pk, st, pass);
  const uint32_t n_passes = st->n_passes;
  const int shift = 8 * pass;
  const uint32_t base = blockIdx.x * kVgTile;
  clear[blockIdx.x * kBins + threadIdx.x] = 0;
  if (base >= n) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t k[kVgRounds], v[kVgRounds], dg[kVgRounds];
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t i = base + r * kVgThreads + threadIdx.x;
    bool ok = i < n;
    if (FIRST) {
      k[r] = 0;
      ok = ok && point_key(pk, st, i, &k[r]);
      v[r] = i;
    } else {
      k[r] = ok ? keys_in[i] : 0u;
      v[r] = ok ? vals_in[i] : 0u;
    }
    dg[r] = ok ? (k[r] >> shift) & 0xffu : 0x100u;
  }
  const uint32_t h = counts[blockIdx.x * kBins + threadIdx.x];
  uint32_t tot = 0, goff = 0;
  if (offsets) {
    tot = digit_total[threadIdx.x];
    goff = offsets[(size_t)blockIdx.x * kBins + threadIdx.x];
  } else {
    static_assert(kVgWarps == 8 && kBins == 256 && kVgThreads == 256, "4 tiles at a time, 64 lanes of 4 digits each");
    const uint4* __restrict__ c4 = reinterpret_cast<const uint4*>(counts) + (threadIdx.x & 63);
    uint4 a = make_uint4(0, 0, 0, 0), p = make_uint4(0, 0, 0, 0);
#pragma unroll 8
    for (uint32_t t = threadIdx.x >> 6; t < gridDim.x; t += 4) {
      const uint4 c = c4[t * (kBins / 4)];
      const uint32_t m = t < blockIdx.x ? 0xffffffffu : 0u;
      a.x += c.x, a.y += c.y, a.z += c.z, a.w += c.w;
      p.x += c.x & m, p.y += c.y & m, p.z += c.z & m, p.w += c.w & m;
    }
    reinterpret_cast<uint4*>(s_wc[threadIdx.x >> 6])[threadIdx.x & 63] = a;
    reinterpret_cast<uint4*>(s_wc[4 + (threadIdx.x >> 6)])[threadIdx.x & 63] = p;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      tot += s_wc[q][threadIdx.x];
      goff += s_wc[4 + q][threadIdx.x];
    }
    __syncthreads();
  }
  // exclusive scans over the 256 digits: the tile's counts and the digit totals
  uint32_t ih = h, it = tot;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, ih, o);
    const uint32_t b = __shfl_up_sync(0xffffffffu, it, o);
    if (lane >= o) {
      ih += a;
      it += b;
    }
  }
  if (lane == 31) {
    s_wc[0][warp] = ih;
    s_wc[1][warp] = it;
  }
  __syncthreads();
  uint32_t bh = 0, bt = 0;
  for (int w = 0; w < warp; ++w) {
    bh += s_wc[0][w];
    bt += s_wc[1][w];
  }
  __syncthreads();
  s_local[threadIdx.x] = bh + ih - h;
  s_run[threadIdx.x] = bh + ih - h;
  s_gbase[threadIdx.x] = bt + it - tot + goff;
  if (threadIdx.x == kBins - 1) {
    s_tile_n = bh + ih;
    if (FIRST && blockIdx.x == 0) st->n_valid = bt + it;
  }
  for (int w = 0; w < kVgWarps; ++w) s_wc[w][threadIdx.x] = 0;
  __syncthreads();
  // stable ranks into the sorted tile
#pragma unroll
  for (int r = 0; r < kVgRounds; ++r) {
    const uint32_t d = dg[r];
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const uint32_t rank = __popc(peers & lanemask_lt());
    if (d < kBins && rank == 0) s_wc[warp][d] = __popc(peers);
    __syncthreads();
    if (d < kBins) {
      uint32_t pos = s_run[d] + rank;
      for (int w = 0; w < warp; ++w) pos += s_wc[w][d];
      s_key[pos] = k[r];
      s_val[pos] = v[r];
    }
    __syncthreads();
    uint32_t t = 0;
    for (int w = 0; w < kVgWarps; ++w) {
      t += s_wc[w][threadIdx.x];
      s_wc[w][threadIdx.x] = 0;
    }
    s_run[threadIdx.x] += t;
    __syncthreads();
  }
  const uint32_t tile_n = s_tile_n;
  const bool count_next = pass + 1 < (int)n_passes;
  for (uint32_t L0 = 0; L0 < tile_n; L0 += kVgThreads) {
    const uint32_t L = L0 + threadIdx.x;
    uint32_t slot = 0xffffffffu;
    if (L < tile_n) {
      const uint32_t key = s_key[L];
      const uint32_t d = (key >> shift) & 0xffu;
      const uint32_t g = s_gbase[d] + (L - s_local[d]);
      keys_out[g] = key;
      vals_out[g] = s_val[L];
      if (count_next) slot = g / kVgTile * kBins + ((key >> (shift + 8)) & 0xffu);
    }
    if (count_next) {
      const uint32_t peers = __match_any_sync(0xffffffffu, slot);
      if (L < tile_n && (peers & lanemask_lt()) == 0) atomicAdd(&next_counts[slot], (uint32_t)__popc(peers));
    }
  }
}

// ---------------------------------------------------------------- centroids
// The float sums run over a leaf in input order exactly as one thread would,
// divided by float(count) at the end.  A leaf near the sensor holds thousands
// of points (9215 of a 131072-point scan at 0.25 m), and its chain of dependent
// additions bounds the kernel: the points are staged in shared memory and one
// lane per component (x, y, z, intensity, reflectivity, ambient) adds them,
// four points per shared load and the next loads ahead of the additions, so
// that a point costs one addition's latency (a 2^20-point scan whose longest
// leaf holds some 70 k points: 790 us a call with one warp per leaf, 351 so).  Leaves of up to kLeafWarp points
// take a warp each; in a longer one the block's other warps gather the next
// kChunk points while the first warp adds, because a warp that gathers for
// itself waits for its loads between batches (19 cycles a point).  A block's
// leaves lie a grid apart: neighbouring leaves are long together.
constexpr int kLeafWarp = 128;
constexpr int kChunk = 896;
constexpr int kStage = kLeafWarp / 32;
constexpr int kGather = kVgThreads - 32;
static_assert(kVgWarps * kLeafWarp <= 2 * kChunk && kChunk % kGather == 0 && kChunk % 4 == 0,
              "the warps' batches and the two chunks share the staging");

// Staged points: [group of 4 points][component][point], so the components'
// 16-byte loads of one group are neighbours.
typedef float VgGroup[6][4];

__device__ __forceinline__ float add4(float sum, float4 v) {
  return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
}

__device__ __forceinline__ float add_points(const VgGroup* __restrict__ g, uint32_t cnt, int comp, float sum) {
  const uint32_t full = cnt >> 2;
  uint32_t t = 0;
  if (full >= 4) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(g[u][comp]);
    for (; t + 8 <= full; t += 4) {
      float4 nx[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) nx[u] = *reinterpret_cast<const float4*>(g[t + 4 + u][comp]);
#pragma unroll
      for (int u = 0; u < 4; ++u) sum = add4(sum, v[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = nx[u];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) sum = add4(sum, v[u]);
    t += 4;
  }
  for (; t < full; ++t) sum = add4(sum, *reinterpret_cast<const float4*>(g[t][comp]));
  for (uint32_t k = 0; k < (cnt & 3u); ++k) sum = __fadd_rn(sum, g[full][comp][k]);
  return sum;
}

struct LeafPoints {
  const float4* __restrict__ pts;
  const float* __restrict__ refl;
  const float* __restrict__ amb;
  const uint32_t* __restrict__ vals;
};

// Points first, first + STRIDE, ... (Q of them, below n) of the run at b into
// the staging: all the indices, then all the points in flight.
template <int Q, int STRIDE>
__device__ __forceinline__ void stage_points(const LeafPoints& lp, uint32_t b, uint32_t n, uint32_t first, VgGroup* g) {
  uint32_t idx[Q];
  float4 p[Q];
  float r[Q], a[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) idx[q] = first + q * STRIDE < n ? lp.vals[b + first + q * STRIDE] : 0xffffffffu;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (idx[q] == 0xffffffffu) continue;
    p[q] = lp.pts[idx[q]];
    r[q] = lp.refl ? lp.refl[idx[q]] : 0.f;
    a[q] = lp.amb ? lp.amb[idx[q]] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (idx[q] == 0xffffffffu) continue;
    const uint32_t i = first + q * STRIDE;
    float* o = &g[i >> 2][0][i & 3u];
    o[0] = p[q].x;
    o[4] = p[q].y;
    o[8] = p[q].z;
    o[12] = p[q].w;
    o[16] = r[q];
    o[20] = a[q];
  }
}

// Lanes 0..5 of one warp hold the components of the leaf's sum.
__device__ __forceinline__ void write_leaf(float sum, uint32_t n, uint32_t j, int lane, float4* out, float* out_refl,
                                           float* out_amb) {
  const float mean = __fdiv_rn(sum, __uint2float_rn(n));
  const float my = __shfl_sync(0xffffffffu, mean, 1), mz = __shfl_sync(0xffffffffu, mean, 2),
              mi = __shfl_sync(0xffffffffu, mean, 3);
  if (lane == 0) out[j] = make_float4(mean, my, mz, mi);
  if (lane == 4 && out_refl) out_refl[j] = mean;
  if (lane == 5 && out_amb) out_amb[j] = mean;
}

__global__ void __launch_bounds__(kVgThreads) k_vg_centroid(const float4* __restrict__ pts,
                                                            const float* __restrict__ refl,
                                                            const float* __restrict__ amb,
                                                            const uint32_t* __restrict__ vals0,
                                                            const uint32_t* __restrict__ vals1,
                                                            const uint32_t* __restrict__ leaf_start,
                                                            VgState* st, float4* out, float* out_refl,
                                                            float* out_amb, int direct) {
  chain_begin();
  __shared__ __align__(16) VgGroup s_c[2 * kChunk / 4];
  __shared__ uint32_t s_b[kVgWarps], s_n[kVgWarps];
  const uint32_t n_leaves = st->n_leaves;
  const uint32_t n_valid = st->n_valid;
  const LeafPoints lp{pts, refl, amb, st->n_passes & 1u ? vals0 : vals1};
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (direct && blockIdx.x == 0 && threadIdx.x == 0) st->n_out = n_leaves;
  const uint32_t step = gridDim.x * kVgWarps;
  for (uint32_t j0 = blockIdx.x; j0 < n_leaves; j0 += step) {
    const uint32_t j = j0 + w * gridDim.x;
    uint32_t b = 0, n = 0;
    if (j < n_leaves) {
      b = leaf_start[j];
      n = (j + 1 < n_leaves ? leaf_start[j + 1] : n_valid) - b;
    }
    if (n && n <= kLeafWarp) {
      VgGroup* g = s_c + w * (kLeafWarp / 4);
      stage_points<kStage, 32>(lp, b, n, lane, g);
      __syncwarp();
      write_leaf(lane < 6 ? add_points(g, n, lane, 0.f) : 0.f, n, j, lane, out, out_refl, out_amb);
    }
    if (lane == 0) {
      s_b[w] = b;
      s_n[w] = n;
    }
    if (!__syncthreads_or(n > kLeafWarp)) continue;
    for (int u = 0; u < kVgWarps; ++u) {
      const uint32_t lb = s_b[u], ln = s_n[u];
      if (ln <= kLeafWarp) continue;
      if (w > 0) stage_points<(kChunk + kGather - 1) / kGather, kGather>(lp, lb, min(ln, (uint32_t)kChunk), threadIdx.x - 32, s_c);
      float sum = 0.f;
      for (uint32_t c = 0; c < ln; c += kChunk) {
        const int buf = (c / kChunk) & 1;
        __syncthreads();
        if (w == 0) {
          if (lane < 6) sum = add_points(s_c + buf * (kChunk / 4), min(ln - c, (uint32_t)kChunk), lane, sum);
        } else if (c + kChunk < ln) {
          stage_points<(kChunk + kGather - 1) / kGather, kGather>(lp, lb + c + kChunk, min(ln - c - kChunk, (uint32_t)kChunk),
                                                                  threadIdx.x - 32, s_c + (buf ^ 1) * (kChunk / 4));
        }
      }
      if (w == 0) {
        __syncwarp();
        write_leaf(sum, ln, j0 + u * gridDim.x, lane, out, out_refl, out_amb);
      }
      __syncthreads();
    }
    // no warp writes the next batch's s_b, s_n before every warp has read this one's to the last leaf
    __syncthreads();
  }
}

uint32_t tiles_for(uint32_t n) { return (n + kVgTile - 1) / kVgTile; }

}  // namespace
}  // namespace phgpu

using namespace phgpu;

struct phgpu_voxel_grid {
  int device = 0;
  uint32_t max_points = 0;
  uint32_t max_tiles = 0;
  cudaStream_t st = nullptr;
  std::string err;
  float4* d_in = nullptr;
  float* d_in_refl = nullptr;
  float* d_in_amb = nullptr;
  uint32_t* keys[2] = {nullptr, nullptr};
  uint32_t* vals[2] = {nullptr, nullptr};
  uint32_t* leaf_start = nullptr;
  uint32_t* counts[3] = {nullptr, nullptr, nullptr};  // kBins * max_tiles: a pass reads one, adds to one, clears one
  uint32_t* offsets = nullptr;      // kBins * max_tiles, beyond kSelfRadixTiles
  uint32_t* digit_total = nullptr;  // kBins
  uint32_t* tile_counts = nullptr;  // 2 * max_tiles: flagged items per tile and their scan
  uint32_t* part = nullptr;         // the bounds pass's partials
  float4* d_out = nullptr;      // outputs when the caller's are host memory; per-leaf staging otherwise
  float* d_out_refl = nullptr;
  float* d_out_amb = nullptr;
  float4* d_tmp = nullptr;      // per-leaf centroids when min points > 1
  float* d_tmp_refl = nullptr;
  float* d_tmp_amb = nullptr;
  VgState* d_state = nullptr;
  VgState* h_state = nullptr;  // pinned
};

namespace {

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

thread_local std::string g_vg_create_error;

#define VG_CK(expr)                                                  \
  do {                                                               \
    cudaError_t _e = (expr);                                         \
    if (_e != cudaSuccess) {                                         \
      vg->err = std::string(#expr) + ": " + cudaGetErrorString(_e); \
      return PHGPU_ERR_CUDA;                                         \
    }                                                                \
  } while (0)

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

}  // namespace

int phgpu_voxel_grid_create(uint32_t max_points, int32_t device, phgpu_voxel_grid** out) {
  if (!out || max_points == 0 || max_points > 0x7fffffffu) {
    g_vg_create_error = "max_points must be in [1, 2^31)";
    return PHGPU_ERR_INVALID;
  }
  *out = nullptr;
  int n_dev = 0;
  if (cudaGetDeviceCount(&n_dev) != cudaSuccess || device < 0 || device >= n_dev) {
    g_vg_create_error = "no such CUDA device";
    return PHGPU_ERR_CUDA;
  }
  DeviceGuard g(device);
  phgpu_voxel_grid* vg = new phgpu_voxel_grid();
  vg->device = device;
  vg->max_points = max_points;
  vg->max_tiles = tiles_for(max_points);
  const size_t P = max_points;
  const size_t words = (size_t)kBins * vg->max_tiles;
  cudaError_t e = cudaStreamCreateWithFlags(&vg->st, cudaStreamNonBlocking);
  auto alloc = [&](void** p, size_t bytes) {
    if (e == cudaSuccess) e = cudaMalloc(p, bytes);
  };
  alloc((void**)&vg->d_in, P * sizeof(float4));
  alloc((void**)&vg->d_in_refl, P * sizeof(float));
  alloc((void**)&vg->d_in_amb, P * sizeof(float));
  for (int k = 0; k < 2; ++k) {
    alloc((void**)&vg->keys[k], P * sizeof(uint32_t));
    alloc((void**)&vg->vals[k], P * sizeof(uint32_t));
  }
  alloc((void**)&vg->leaf_start, P * sizeof(uint32_t));
  for (int k = 0; k < 3; ++k) alloc((void**)&vg->counts[k], words * sizeof(uint32_t));
  if (vg->max_tiles > kSelfRadixTiles) alloc((void**)&vg->offsets, words * sizeof(uint32_t));
  alloc((void**)&vg->tile_counts, 2 * (size_t)vg->max_tiles * sizeof(uint32_t));
  alloc((void**)&vg->part, kBoundsBlocks * 6 * sizeof(uint32_t));
  alloc((void**)&vg->digit_total, kBins * sizeof(uint32_t));
  alloc((void**)&vg->d_out, P * sizeof(float4));
  alloc((void**)&vg->d_out_refl, P * sizeof(float));
  alloc((void**)&vg->d_out_amb, P * sizeof(float));
  alloc((void**)&vg->d_tmp, P * sizeof(float4));
  alloc((void**)&vg->d_tmp_refl, P * sizeof(float));
  alloc((void**)&vg->d_tmp_amb, P * sizeof(float));
  alloc((void**)&vg->d_state, sizeof(VgState));
  if (e == cudaSuccess) e = cudaMallocHost((void**)&vg->h_state, sizeof(VgState));
  if (e != cudaSuccess) {
    g_vg_create_error = std::string("voxel grid allocation: ") + cudaGetErrorString(e);
    phgpu_voxel_grid_destroy(vg);
    return e == cudaErrorMemoryAllocation ? PHGPU_ERR_MEMORY : PHGPU_ERR_CUDA;
  }
  *out = vg;
  return PHGPU_OK;
}

int phgpu_voxel_grid_destroy(phgpu_voxel_grid* vg) {
  if (!vg) return PHGPU_ERR_INVALID;
  DeviceGuard g(vg->device);
  if (vg->st) cudaStreamSynchronize(vg->st);
  void* bufs[] = {vg->d_in, vg->d_in_refl, vg->d_in_amb, vg->keys[0], vg->keys[1], vg->vals[0], vg->vals[1],
                  vg->leaf_start, vg->counts[0], vg->counts[1], vg->counts[2], vg->offsets, vg->digit_total, vg->tile_counts, vg->part,
                   vg->d_out, vg->d_out_refl, vg->d_out_amb, vg->d_tmp,
                  vg->d_tmp_refl, vg->d_tmp_amb, vg->d_state};
  for (void* b : bufs)
    if (b) cudaFree(b);
  if (vg->h_state) cudaFreeHost(vg->h_state);
  if (vg->st) cudaStreamDestroy(vg->st);
  delete vg;
  return PHGPU_OK;
}

const char* phgpu_voxel_grid_last_error(const phgpu_voxel_grid* vg) {
  return vg ? vg->err.c_str() : g_vg_create_error.c_str();
}

int phgpu_voxel_grid_filter(phgpu_voxel_grid* vg, const phgpu_cloud* in, const float leaf[3],
                            uint32_t min_points_per_voxel, float* out_xyzi, float* out_reflectivity,
                            float* out_ambient, int out_on_device, uint32_t* n_out) {
  if (!vg) return PHGPU_ERR_INVALID;
  vg->err.clear();
  if (!in || !leaf || !out_xyzi || !n_out) {
    vg->err = "null argument";
    return PHGPU_ERR_INVALID;
  }
  if (in->n_points > vg->max_points) {
    vg->err = "cloud larger than max_points";
    return PHGPU_ERR_INVALID;
  }
  for (int a = 0; a < 3; ++a)
    if (!(leaf[a] > 0.f) || !isfinite(leaf[a])) {
      vg->err = "leaf sizes must be positive and finite";
      return PHGPU_ERR_INVALID;
    }
  if ((in->on_device && in->n_points && !aligned16(in->xyzi)) || (out_on_device && !aligned16(out_xyzi))) {
    vg->err = "device xyzi buffers must be 16-byte aligned";
    return PHGPU_ERR_INVALID;
  }
  DeviceGuard g(vg->device);
  ChainScope chain(true);
  cudaStream_t st = vg->st;
  const uint32_t n = in->n_points;
  *n_out = 0;
  if (n == 0) return PHGPU_OK;

  const float4* pts = (const float4*)in->xyzi;
  const float* refl = in->reflectivity;
  const float* amb = in->ambient;
  if (!in->on_device) {
    VG_CK(cudaMemcpyAsync(vg->d_in, in->xyzi, (size_t)n * sizeof(float4), cudaMemcpyHostToDevice, st));
    pts = vg->d_in;
    if (refl) {
      VG_CK(cudaMemcpyAsync(vg->d_in_refl, refl, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, st));
      refl = vg->d_in_refl;
    }
    if (amb) {
      VG_CK(cudaMemcpyAsync(vg->d_in_amb, amb, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, st));
      amb = vg->d_in_amb;
    }
  }
  // outputs: the caller's device buffers, or device staging for host ones
  float4* out = out_on_device ? (float4*)out_xyzi : vg->d_out;
  float* o_refl = refl && out_reflectivity ? (out_on_device ? out_reflectivity : vg->d_out_refl) : nullptr;
  float* o_amb = amb && out_ambient ? (out_on_device ? out_ambient : vg->d_out_amb) : nullptr;

  const float inv[3] = {1.0f / leaf[0], 1.0f / leaf[1], 1.0f / leaf[2]};
  const uint32_t tiles = tiles_for(n);
  VgState* s = vg->d_state;
  int launches = 0;
  VG_CK(cudaMemsetAsync(s, 0, sizeof(VgState), st));
  const int bounds_blocks = (int)std::min<uint32_t>((n + kVgThreads - 1) / kVgThreads, (uint32_t)kBoundsBlocks);
  launch_kernel(k_vg_bounds, dim3(bounds_blocks), dim3(kVgThreads), 0, st, pts, n, vg->part, s, inv[0], inv[1], inv[2]);
  launches += 1;

  const PointKeys pk{pts, n, {inv[0], inv[1], inv[2]}};
  const bool self_radix = tiles <= kSelfRadixTiles;
  launch_kernel(k_radix_count, dim3(tiles), dim3(kVgThreads), 0, st, pk, s, vg->counts[0], vg->counts[1]);
  launches += 1;
  for (int pass = 0; pass < 4; ++pass) {
    uint32_t *cnt = vg->counts[pass % 3], *nxt = vg->counts[(pass + 1) % 3], *clr = vg->counts[(pass + 2) % 3];
    if (!self_radix) {
      launch_kernel(k_radix_scan, dim3(kBins / 32), dim3(kRadixScanThreads), 0, st, s, pass, cnt, tiles, vg->offsets,
                    vg->digit_total);
      launches += 1;
    }
    launch_kernel(pass ? k_radix_scatter<false> : k_radix_scatter<true>, dim3(tiles), dim3(kVgThreads), 0, st,
                  vg->keys[(pass & 1) ^ 1], vg->vals[(pass & 1) ^ 1], vg->keys[pass & 1], vg->vals[pass & 1], pk, s, pass,
                  cnt, self_radix ? nullptr : vg->offsets, vg->digit_total, nxt, clr);
    launches += 1;
  }

  // flagged items of the tiles to their place: counts, their scan beyond kSelfScanTiles, the scatter
  auto compact = [&](auto op, uint32_t* total) {
    launch_kernel(k_flag_count<decltype(op)>, dim3(tiles), dim3(kVgThreads), 0, st, op, vg->tile_counts);
    const bool self = tiles <= kSelfScanTiles;
    if (!self) launch_kernel(k_scan_words, dim3(1), dim3(kScanThreads), 0, st, vg->tile_counts, tiles, vg->tile_counts + vg->max_tiles, total);
    launch_kernel(k_flag_scatter<decltype(op)>, dim3(tiles), dim3(kVgThreads), 0, st, op, vg->tile_counts,
                  self ? nullptr : vg->tile_counts + vg->max_tiles, total);
    launches += self ? 2 : 3;
  };
  compact(HeadOp{vg->keys[0], vg->keys[1], s, vg->leaf_start}, &s->n_leaves);

  const bool direct = min_points_per_voxel <= 1;
  const uint32_t leaf_blocks = std::min<uint32_t>((n + kVgWarps - 1) / kVgWarps, 148u * 16u);
  launch_kernel(k_vg_centroid, dim3(leaf_blocks), dim3(kVgThreads), 0, st, pts, o_refl ? refl : nullptr, o_amb ? amb : nullptr,
                                                    vg->vals[0], vg->vals[1], vg->leaf_start, s, direct ? out : vg->d_tmp,
                                                    direct ? o_refl : (o_refl ? vg->d_tmp_refl : nullptr),
                                                    direct ? o_amb : (o_amb ? vg->d_tmp_amb : nullptr), direct ? 1 : 0);
  launches += 1;
  if (!direct) {
    compact(KeepOp{vg->leaf_start, s, min_points_per_voxel, vg->d_tmp, vg->d_tmp_refl, vg->d_tmp_amb, out, o_refl, o_amb},
            &s->n_out);
  }
  count_launches(launches);
  VG_CK(cudaGetLastError());
  VG_CK(cudaMemcpyAsync(vg->h_state, s, sizeof(VgState), cudaMemcpyDeviceToHost, st));
  VG_CK(cudaStreamSynchronize(st));
  const VgState& hs = *vg->h_state;
  if (hs.status == kVgRange) {
    vg->err = "leaf indices leave the int32 / 32-bit cell range for this leaf size";
    return PHGPU_ERR_LIMIT;
  }
  const cudaMemcpyKind to_out = out_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
  if (hs.status == kVgOverflow) {
    // the reference's "Integer indices would overflow" branch: output = input
    VG_CK(cudaMemcpyAsync(out_xyzi, pts, (size_t)n * sizeof(float4), to_out, st));
    if (o_refl) VG_CK(cudaMemcpyAsync(out_reflectivity, refl, (size_t)n * sizeof(float), to_out, st));
    if (o_amb) VG_CK(cudaMemcpyAsync(out_ambient, amb, (size_t)n * sizeof(float), to_out, st));
    VG_CK(cudaStreamSynchronize(st));
    *n_out = n;
    return PHGPU_OK;
  }
  const uint32_t m = hs.status == kVgOk ? hs.n_out : 0u;
  if (!out_on_device && m) {
    VG_CK(cudaMemcpyAsync(out_xyzi, out, (size_t)m * sizeof(float4), cudaMemcpyDeviceToHost, st));
    if (o_refl) VG_CK(cudaMemcpyAsync(out_reflectivity, o_refl, (size_t)m * sizeof(float), cudaMemcpyDeviceToHost, st));
    if (o_amb) VG_CK(cudaMemcpyAsync(out_ambient, o_amb, (size_t)m * sizeof(float), cudaMemcpyDeviceToHost, st));
    VG_CK(cudaStreamSynchronize(st));
  }
  *n_out = m;
  return PHGPU_OK;
}
