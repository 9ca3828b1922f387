// Translation stage: voxelisation, 3-D real FFTs, fused cross power, inverse
// real FFT and argmax.
//
// Reference behaviour:
//  * PhaseAligner::discretizePointcloud (phaser_core/src/backend/alignment/
//    phase-aligner.cc:71-131) with igl::histc (phaser_core/include/igl/
//    histc.cpp:34-73): float edges, binary search, -1 for out-of-range
//    coordinates, lin = uint32(bx)*N + uint32(by) + N*N*uint32(bz) with uint32
//    wrap-around and the `lin > N^3` guard; per-voxel means of intensity,
//    range (sqrtf of the float squared norm), reflectivity, ambient; empty
//    voxels 0.  Channel order {intensity, range, reflectivity, ambient}.
//  * SpatialCorrelationLaplace::correlateSignals (phaser_core/src/backend/
//    correlation/spatial-correlation-laplace.cc:17-89) with
//    SpatialCorrelation::complexMulSeq / c2r (spatial-correlation.cc:52-161):
//    r2c_3d over [z][x][y] (y halved), positional pyramid fusion on the
//    FFT-shifted linear index of the N*N*(N/2+1) half spectrum, C = F conj(G),
//    unnormalised c2r_3d (complex inverse over z and x, then the real
//    half-complex inverse over y, which reads only the real part of the DC and
//    Nyquist terms), first-occurrence argmax of the signed output.
//
// Passes (FP32): sums along y of the rows' occupied voxels (an FFT for grids
// handed in by the host); forward along x of the z slabs that hold a voxel; forward along z of all channels of both clouds
// per (x, ky tile) + fusion + cross power + inverse along z; inverse along x;
// complex-to-real along y with argmax.  Forward transforms leave x and z in
// digit-reversed order; the inverse transforms consume that order directly.
#include <algorithm>

#include "fft_pass.cuh"
#include "kernels.h"

namespace phgpu {

// histc's bin (igl/histc.cpp:34-73): -1 outside [E[0], E[N-1]], else the
// result of its binary search over the sorted edges -- the largest l <= N-2
// with E[l] <= x, or N-1 when x == E[N-1] (NaN: N-2, where the search ends;
// N = 1: 0).
// The search is replaced by a start at the linear estimate (x - E[0]) * inv,
// inv = (N-1) / (E[N-1] - E[0]), corrected by exact comparisons with the
// edges, which gives the same bin in one or two loads instead of log2 N.
__device__ __forceinline__ int histc_bin(float x, const float* __restrict__ E, int N, float e0, float e1,
                                         float inv) {
  if (x < e0 || x > e1) return -1;
  if (N < 2) return 0;
  if (x != x) return N - 2;
  int l = (int)((x - e0) * inv);
  l = min(max(l, 0), N - 2);
  while (l > 0 && x < E[l]) --l;
  while (l < N - 2 && x >= E[l + 1]) ++l;
  return (x == E[l + 1]) ? l + 1 : l;
}

// A voxel's channel sums lie together (one 16-byte vector atomic per update,
// one load per voxel later), the point counts in an array of their own (which
// the row sums scan).  Neighbouring points of a scan mostly share a voxel --
// near the sensor dozens do, and their atomics on one address serialised -- so a
// warp sums each run of equal voxels with shuffles and the run's last lane
// issues the atomics (131072 points, N = 200: 30 -> 10.8 us).
__global__ void k_voxelize(const __grid_constant__ VoxelArgs a) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int np = a.n_dev ? (int)*a.n_dev : a.n_points;
  const int lane = threadIdx.x & 31;
  if (i - lane >= np) return;  // whole warps
  uint32_t lin = 0xffffffffu;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < np) {
    const float4 p = a.xyzi[i];
    float x = p.x, y = p.y, z = p.z;
    if (a.has_T || a.T_dev) {
      // PCL 1.8 transformPointCloud order ((T0 x + T1 y) + T2 z) + T3
      float Tl[12];
      if (a.T_dev) {
#pragma unroll
        for (int k = 0; k < 12; ++k) Tl[k] = __ldg(&a.T_dev[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 12; ++k) Tl[k] = a.T[k];
      }
      const float* T = Tl;
      const float nx = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(T[0], x), __fmul_rn(T[1], y)), __fmul_rn(T[2], z)), T[3]);
      const float ny = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(T[4], x), __fmul_rn(T[5], y)), __fmul_rn(T[6], z)), T[7]);
      const float nz = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(T[8], x), __fmul_rn(T[9], y)), __fmul_rn(T[10], z)), T[11]);
      x = nx;
      y = ny;
      z = nz;
    }
    const uint32_t N = (uint32_t)a.N;
    const float e0 = __ldg(&a.edges[0]), e1 = __ldg(&a.edges[a.N - 1]);
    const float inv = a.N > 1 ? (float)(a.N - 1) / (e1 - e0) : 0.0f;
    const uint32_t bx = (uint32_t)histc_bin(x, a.edges, a.N, e0, e1, inv);
    const uint32_t by = (uint32_t)histc_bin(y, a.edges, a.N, e0, e1, inv);
    const uint32_t bz = (uint32_t)histc_bin(z, a.edges, a.N, e0, e1, inv);
    lin = (bx * N + by) + (N * N * bz);
    if (lin >= N * N * N) lin = 0xffffffffu;
    if (a.lin_out) a.lin_out[i] = lin;
    if (lin != 0xffffffffu) {
      v.x = p.w;
      v.y = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
      if (a.n_data_ch > 2 && a.refl) v.z = a.refl[i];
      if (a.n_data_ch > 3 && a.amb) v.w = a.amb[i];
    }
  }
  // runs of equal voxels: sums up to each lane from its run's first lane
  const uint32_t prev = __shfl_up_sync(0xffffffffu, lin, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || lin != prev);
  const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
  if (heads != 0xffffffffu) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float ux = __shfl_up_sync(0xffffffffu, v.x, o), uy = __shfl_up_sync(0xffffffffu, v.y, o);
      const bool add = lane - o >= first;
      v.x += add ? ux : 0.f;
      v.y += add ? uy : 0.f;
      if (a.n_data_ch > 2) {
        const float uz = __shfl_up_sync(0xffffffffu, v.z, o);
        v.z += add ? uz : 0.f;
      }
      if (a.n_data_ch > 3) {
        const float uw = __shfl_up_sync(0xffffffffu, v.w, o);
        v.w += add ? uw : 0.f;
      }
    }
  }
  const bool last = lane == 31 || ((heads >> (lane + 1)) & 1u);
  if (!last || lin == 0xffffffffu) return;
  // the row of lin, not (bz, bx): an out-of-range bin (-1) wraps into another row
  if (a.rowlive) a.rowlive[lin / (uint32_t)a.N] = 1;
  if (a.n_data_ch > 2)
    atomicAdd(&a.sums[lin], v);
  else
    atomicAdd(reinterpret_cast<float2*>(&a.sums[lin]), make_float2(v.x, v.y));
  atomicAdd(&a.counts[lin], (float)(lane - first + 1));
}

cudaError_t launch_voxelize(const VoxelArgs& a, cudaStream_t st) {
  if (a.n_points > 0) {
    launch_kernel(k_voxelize, dim3((a.n_points + 255) / 256), dim3(256), 0, st, a);
    count_launches(1);
  }
  return cudaGetLastError();
}

// Zeroes what the voxelisation that left these indices wrote.
__global__ void k_clear_voxels(const uint32_t* __restrict__ lin, int n_points, float4* __restrict__ sums,
                               float* __restrict__ counts, uint8_t* __restrict__ rowlive, int N) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_points) return;
  const uint32_t l = lin[i];
  if (l == 0xffffffffu || (i > 0 && lin[i - 1] == l)) return;
  sums[l] = make_float4(0.f, 0.f, 0.f, 0.f);
  counts[l] = 0.f;
  rowlive[l / (uint32_t)N] = 0;
}

// Zeroes the rows that hold a point, a warp per row.
constexpr int kClearRowWarps = 8;
__global__ void __launch_bounds__(kClearRowWarps * 32) k_clear_rows(int N, float4* __restrict__ sums,
                                                                    float* __restrict__ counts,
                                                                    uint8_t* __restrict__ rowlive) {
  chain_begin();
  const int row = blockIdx.x * kClearRowWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= N * N || !rowlive[row]) return;
  const size_t base = (size_t)row * N;
  for (int y = lane; y < N; y += 32) {
    sums[base + y] = make_float4(0.f, 0.f, 0.f, 0.f);
    counts[base + y] = 0.f;
  }
  __syncwarp();
  if (lane == 0) rowlive[row] = 0;
}

// Clears voxel by voxel while the points are few beside the grid: a scan of
// 131 k points takes 2 us so at any N, where a clear of the whole grid takes 25 us
// at N = 200 and 365 at N = 512.  Its stores are scattered, though, and a cloud
// that fills the grid pays one for every point: from an eighth of the voxels on
// the live rows are cleared whole (a voxelisation of 1 M points spread evenly
// over N = 64: 362 us by points, 191 so; N = 100: 218 and 121; N = 200, an eighth,
// 122 and 95; a scan of 131 k points 23 either way at N = 64 and 100).
cudaError_t launch_clear_voxels(const uint32_t* lin, int n_points, float4* sums, float* counts, uint8_t* rowlive, int N,
                                cudaStream_t st) {
  if (n_points <= 0) return cudaGetLastError();
  if ((size_t)n_points < (size_t)N * N * N / 8)
    launch_kernel(k_clear_voxels, dim3((n_points + 255) / 256), dim3(256), 0, st, lin, n_points, sums, counts, rowlive, N);
  else
    launch_kernel(k_clear_rows, dim3((N * N + kClearRowWarps - 1) / kClearRowWarps), dim3(kClearRowWarps * 32), 0, st, N,
                  sums, counts, rowlive);
  count_launches(1);
  return cudaGetLastError();
}

constexpr int kMaxVoxels = 1024;  // longest transform

// ---------------------------------------------------------------- rows of scans (y)
// A scan occupies a few voxels per row (N = 200 over a 20 m cube: three to
// five of 200), so a row's transform along y is summed directly from them,
//   X[ky] = sum_v mean_v exp(-2 pi i ky y_v / N),
// instead of an FFT over every row that holds a point: per voxel and 32
// frequencies one table twiddle (its index, ky y mod N, is exact) and one
// packed multiply-add per channel.  Rows without a point are neither read nor
// written: the x transform takes them as zero.
//
// Block: 16 rows (fewer on small grids, scan_rows_block) of one z-slab; a warp
// takes a live row, gathers its occupied voxels in order (counts, then every
// channel's sums, all loads of 256 voxels in flight) into shared memory and gives
// each lane up to four frequencies at a time.  Small blocks spread a slab full of long rows (a floor
// seen level) over many SMs.  With `clear` the voxels and row flags are zeroed
// on the way, so a grid that is only transformed needs no memset and no
// separate pass before its next voxelisation.  With the x pass behind it a side
// of an N = 200 room takes 39 us (whole slabs at one block an SM: 43 to 65) and
// of an N = 512 one 285 (dense rows and columns: some 1450).
constexpr int kRowsWarps = 4;
// One running sum over a row rounds in proportion to the root of its voxels:
// from some twenty on it is further off than an FFT (a full row of 512: 3.9e-7
// against 0.9e-7, relative L2; of 16 voxels 0.7e-7 against 0.8e-7).  Rows of more
// than kShortRow voxels are summed in parts: sums of 8 voxels, of 8 such sums and
// then over the row stay below the FFT's error at every length and occupancy
// (0.9e-7 there).  Sums beyond the first 64 voxels are added to the stored ones: no
// third set of registers.
constexpr int kShortRow = 16;
constexpr int kPartSum = 8;
constexpr int kRunSum = 64;

// A row of many voxels takes an FFT after all: a real transform of n points as
// a complex one of n / 2 (even and odd columns as real and imaginary parts) per
// channel, by the warp that gathered the row, where n / 2 has a plan of
// register radices (n is even, no prime above 7).  A voxel's sum costs every
// frequency an addition, the FFT costs the same whatever the row holds.  Over
// grids full of such rows they meet at 12 (N = 64) to 30 voxels, but among a
// scan's rows (four to six voxels) a single one that takes the FFT's stages in turn
// is the last to finish: with 16 voxels for the limit a side of some N = 200 rooms
// takes 2 to 3 us more, with 40 none.  The correlation of two full grids took 107 us
// summed at N = 64 and now 73, 376 and 211 at N = 128, 1370 and 515 at N = 200, 4518
// and 1395 at N = 256.
static int dense_row_limit(int N) { return std::min(std::max(N / 5, 16), 40); }

struct ScanRowArgs {
  int N, rows_block;
  float4* sums;         // [N^3] channel sums
  float* counts;        // [N^3] points
  const float2* tw;     // N twiddles
  uint8_t* rowlive;     // [N (z)][N (x)] rows that hold a point
  uint8_t* rowmask;     // [N][N]: the flags again, kept for the x transform
  float2* spec;         // [channel][z][x][H2p]
  size_t spec_stride;
  int clear;
  int dense;            // rows of more voxels are transformed
  FftPlan half;         // length N / 2 for them
  const uint16_t* half_pos;  // [N / 2] position of each of its frequencies
};

// Channel c of a row as N / 2 complex values in place of its [N] float4 means:
// element i is columns 2 i and 2 i + 1.
struct EvenOddCursor {
  float* p;
  int es;
  __device__ __forceinline__ float2 operator()(int, int j) const { return make_float2(p[j * es], p[j * es + 4]); }
  __device__ __forceinline__ void operator()(int, int j, float2 v) const {
    p[j * es] = v.x;
    p[j * es + 4] = v.y;
  }
};

// Transforms one dense row by the calling warp.  s_val, s_y: the row's cnt
// occupied columns in order; occ: lane w's bits are columns 32 w .. 32 w + 31.
template <int CC>
__device__ __noinline__ void dense_row(const ScanRowArgs& a, float4* s_val, const uint16_t* s_y,
                                          const float2* __restrict__ s_tw, unsigned occ, int cnt, int lane, float2* out) {
  const int n = a.N, nh = n / 2;
  // the list spread to its columns, last entries first: a column is never before its place in the list
  for (int e0 = (cnt - 1) & ~31; e0 >= 0; e0 -= 32) {
    const bool ok = e0 + lane < cnt;
    const float4 v = ok ? s_val[e0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int y = ok ? s_y[e0 + lane] : 0;
    __syncwarp();
    if (ok) s_val[y] = v;
    __syncwarp();
  }
  for (int w = 0; 32 * w < n; ++w) {
    const unsigned m = __shfl_sync(0xffffffffu, occ, w);
    if (32 * w + lane < n && !((m >> lane) & 1u)) s_val[32 * w + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncwarp();
  float* f = reinterpret_cast<float*>(s_val);
  auto at = [=](int, int t, int i, int m) { return EvenOddCursor{f + 8 * i + t, 8 * m}; };
  const PassMap map{1, CC == 1 ? 0 : (CC == 2 ? 1 : 2)};
  for (int s = 0; s < a.half.nstage; ++s) {
    pass_stage_rt<false, 1>(a.half, s, map, lane, 32, at, at);
    __syncwarp();
  }
  // X[k] = (Z[k] + conj Z[-k]) / 2 + w^k (Z[k] - conj Z[-k]) / 2i
  for (int k = lane; k < nh; k += 32) {
    const int p0 = 2 * __ldg(a.half_pos + k), p1 = 2 * __ldg(a.half_pos + (k == 0 ? 0 : nh - k));
    const float4 ur = s_val[p0], ui = s_val[p0 + 1], vr = s_val[p1], vi = s_val[p1 + 1];
    const float2 w = s_tw[k];
    auto bin = [&](int c, float xr, float xi, float yr, float yi) {
      if (c >= CC) return;
      float2* o = out + c * a.spec_stride + k;
      *o = cadd(make_float2(0.5f * (xr + yr), 0.5f * (xi - yi)), cmul(w, make_float2(0.5f * (xi + yi), -0.5f * (xr - yr))));
      if (k == 0) o[nh] = make_float2(xr - xi, 0.f);
    };
    bin(0, ur.x, ui.x, vr.x, vi.x);
    bin(1, ur.y, ui.y, vr.y, vi.y);
    bin(2, ur.z, ui.z, vr.z, vi.z);
    bin(3, ur.w, ui.w, vr.w, vi.w);
  }
}

// Adds a voxel to the sums for frequencies k + 32 i.
template <int CC, int Q>
__device__ __forceinline__ void add_voxel(float2 (&acc)[CC][Q], float4 w, uint32_t y, const float2* s_tw, int n,
                                          uint32_t mul, int k) {
  const float ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const uint32_t p = (uint32_t)(k + 32 * i) * y;
    const float2 t = s_tw[p - __umulhi(p, mul) * (uint32_t)n];
#pragma unroll
    for (int ch = 0; ch < CC; ++ch) acc[ch][i] = __ffma2_rn(make_float2(ws[ch], ws[ch]), t, acc[ch][i]);
  }
}
template <int CC, int Q>
__device__ __forceinline__ void zero_sums(float2 (&acc)[CC][Q]) {
#pragma unroll
  for (int ch = 0; ch < CC; ++ch)
#pragma unroll
    for (int i = 0; i < Q; ++i) acc[ch][i] = make_float2(0.f, 0.f);
}
template <int CC, int Q>
__device__ __forceinline__ void store_sums(const float2 (&acc)[CC][Q], float2* out, size_t stride, int k, int H2,
                                           bool more) {
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int ky = k + 32 * i;
    if (ky < H2) {
#pragma unroll
      for (int ch = 0; ch < CC; ++ch) {
        float2* o = out + ch * stride + ky;
        *o = more ? cadd(*o, acc[ch][i]) : acc[ch][i];
      }
    }
  }
}

// The sums of a row in parts.
template <int CC>
__device__ __noinline__ void part_row(const ScanRowArgs& a, const float4* s_val, const uint16_t* s_y, const float2* s_tw,
                                      int cnt, int lane, float2* out) {
  const int n = a.N, H2 = n / 2 + 1;
  const uint32_t mul = fast_div_mul(n);
  constexpr int Q = 2;  // two sets of sums: fewer frequencies at a time, for the caller's registers
  for (int k = lane; k < H2 + lane; k += 32 * Q) {
    for (int e = 0; e < cnt;) {
      float2 sum[CC][Q];
      zero_sums(sum);
      const int stored = e, run = min(cnt, e + kRunSum);
      for (; e < run; e = min(run, e + kPartSum)) {
        float2 part[CC][Q];
        zero_sums(part);
#pragma unroll
        for (int u = 0; u < kPartSum; ++u) {  // all the part's loads in flight; past the end a zero at column 0
          const bool in = e + u < run;
          add_voxel(part, in ? s_val[e + u] : make_float4(0.f, 0.f, 0.f, 0.f), in ? s_y[e + u] : 0, s_tw, n, mul, k);
        }
#pragma unroll
        for (int ch = 0; ch < CC; ++ch)
#pragma unroll
          for (int i = 0; i < Q; ++i) sum[ch][i] = cadd(sum[ch][i], part[ch][i]);
      }
      store_sums(sum, out, a.spec_stride, k, H2, stored > 0);
    }
  }
}

// Shared memory: N twiddles, then per warp N float4 (means) and N uint16 (y).
static size_t scan_rows_smem(int N) { return (size_t)N * (8 + kRowsWarps * 18) + 16 * (kRowsWarps + 1); }

// Rows of a block: 16, halved down to one a warp while the blocks are fewer
// than twice those resident (six an SM), so a slab of dense rows does not wait
// for one warp's four in turn (the correlation of two full grids with 16 rows: N =
// 64 87 us, with 4 75; N = 128 215, with 8 202; with 4 rows at N = 200 a scan's
// empty blocks cost 11 us).
static int scan_rows_block(int N) {
  int rows = 16;
  while (rows > kRowsWarps && N * ((N + rows - 1) / rows) < 2 * 6 * 148) rows /= 2;
  return rows;
}

template <int CC>
__global__ void __launch_bounds__(kRowsWarps * 32) k_scan_rows(const __grid_constant__ ScanRowArgs a) {
  chain_begin();
  extern __shared__ __align__(16) float4 s_mem[];
  constexpr int U = 8;
  const int n = a.N, H2 = n / 2 + 1, H2p = spatial_h2p(n);
  const int z = blockIdx.x, x0 = blockIdx.y * a.rows_block, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool mine = lane < a.rows_block && x0 + lane < n;
  const bool live_l = mine && a.rowlive[(size_t)z * n + x0 + lane];
  const unsigned live = __ballot_sync(0xffffffffu, live_l);  // every warp: the block's rows
  if (warp == 0 && mine) a.rowmask[(size_t)z * n + x0 + lane] = live_l ? 1 : 0;
  if (!live) return;
  float4* s_val = s_mem + (size_t)warp * n;
  float2* s_tw = reinterpret_cast<float2*>(s_mem + (size_t)kRowsWarps * n);
  uint16_t* s_y = reinterpret_cast<uint16_t*>(s_tw + n) + (size_t)warp * n;
  for (int i = threadIdx.x; i < n; i += kRowsWarps * 32) s_tw[i] = __ldg(a.tw + i);
  __syncthreads();
  if (a.clear && warp == 0 && live_l) a.rowlive[(size_t)z * n + x0 + lane] = 0;
  const uint32_t mul = fast_div_mul(n);
  int seen = 0;
  for (unsigned todo = live; todo; todo &= todo - 1) {
    if ((seen++ & (kRowsWarps - 1)) != warp) continue;
    const size_t row = (size_t)z * n + x0 + __ffs(todo) - 1;
    float* c = a.counts + row * n;
    float4* g = a.sums + row * n;
    int cnt = 0;
    unsigned bits = 0;  // occupied columns 32 lane .. 32 lane + 31
    for (int y0 = 0; y0 < n; y0 += 32 * U) {
      float q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) q[u] = y0 + 32 * u + lane < n ? c[y0 + 32 * u + lane] : 0.f;
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = q[u] > 0.f ? g[y0 + 32 * u + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool occ = q[u] > 0.f;
        const unsigned m = __ballot_sync(0xffffffffu, occ);
        if (lane == y0 / 32 + u) bits = m;
        if (occ) {
          const int y = y0 + 32 * u + lane, at = cnt + __popc(m & ((1u << lane) - 1u));
          const float inv = __frcp_rn(q[u]);  // mean = sum * (1 / count)
          s_y[at] = (uint16_t)y;
          s_val[at] = make_float4(v[u].x * inv, v[u].y * inv, v[u].z * inv, v[u].w * inv);
          if (a.clear) {
            c[y] = 0.f;
            g[y] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        cnt += __popc(m);
      }
    }
    __syncwarp();
    float2* out = a.spec + row * H2p;
    if (cnt > kShortRow) {
      if (cnt > a.dense)
        dense_row<CC>(a, s_val, s_y, s_tw, bits, cnt, lane, out);
      else
        part_row<CC>(a, s_val, s_y, s_tw, cnt, lane, out);
    } else {
      constexpr int Q = 4;
      for (int k0 = 0; k0 < H2; k0 += 32 * Q) {
        float2 sum[CC][Q];
        zero_sums(sum);
#pragma unroll 2
        for (int e = 0; e < cnt; ++e) add_voxel(sum, s_val[e], s_y[e], s_tw, n, mul, k0 + lane);
        store_sums(sum, out, a.spec_stride, k0 + lane, H2, false);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- rows (y)
constexpr int kRowPairs = 16;      // row pairs per block of the forward row transforms
constexpr int kInvPairs = 16;      // row pairs per block of the inverse row transforms
// Row stride in shared memory: odd, so threads that take one element of
// neighbouring rows touch different banks.
__host__ __device__ constexpr int row_stride(int n) { return n | 1; }

// Real transforms along y of every row of a grid of values (grids handed in
// by the host; voxelised clouds take the list of occupied voxels instead).
// Rows are transformed two at a time as the real and imaginary parts of one
// complex row, Z = X0 + i X1, separated afterwards by
//   X0[k] = (Z[k] + conj Z[-k]) / 2,   X1[k] = (Z[k] - conj Z[-k]) / 2i.
template <int NF>
__global__ void __launch_bounds__(320, NF > 0 ? 3 : 2) k_r2c_rows(int N, const float* __restrict__ grids,
                                                                  size_t grid_stride, float2* __restrict__ specs,
                                                                  size_t spec_stride,
                                                                  const __grid_constant__ FftPlan plan) {
  chain_begin();
  extern __shared__ __align__(16) float2 rows[];  // [kRowPairs][st] | float4 cs[] (runtime plans)
  __shared__ short s_pos[kMaxVoxels];
  const int n = NF > 0 ? NF : N;
  const int H2 = n / 2 + 1, H2p = spatial_h2p(n), st = row_stride(n);
  const int tid = threadIdx.x, nthr = blockDim.x;
  float4* cs = reinterpret_cast<float4*>(rows + (size_t)kRowPairs * st);
  const int r0 = blockIdx.x * 2 * kRowPairs;
  const int rows_here = min(2 * kRowPairs, n * n - r0), np = (rows_here + 1) / 2;
  const int lwp = 32 - __clz(np - 1);  // columns of the shared stages: the next power of two
  const float* grid = grids + (size_t)blockIdx.y * grid_stride + (size_t)r0 * n;
  float2* spec = specs + (size_t)blockIdx.y * spec_stride + (size_t)r0 * H2p;
  for (int k = tid; k < n; k += nthr) s_pos[k] = (short)freq2pos<NF>(k, plan);
  auto at = [=](int g, int t, int i, int m) { return SmemCursor{rows + (g + t) * st + i, m, 0}; };
  auto ld = [=](int g, int t, int i, int m) {
    const float* p = grid + 2 * (g + t) * n + i;
    const bool two = 2 * (g + t) + 1 < rows_here;
    return [=](int, int j) { return make_float2(__ldg(p + j * m), two ? __ldg(p + n + j * m) : 0.f); };
  };
  if constexpr (NF > 0) {
    pass_ct<NF, false, 1, false, 0, 1>(PassMap{np, 0}, plan.tw, tid, nthr, ld, at, at);
    __syncthreads();
    pass_ct<NF, false, 1, true, 1, -1>(PassMap{1, lwp}, plan.tw, tid, nthr, at, at, at);
  } else {
    pass_rt<false, 1, false>(plan, PassMap{np, 0}, PassMap{1, lwp}, PassMap{1, lwp}, cs, tid, nthr, ld, at, at);
  }
  __syncthreads();
  // separate the rows: one warp per row
  for (int rr = tid >> 5; rr < rows_here; rr += nthr >> 5) {
    const float2* Z = rows + (rr >> 1) * st;
    for (int ky = tid & 31; ky < H2; ky += 32) {
      const float2 u = Z[s_pos[ky]], v = Z[s_pos[ky == 0 ? 0 : n - ky]];
      spec[rr * H2p + ky] = (rr & 1) ? make_float2(0.5f * (u.y + v.y), -0.5f * (u.x - v.x))   // (u - conj v) / 2i
                                     : make_float2(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));  // (u + conj v) / 2
    }
  }
}

// Real inverse over y of 2 kInvPairs consecutive rows with first-occurrence
// argmax.  A half-complex inverse reads only the real parts of the ky = 0 and
// ky = N/2 terms, so each row is made exactly Hermitian that way, and rows are
// inverted two at a time as Z = X0 + i X1 (output x0 = Re, x1 = Im).  The
// first inverse stage reads the spectrum directly: the R positions it joins
// hold the frequencies b, b + n/R, ..., so neighbouring threads (b) read
// neighbouring frequencies; the last stage's outputs go to the argmax without
// passing through shared memory.
template <int NF>
__global__ void __launch_bounds__(320, NF > 0 ? 3 : 2) k_c2r_rows(int N, const float2* __restrict__ cspec, const __grid_constant__ FftPlan plan,
                                                  unsigned long long* __restrict__ argmax, float* __restrict__ volume,
                                                  uint32_t limit) {
  chain_begin();
  extern __shared__ __align__(16) float2 rows[];  // [kInvPairs][st] | float4 cs[] | int pos[n] (runtime plans)
  const int n = NF > 0 ? NF : N;
  const int H2p = spatial_h2p(n), st = row_stride(n);
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int nrows = n * n;
  const int r0 = blockIdx.x * 2 * kInvPairs;
  const int np = min(kInvPairs, (nrows - r0 + 1) / 2);
  const int lwp = 32 - __clz(np - 1);
  auto at = [&](int g, int t, int i, int m) { return SmemCursor{rows + (g + t) * st + i, m, 0}; };
  // Z at frequency k (mirrored: read at n - k) of a row pair, edge: k = 0 or 2 k = n
  auto zval = [&](const float2* ca, int k, bool mir, bool edge, bool two) -> float2 {
    ca += mir ? n - k : k;
    float2 u = __ldg(ca), v = two ? __ldg(ca + H2p) : make_float2(0.f, 0.f);
    if (edge) u.y = v.y = 0.f;
    return mir ? make_float2(u.x + v.y, v.x - u.y)   // conj u + i conj v
               : make_float2(u.x - v.y, u.y + v.x);  // u + i v
  };
  // per thread: the first index of its largest value (NaN compares false; a
  // thread that saw nothing else keeps its first value)
  float bv = -INFINITY, fv = 0.f;
  uint32_t bi = 0xffffffffu, fi = 0xffffffffu;
  const bool bounded = limit < (uint32_t)nrows * (uint32_t)n;
  auto take = [&](float v, uint32_t idx) {
    if (bounded && idx >= limit) return;
    if (fi == 0xffffffffu) {
      fi = idx;
      fv = v;
    }
    if (v > bv || (v == bv && idx < bi)) {
      bv = v;
      bi = idx;
    }
  };
  auto sv = [&](int g, int t, int y, int m) {
    const uint32_t idx = (uint32_t)((r0 + 2 * (g + t)) * n + y);
    const bool two = r0 + 2 * (g + t) + 1 < nrows;
    return [=, &take](int, int j, float2 v) {
      take(v.x, idx + j * m);
      if (two) take(v.y, idx + j * m + n);
      if (volume) {
        volume[idx + j * m] = v.x;
        if (two) volume[idx + j * m + n] = v.y;
      }
    };
  };
  if constexpr (NF > 0) {
    constexpr int R = FixedFft<NF>::r[FixedFft<NF>::count - 1];
    constexpr int nb = NF / R;
    for (int it = tid; it < np * nb; it += nthr) {
      const int pk = it / nb, b = it - pk * nb;
      const float2* ca = cspec + (size_t)(r0 + 2 * pk) * H2p;
      float2 x[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        // NF is even: whole runs of b lie on one side of the Nyquist term
        const bool below = 2 * (i * nb + nb - 1) < NF, above = 2 * i * nb > NF;
        const int k = b + i * nb;
        const bool mir = above || (!below && 2 * k > NF);
        x[i] = zval(ca, k, mir, (i == 0 && b == 0) || (!below && !above && 2 * k == NF), true);
      }
      dft_small<R, true>(x);
      float2* d = rows + pk * st + fixed_freq2pos<NF>(b);
#pragma unroll
      for (int i = 0; i < R; ++i) d[i] = x[i];
    }
    __syncthreads();
    constexpr int cnt = FixedFft<NF>::count;
    pass_ct<NF, true, 1, true, 1, cnt - 1>(PassMap{1, lwp}, plan.tw, tid, nthr, at, at, sv);
    if constexpr (cnt > 2) __syncthreads();
    if (volume || bounded) {
      pass_ct<NF, true, 1, false, cnt - 1, -1>(PassMap{np, 0}, plan.tw, tid, nthr, at, at, sv);
    } else {
      // A thread's items lie in increasing row pairs (nthr >= the butterflies
      // of a row), and an item's values are taken in increasing index: the
      // first of equal values is the one met first.
      constexpr int R0 = FixedFft<NF>::r[0], m = NF / R0;
      static_assert(m <= 128, "a block has at least 128 threads");
      for (int it = tid; it < np * m; it += nthr) {
        const int pk = it / m, j2 = it - pk * m;
        const float2* row = rows + pk * st + j2;
        float2 x[R0];
#pragma unroll
        for (int j = 0; j < R0; ++j) x[j] = row[j * m];
#pragma unroll
        for (int k = 1; k < R0; ++k) x[k] = cmul(x[k], cconj(__ldg(plan.tw + j2 * k)));
        dft_small<R0, true>(x);
        const uint32_t idx = (uint32_t)((r0 + 2 * pk) * NF + j2);
        if (fi == 0xffffffffu) {
          fi = idx;
          fv = x[0].x;
        }
#pragma unroll
        for (int j = 0; j < R0; ++j)
          if (x[j].x > bv) {
            bv = x[j].x;
            bi = idx + j * m;
          }
#pragma unroll
        for (int j = 0; j < R0; ++j)
          if (x[j].y > bv) {
            bv = x[j].y;
            bi = idx + NF + j * m;
          }
      }
    }
  } else {
    float4* cs = reinterpret_cast<float4*>(rows + (size_t)kInvPairs * st);
    int* pos = reinterpret_cast<int*>(cs + kMaxGenericRadix);
    for (int k = tid; k < n; k += nthr) pos[k] = freq2pos<NF>(k, plan);
    __syncthreads();
    for (int pk = tid >> 5; pk < np; pk += nthr >> 5) {
      const float2* ca = cspec + (size_t)(r0 + 2 * pk) * H2p;
      const bool two = r0 + 2 * pk + 1 < nrows;
      for (int k = tid & 31; k < n; k += 32) rows[pk * st + pos[k]] = zval(ca, k, 2 * k > n, k == 0 || 2 * k == n, two);
    }
    __syncthreads();
    pass_rt<true, 1, true>(plan, PassMap{1, lwp}, PassMap{1, lwp}, PassMap{np, 0}, cs, tid, nthr, at, at, sv);
  }
  if (bi == 0xffffffffu) {
    bi = fi;
    bv = fv;
  }
  // + 0: a negative zero orders as zero
  warp_argmax_commit(bi == 0xffffffffu ? 0ull : pack_argmax(bv + 0.0f, bi), argmax);
}

// ---------------------------------------------------------------- columns (x)
struct ColArgs {
  int N;
  float2* spec;  // [channel][z][x][H2p]
  size_t spec_stride;
  const uint8_t* rowmask;  // forward: [N (z)][N (x)] rows that hold a voxel, the others are taken as zero; null: all
  uint8_t* slab_live;      // forward: [N] set to whether any row of the slab holds a voxel
  int write_empty;         // forward: empty slabs are written as zeros (else left alone)
  FftPlan plan;
};

// In-place transform along x of a tile of 2^LW ky columns at one z of CC
// arrays (forward: every channel of a side, which share the row flags, the
// index arithmetic and the twiddles).  Forward: x natural in, digit-reversed
// out; inverse: the reverse.  The first stage reads and the last stage writes
// global memory directly.  Slabs without a voxel are left alone: the z pass
// does not read them.
constexpr int kXThreads = 320;
template <int NF, bool INV, int CC, int LW>
__global__ void __launch_bounds__(kXThreads, NF > 0 ? 4 : 2) k_fft_x(const __grid_constant__ ColArgs a) {
  chain_begin();
  extern __shared__ __align__(16) float2 tile[];  // [CC][n][W] | float4 cs[] (runtime plans) | uint8 live[n]
  __shared__ uint16_t s_mask[(INV || NF == 0) ? 1 : NF / 2];
  constexpr int W = 1 << LW;
  const int n = NF > 0 ? NF : a.N;
  const int H2 = n / 2 + 1, H2p = spatial_h2p(n);
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int z = blockIdx.y, ky0 = blockIdx.x * W, wt = min(W, H2 - ky0);
  const int slot = n * W;
  float4* cs = reinterpret_cast<float4*>(tile + (size_t)CC * slot);
  uint8_t* s_live = reinterpret_cast<uint8_t*>(cs + (NF > 0 ? 0 : kMaxGenericRadix));
  const size_t stride = a.spec_stride;
  if constexpr (!INV) {
    int any = 0;
    for (int x = tid; x < n; x += nthr) {
      const uint8_t f = a.rowmask ? a.rowmask[(size_t)z * n + x] : 1;
      s_live[x] = f;
      any |= f;
    }
    any = __syncthreads_or(any);
    if (blockIdx.x == 0 && tid == 0) a.slab_live[z] = any ? 1 : 0;
    if (!any && !a.write_empty) return;
  }
  float2* base = a.spec + (size_t)z * n * H2p + ky0;
  auto at = [=](int c, int t, int i, int m) { return SmemCursor{tile + c * slot + i * W + t, m * W, slot}; };
  auto sv = [=](int g, int t, int i, int m) {
    float2* p = base + g * stride + i * H2p + t;
    const bool ok = t < wt;
    const int js = m * H2p;
    return [=](int c, int j, float2 v) {
      if (ok) p[c * stride + j * js] = v;
    };
  };
  const PassMap map{1, LW};
  if constexpr (NF > 0 && !INV) {
    // which of the R rows of each first-stage butterfly are live
    constexpr int R = FixedFft<NF>::r[0], m0 = NF / R;
    for (int i = tid; i < m0; i += nthr) {
      unsigned k = 0;
#pragma unroll
      for (int j = 0; j < R; ++j) k |= (s_live[i + j * m0] ? 1u : 0u) << j;
      s_mask[i] = (uint16_t)k;
    }
    __syncthreads();
    const uint16_t* mask = s_mask;
    auto ld = [=](int, int t, int i, int m) {
      const float2* p = base + i * H2p + t;
      const unsigned k = t < wt ? mask[i] : 0u;
      const int js = m * H2p;
      return [=](int c, int j) { return (k >> j) & 1u ? p[c * stride + j * js] : make_float2(0.f, 0.f); };
    };
    pass_ct<NF, false, CC, true, 0, -1>(map, a.plan.tw, tid, nthr, ld, at, sv);
  } else {
    auto ld = [=](int g, int t, int i, int m) {
      const float2* p = base + g * stride + i * H2p + t;
      const bool ok = t < wt;
      const int js = m * H2p;
      const uint8_t* l = s_live + i;
      return [=](int c, int j) {
        bool take = ok;
        if constexpr (!INV) take = take && l[j * m];
        return take ? p[c * stride + j * js] : make_float2(0.f, 0.f);
      };
    };
    if constexpr (NF > 0)
      pass_ct<NF, true, CC, true, 0, -1>(map, a.plan.tw, tid, nthr, ld, at, sv);
    else {
      const PassMap ch{CC, LW};  // the channels as groups of transforms
      pass_rt<INV, 1, false>(a.plan, ch, ch, ch, cs, tid, nthr, ld, at, sv);
    }
  }
}

// ---------------------------------------------------------------- z, fusion
// For one x position (digit-reversed) and a tile of ky: forward z transform of
// all channels of both clouds, channel fusion, cross power and the inverse z
// transform of the product.
//
// The sides follow one another through one set of C channel slots (slot C
// holds the fused target, then the product), so a block of 3 channels keeps
// 4 n W complex values rather than 6, and four blocks fit on an SM at N = 200.
// With a compile-time plan the last forward stage, the fusion and the first
// inverse stage run in registers: the last stage of a forward transform and
// the first of an inverse one join the same R neighbouring positions, so a
// thread transforms its R positions of every channel, keeps the running
// fusion, and hands the product to the inverse butterfly without a shared
// round trip.  Slabs without a point (slab_live) are not read.  Bound by issue,
// barriers and the loads' latency at the two to four blocks an SM that registers
// and slots allow: N = 200 104 -> 85 us, N = 512 1957 -> 1770, N = 201 (prime
// stage) 1065 -> 375.

constexpr int kFuseMixed = 3;  // the rule varies over the run of positions
// The fusion rule of a run of positions [p0, p1] (p1 < p0: it wraps): one
// descent of the levels with both ends, which stops at the first level that
// keeps neither (about two on average).
__device__ __forceinline__ int fusion_op_run(uint32_t p0, uint32_t p1, const FusionBands& b) {
  if (p1 < p0) return kFuseMixed;
  for (int l = 0; l < b.levels; ++l) {
    const uint32_t lb = b.lb[l], eub = b.eub[l], sub = b.sub[l];
    if (p0 >= lb && p1 < eub) {
      p0 -= lb;
      p1 -= lb;
      continue;
    }
    if (p1 < lb || (p0 >= eub && p0 >= sub)) return kFuseMax;
    return p0 >= eub && p1 < sub ? kFuseZero : kFuseMixed;
  }
  return kFuseMean;
}

// Shared-memory element of position i: one extra column group after every
// R_last positions when R_last is even, so the butterflies of neighbouring
// position groups start on different banks.
template <int NF>
__host__ __device__ constexpr int z_pad() {
  if constexpr (NF > 0) {
    constexpr int R = FixedFft<NF>::r[FixedFft<NF>::count - 1];
    return R % 2 == 0 ? R : 0;
  } else {
    return 0;
  }
}
template <int NF>
__host__ __device__ constexpr int z_off(int i) {
  if constexpr (z_pad<NF>() > 0)
    return i + i / z_pad<NF>();
  else
    return i;
}

// Blocks of up to 320 threads, four to an SM (three for plans that end in
// radix 8, whose fused middle stage needs 64 registers); runtime plans two of
// up to 384.
template <int NF>
constexpr int fuse_z_max_threads() {
  return NF > 0 ? 320 : 384;
}
template <int NF>
constexpr int fuse_z_blocks() {
  if constexpr (NF > 0)
    return FixedFft<NF>::r[FixedFft<NF>::count - 1] == 8 ? 3 : 4;
  else
    return 2;
}
// LW >= 0: the tile is 2^LW columns wide; LW < 0: 2^lw_arg.
template <int NF, int CC, int LW>
__global__ void __launch_bounds__(fuse_z_max_threads<NF>(), fuse_z_blocks<NF>()) k_fuse_z(const __grid_constant__ SpatialArgs a, const __grid_constant__ FftPlan plan, int lw_arg) {
  chain_begin();
  // [CC + 1][z_off(n)][W] | float4 cs[] (runtime plans) | int16 kz[n], uint16 mask[n], uint8 live[2 n], op[n], gop[n]
  extern __shared__ __align__(16) float2 tile[];
  __shared__ FusionBands s_bands;
  const int n = NF > 0 ? NF : a.N;
  const int H2 = n / 2 + 1, H2p = spatial_h2p(n);
  const int lw = LW >= 0 ? LW : lw_arg;
  const int W = 1 << lw;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int ky0 = blockIdx.x * W, wt = min(W, H2 - ky0);
  const int xp = blockIdx.y;
  const size_t plane = (size_t)n * n * H2p;
  const int slot = z_off<NF>(n) * W;
  const int kx = pos2freq<NF>(xp, plan);
  const uint32_t nv = (uint32_t)n * n * n;
  float4* cs = reinterpret_cast<float4*>(tile + (size_t)(CC + 1) * slot);
  short* s_kz = reinterpret_cast<short*>(cs + (NF > 0 ? 0 : kMaxGenericRadix));
  uint16_t* s_mask = reinterpret_cast<uint16_t*>(s_kz + n);
  uint8_t* s_live = reinterpret_cast<uint8_t*>(s_mask + n);
  uint8_t *s_op = s_live + 2 * n, *s_gop = s_op + n;
  if (tid == 0) s_bands = a.bands;
  // the inverse that follows on the stream finds an empty argmax
  if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) *a.argmax = 0ull;
  constexpr int R = NF > 0 ? FixedFft<NF == 0 ? 64 : NF>::r[FixedFft<NF == 0 ? 64 : NF>::count - 1] : 1;
  for (int g = tid; g < n / R; g += nthr) s_gop[g] = 0;
  __syncthreads();
  auto shifted = [&](int kz, int t) -> uint32_t {  // (klin + nv / 2) mod nv with klin < nv
    const uint32_t klin = ((uint32_t)kz * n + (uint32_t)kx) * (uint32_t)H2 + (uint32_t)(ky0 + t);
    uint32_t p = klin + (nv >> 1);
    if (p >= nv || p < klin) p -= nv;
    return p;
  };
  for (int zp = tid; zp < n; zp += nthr) {
    const int kz = pos2freq<NF>(zp, plan);
    s_kz[zp] = (short)kz;
    s_live[zp] = a.slab_live[zp];
    s_live[n + zp] = a.slab_live[n + zp];
    if (a.laplace) {
      const uint32_t p0 = shifted(kz, 0), p1 = shifted(kz, wt - 1);
      const int op = fusion_op_run(p0, p1, s_bands);
      s_op[zp] = (uint8_t)op;
      if (op != kFuseMax) s_gop[zp / R] = 1;
    }
  }
  __syncthreads();
  if constexpr (NF > 0) {
    // which of the R slabs of each first-stage butterfly are live
    constexpr int R0 = FixedFft<NF>::r[0], m0 = NF / R0;
    for (int i = tid; i < 2 * m0; i += nthr) {
      const uint8_t* l = s_live + (i < m0 ? i : n + i - m0);
      unsigned k = 0;
#pragma unroll
      for (int j = 0; j < R0; ++j) k |= (l[j * m0] ? 1u : 0u) << j;
      s_mask[i] = (uint16_t)k;
    }
    __syncthreads();
  }
  // MEAN divides by the total channel count: a product with the reciprocal,
  // exact for the reference's 4 channels (within one rounding otherwise)
  const float inv_total = 1.0f / (float)a.n_total_ch;
  auto val = [&](int c, int t, int i) -> float2& { return tile[c * slot + z_off<NF>(i) * W + t]; };
  // z_off(r0 + j m) is linear in j: m is a multiple of the pad's period, or m = 1 within one period
  auto at = [=](int c, int t, int i, int m) {
    return SmemCursor{tile + c * slot + z_off<NF>(i) * W + t, (m == 1 ? 1 : z_off<NF>(m)) * W, slot};
  };
  // low-pass: keep the products whose FFT-shifted index p = (i N + j) + N^2 k
  // has i, j, k in [lp_lo, lp_hi]
  auto passed = [&](int i, int t) -> bool {
    if (!a.lowpass) return true;
    const uint32_t p = shifted(s_kz[i], t), n2 = (uint32_t)n * (uint32_t)n, kk = p / n2, rem = p - kk * n2;
    const uint32_t ii = rem / (uint32_t)n, jj = rem - ii * (uint32_t)n;
    return !(ii < a.lp_lo || ii > a.lp_hi || jj < a.lp_lo || jj > a.lp_hi || kk < a.lp_lo || kk > a.lp_hi);
  };
  // the fused value at a position whose channels are in the slots
  auto fused_at = [&](int t, int i) -> float2 {
    if (!a.laplace) return passed(i, t) ? val(0, t, i) : make_float2(0.f, 0.f);
    int op = s_op[i];
    if (op == kFuseMixed) op = fusion_op(shifted(s_kz[i], t), s_bands);
    float2 sum = make_float2(0.f, 0.f), mx = sum;
    float best = -1.f;
#pragma unroll
    for (int c = 0; c < CC; ++c) {
      const float2 u = val(c, t, i);
      sum = cadd(sum, u);
      const float e = u.x * u.x + u.y * u.y;
      mx = e > best ? u : mx;
      best = e > best ? e : best;
    }
    return op == kFuseMax ? mx
                          : (op == kFuseMean ? make_float2(sum.x * inv_total, sum.y * inv_total) : make_float2(0.f, 0.f));
  };
  // complexMulSeq: C = F * conj(G)
  auto cross = [](float2 F, float2 G) { return make_float2(F.x * G.x - F.y * (-G.y), F.x * (-G.y) + F.y * G.x); };
  for (int side = 0; side < 2; ++side) {
    // plain correlation: channel 0 of each side, low-pass: channel 1
    const float2* src = a.spec + (size_t)(side * a.n_data_ch + (a.laplace ? 0 : a.lowpass)) * plane +
                        (size_t)xp * H2p + ky0;
    const int zs = n * H2p;
    if constexpr (NF > 0) {
      constexpr int cnt = FixedFft<NF>::count;
      const uint16_t* mask = s_mask + side * (NF / FixedFft<NF>::r[0]);
      auto ld = [=](int, int t, int i, int m) {
        const float2* p = src + (size_t)i * zs + t;
        const unsigned k = t < wt ? mask[i] : 0u;
        const size_t js = (size_t)m * zs;
        return [=](int c, int j) { return (k >> j) & 1u ? __ldg(p + c * plane + j * js) : make_float2(0.f, 0.f); };
      };
      // the first stage's items are one channel's (they are the fewest: n / R0 butterflies a column), the others'
      // all channels'
      auto ld1 = [=](int c, int t, int i, int m) {
        const auto f = ld(0, t, i, m);
        return [=](int, int j) { return f(c, j); };
      };
      pass_ct<NF, false, 1, false, 0, 1>(PassMap{CC, lw}, plan.tw, tid, nthr, ld1, at, at);
      if constexpr (cnt > 2) __syncthreads();
      pass_ct<NF, false, CC, true, 1, cnt - 1>(PassMap{1, lw}, plan.tw, tid, nthr, at, at, at);
      __syncthreads();
      for (int it = tid; it < (n / R) << lw; it += nthr) {
        const int t = it & (W - 1), g = it >> lw, i0 = g * R;
        float2 F[R];
        float2* row = tile + z_off<NF>(i0) * W + t;
        if (!a.laplace || s_gop[g]) {
          // rare: rules other than the maximum near the spectrum's centre, or the plain and low-pass modes
#pragma unroll 1
          for (int c = 0; c < CC; ++c) {
            float2 x[R];
#pragma unroll
            for (int j = 0; j < R; ++j) x[j] = row[c * slot + j * W];
            dft_small<R, false>(x);
#pragma unroll
            for (int j = 0; j < R; ++j) row[c * slot + j * W] = x[j];
          }
#pragma unroll
          for (int j = 0; j < R; ++j) F[j] = fused_at(t, i0 + j);
        } else {
          // the first channel of largest energy
          float best[R];
#pragma unroll
          for (int j = 0; j < R; ++j) {
            F[j] = make_float2(0.f, 0.f);
            best[j] = -1.f;
          }
#pragma unroll
          for (int c = 0; c < CC; ++c) {
            float2 x[R];
#pragma unroll
            for (int j = 0; j < R; ++j) x[j] = row[c * slot + j * W];
            dft_small<R, false>(x);
#pragma unroll
            for (int j = 0; j < R; ++j) {
              const float e = x[j].x * x[j].x + x[j].y * x[j].y;
              F[j] = e > best[j] ? x[j] : F[j];
              best[j] = e > best[j] ? e : best[j];
            }
          }
        }
        row += CC * slot;
        if (side == 1) {
          float2 x[R];
#pragma unroll
          for (int j = 0; j < R; ++j) x[j] = cross(row[j * W], F[j]);
          dft_small<R, true>(x);
#pragma unroll
          for (int j = 0; j < R; ++j) F[j] = x[j];
        }
#pragma unroll
        for (int j = 0; j < R; ++j) row[j * W] = F[j];
      }
    } else {
      // channels as groups of transforms: an item of one channel keeps to the registers of two blocks per SM
      const PassMap map{CC, lw};
      const uint8_t* live = s_live + side * n;
      auto ld = [=](int c, int t, int i, int m) {
        const float2* p = src + (size_t)c * plane + (size_t)i * zs + t;
        const bool ok = t < wt;
        const size_t js = (size_t)m * zs;
        const uint8_t* l = live + i;
        return [=](int, int j) { return ok && l[j * m] ? __ldg(p + j * js) : make_float2(0.f, 0.f); };
      };
      pass_rt<false, 1, false>(plan, map, map, map, cs, tid, nthr, ld, at, at);
      __syncthreads();
      for (int it = tid; it < n << lw; it += nthr) {
        const int t = it & (W - 1), i = it >> lw;
        const float2 v = fused_at(t, i);
        float2& o = val(CC, t, i);
        o = side == 0 ? v : cross(o, v);
      }
    }
    __syncthreads();
  }
  float2* dst = a.cspec + (size_t)xp * H2p + ky0;
  auto pat = [=](int, int t, int i, int m) { return at(CC, t, i, m); };
  auto sv = [=](int, int t, int i, int m) {
    float2* p = dst + (size_t)i * n * H2p + t;
    const bool ok = t < wt;
    const size_t js = (size_t)m * n * H2p;
    return [=](int, int j, float2 v) {
      if (ok) p[j * js] = v;
    };
  };
  if constexpr (NF > 0) {
    pass_ct<NF, true, 1, true, 1, -1>(PassMap{1, lw}, plan.tw, tid, nthr, pat, pat, sv);
  } else {
    const PassMap map{1, lw};
    pass_rt<true, 1, true>(plan, map, map, map, cs, tid, nthr, pat, pat, sv);
  }
}

// ---------------------------------------------------------------- launchers

constexpr int kMaxSmem = 227 * 1024;

// Opt-in dynamic shared memory: everything the static shared memory leaves.
static cudaError_t allow_max_smem(const void* fn) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem - (int)fa.sharedSizeBytes);
}

// The z pass of C channels per side with tiles of wt columns: the width is a
// compile-time constant (4 or 8) for the compile-time lengths.
using FuseZFn = void (*)(const SpatialArgs, const FftPlan, int);
template <int NF, int LW>
static FuseZFn fuse_z_channels(int C) {
  return C == 1 ? k_fuse_z<NF, 1, LW> : (C == 2 ? k_fuse_z<NF, 2, LW> : (C == 3 ? k_fuse_z<NF, 3, LW> : k_fuse_z<NF, 4, LW>));
}
template <int NF>
static FuseZFn fuse_z_kernel(int C, int wt) {
  if constexpr (NF > 0)
    return wt >= 8 ? fuse_z_channels<NF, 3>(C) : fuse_z_channels<NF, 2>(C);
  else
    return fuse_z_channels<0, -1>(C);
}

// The forward x pass of C channels: tiles of 8 columns (64-byte rows), so four
// or more blocks fit on an SM at N = 200 with three channels.
constexpr int kXFwdLog2 = 3, kXInvLog2 = 4;
using FftXFn = void (*)(const ColArgs);
template <int NF>
static FftXFn fft_x_forward(int C) {
  return C == 1 ? k_fft_x<NF, false, 1, kXFwdLog2>
                : (C == 2 ? k_fft_x<NF, false, 2, kXFwdLog2>
                          : (C == 3 ? k_fft_x<NF, false, 3, kXFwdLog2> : k_fft_x<NF, false, 4, kXFwdLog2>));
}

static auto scan_rows_kernel(int C) {
  return C == 1 ? k_scan_rows<1> : (C == 2 ? k_scan_rows<2> : (C == 3 ? k_scan_rows<3> : k_scan_rows<4>));
}

template <int NF>
static cudaError_t set_attrs() {
  cudaError_t e = cudaSuccess;
  for (auto fn : {(const void*)k_r2c_rows<NF>, (const void*)k_c2r_rows<NF>, (const void*)k_fft_x<NF, true, 1, 4>})
    if (e == cudaSuccess) e = allow_max_smem(fn);
  for (int C = 1; C <= 4; ++C)
    if (e == cudaSuccess) e = allow_max_smem((const void*)fft_x_forward<NF>(C));
  for (int C = 1; C <= 4; ++C)
    for (int wt : {4, 8})
      if (e == cudaSuccess) e = allow_max_smem((const void*)fuse_z_kernel<NF>(C, wt));
  return e;
}

cudaError_t spatial_init_attributes(int N, int M) {
  cudaError_t e = cudaSuccess;
  PHGPU_DISPATCH_N(N, e = set_attrs<NF>());
  if (e == cudaSuccess && M != N) PHGPU_DISPATCH_N(M, e = set_attrs<NF>());
  for (int C = 1; C <= 4; ++C)
    if (e == cudaSuccess) e = allow_max_smem((const void*)scan_rows_kernel(C));
  return e;
}

// Whether PHGPU_DISPATCH_N gives N a compile-time plan.
static bool fixed_length(int N) {
  bool fixed = false;
  PHGPU_DISPATCH_N(N, fixed = NF > 0);
  return fixed;
}

// Registers a thread of the passes with runtime plans (their launch bounds' share); 0 for compile-time ones.
static int pass_regs(int N) { return fixed_length(N) ? 0 : 96; }

// Shared memory of the prime-radix scratch of runtime plans.
static size_t prime_scratch(int N) { return fixed_length(N) ? 0 : kMaxGenericRadix * sizeof(float4); }

static size_t fuse_z_smem(int N, int C, int wt) {
  int rows = N;
  PHGPU_DISPATCH_N(N, rows = z_off<NF>(N));
  return (size_t)(C + 1) * rows * wt * sizeof(float2) + prime_scratch(N) + 8 * (size_t)N;
}

constexpr size_t kFuseZStatic = 2 * 1024;  // the kernel's static and the system's shared memory, rounded up

// Tile width of the z pass: the widest (<= 8: 64-byte rows) of which two
// blocks fit on an SM, since the blocks hide one another's barriers and loads.
static int fuse_z_tile(int N, int C) {
  int wt = 8;
  while (wt > 2 && fuse_z_smem(N, C, wt) + kFuseZStatic > (size_t)kMaxSmem / 2) wt >>= 1;
  return wt;
}

int fuse_z_width(int N, int C, int tile) {
  const bool fits = (tile == 2 || tile == 4 || tile == 8 || tile == 16) && fuse_z_smem(N, C, tile) + kFuseZStatic <= (size_t)kMaxSmem;
  const int wt = fits ? tile : fuse_z_tile(N, C);
  return fixed_length(N) ? (wt >= 8 ? 8 : 4) : wt;
}

// Threads of a z-pass block: the least idle time over its stages.  With a
// compile-time plan an item carries the C channels of a side; runtime plans
// take the channels as transforms of their own.
static int fuse_z_threads(const FftPlan& p, int C, int wt) {
  if (!fixed_length(p.n))
    return pass_threads(p, C * wt, 1, 128, fuse_z_max_threads<0>(), 80, fuse_z_smem(p.n, C, wt));
  // a grid of at most three blocks an SM (of the compile-time lengths N = 64): one thread per item of the first
  // stage, whose items are one channel's (15 -> 13 us); runtime plans weigh the threads resident on an SM above
  if ((p.n / 2 + wt) / wt * p.n <= 3 * 148)
    return std::max(64, std::min((C * wt * p.n / p.radix[0] + 31) / 32 * 32, fuse_z_max_threads<64>()));
  int best = 256;
  double best_cost = 1e300;
  const int lo = std::min(192, (wt * p.n / p.radix[0] + 31) / 32 * 32);
  for (int t = std::max(lo, 64); t <= fuse_z_max_threads<64>(); t += 32) {
    double cost = 0.0;
    for (int s = 0; s < p.nstage; ++s) {
      const int items = wt * p.n / p.radix[s];
      cost += p.radix[s] * (2.0 * C + 1.0) * ((items + t - 1) / t) * t;
    }
    if (cost <= best_cost * 1.0001) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}

cudaError_t launch_spatial_forward(const SpatialArgs& a, int side, cudaStream_t st) {
  const int N = a.N, H2 = N / 2 + 1;
  const size_t nv = (size_t)N * N * N;
  const size_t plane = (size_t)N * N * spatial_h2p(N);
  float* grids = side == 0 ? a.grids_f : a.grids_g;
  const int nch = a.laplace ? a.n_data_ch : (a.lowpass ? 2 : 1);
  float2* spec = a.spec + (size_t)(side * a.n_data_ch) * plane;
  const ColArgs c{N, spec, plane, a.grids_are_means ? nullptr : a.rowmask + (size_t)side * N * N,
                  a.slab_live + (size_t)side * N, a.full_spec, *a.plan};
  if (a.grids_are_means) {
    const dim3 gr((N * N + 2 * kRowPairs - 1) / (2 * kRowPairs), nch);
    const size_t smr = (size_t)kRowPairs * row_stride(N) * sizeof(float2) + prime_scratch(N);
    const int tr = pass_threads(*a.plan, kRowPairs, 1, 128, 320, pass_regs(N), smr);
    PHGPU_DISPATCH_N(N, launch_kernel(k_r2c_rows<NF>, dim3(gr), dim3(tr), smr, st, N, grids, nv, spec, plane, *a.plan));
  } else {
    const ScanRowArgs r{N, scan_rows_block(N), reinterpret_cast<float4*>(grids), grids + 4 * nv, a.plan->tw, a.rowlive[side],
                        a.rowmask + (size_t)side * N * N, spec, plane, a.clear,
                        a.plan_half ? dense_row_limit(N) : N, a.plan_half ? *a.plan_half : FftPlan{}, a.half_pos};
    const dim3 gr(N, (N + r.rows_block - 1) / r.rows_block);
    const size_t smr = scan_rows_smem(N);
    launch_kernel(scan_rows_kernel(nch), dim3(gr), dim3(kRowsWarps * 32), smr, st, r);
  }
  // channels of one launch: as many as leave two blocks an SM's shared memory
  const size_t per = (size_t)N * (1 << kXFwdLog2) * sizeof(float2), extra = prime_scratch(N) + (size_t)N;
  int cc = nch;
  while (cc > 1 && cc * per + extra + 2048 > (size_t)kMaxSmem / 2) --cc;
  const dim3 gx((H2 + (1 << kXFwdLog2) - 1) >> kXFwdLog2, N);
  for (int ch = 0; ch < nch; ch += cc) {
    ColArgs cx = c;
    cx.spec += (size_t)ch * plane;
    const int k = std::min(cc, nch - ch);
    const bool fixed = fixed_length(N);  // an item carries all channels, or one of them
    const int tx = pass_threads(*a.plan, (1 << kXFwdLog2) * (fixed ? 1 : k), fixed ? k : 1, fixed || ends_in_prime_stage(*a.plan) ? 160 : 128, kXThreads,
                                pass_regs(N), k * per + extra);
    FftXFn fn = nullptr;
    PHGPU_DISPATCH_N(N, fn = fft_x_forward<NF>(k));
    launch_kernel(fn, dim3(gx), dim3(tx), k * per + extra, st, cx);
    count_launches(1);
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_spatial_fuse_z(const SpatialArgs& a, cudaStream_t st) {
  const int N = a.N, H2 = N / 2 + 1;
  const int C = a.laplace ? a.n_data_ch : 1;
  const int wt = fuse_z_width(N, C, a.fuse_tile);
  const size_t sm = fuse_z_smem(N, C, wt);
  if (sm + kFuseZStatic > (size_t)kMaxSmem) return cudaErrorInvalidConfiguration;
  const dim3 g((H2 + wt - 1) / wt, N);
  const int lw = wt == 16 ? 4 : (wt == 8 ? 3 : (wt == 4 ? 2 : 1));
  FuseZFn fn = nullptr;
  PHGPU_DISPATCH_N(N, fn = fuse_z_kernel<NF>(C, wt));
  launch_kernel(fn, dim3(g), dim3(fuse_z_threads(*a.plan, C, wt)), sm, st, a, *a.plan, lw);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_spatial_inverse(const SpatialArgs& a, cudaStream_t st) {
  const int N = a.N, H2 = N / 2 + 1;
  const uint32_t limit = a.argmax_limit ? a.argmax_limit : 0xffffffffu;
  const ColArgs c{N, a.cspec, 0, nullptr, nullptr, 1, *a.plan};
  const dim3 gx((H2 + (1 << kXInvLog2) - 1) >> kXInvLog2, N);
  const size_t smx = (size_t)N * (1 << kXInvLog2) * sizeof(float2) + prime_scratch(N);
  const int nblk = (N * N + 2 * kInvPairs - 1) / (2 * kInvPairs);
  const size_t smr = (size_t)kInvPairs * row_stride(N) * sizeof(float2) +
                     (fixed_length(N) ? 0 : prime_scratch(N) + (size_t)N * sizeof(int) + 16);
  const int tr = pass_threads(*a.plan, kInvPairs, 1, 128, 320, pass_regs(N), smr);
  const int tx = pass_threads(*a.plan, 1 << kXInvLog2, 1, fixed_length(N) ? 160 : 128, kXThreads, pass_regs(N), smx);
  PHGPU_DISPATCH_N(N, launch_kernel(k_fft_x<NF, true, 1, kXInvLog2>, dim3(gx), dim3(tx), smx, st, c);
                   launch_kernel(k_c2r_rows<NF>, dim3(nblk), dim3(tr), smr, st, N, a.cspec, *a.plan, a.argmax, a.volume, limit));
  count_launches(2);
  return cudaGetLastError();
}

}  // namespace phgpu
