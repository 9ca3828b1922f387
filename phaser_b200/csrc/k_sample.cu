// S^2 sampling on the GPU: spherical projection of each point and exact 1-NN
// of every Driscoll-Healy grid direction among the projected points.
//
// Reference behaviour: SphericalProjection::naiveProjection
// (phaser_common/src/common/spherical-projection.cc:19-41) and
// PointCloud::getNearestPoints / sampleNearestWithoutCloudInfo
// (phaser_common/src/model/point-cloud.cc:93-157).  Distances are float L2^2
// accumulated as ((dx^2 + dy^2) + dz^2) without contraction; the lowest point
// index wins exact ties; a match farther than the squared voxel size is
// dropped (all channels 0).
//
// Search structure: the projected points are counting-sorted by the grid's
// own (theta, phi) bins -- row i covers colatitudes [i, i + 1) pi / 2B,
// column j longitudes within pi / 2B of 2 pi j / 2B -- so every bin, and
// every run of neighbouring columns of a row, is one contiguous point range.
// A direction (i, j), one group of 8 lanes, sweeps the non-empty rows outward from its
// own row while the row's colatitude distance |theta_q - row| can still beat
// the bound; a row whose window is wide and full is probed at columns j-1..j+1 for a
// tighter bound, and in each row only the columns whose longitudes lie within
// the bound's spherical cap are scanned (the cap's longitude half-width at
// the row's colatitudes).  A LiDAR scan needs about two rows and fifty
// points per direction, so the search is a short chain of dependent loads
// per direction, run for all directions at once.  The bound is kept as an
// upper bound hb of hav(beta) = sin^2(beta / 2) of the best distance's angle
// inflated by 1e-4 rad, and a row's window follows from the haversine law
//   hav(d) = hav(t - t_q) + sin t sin t_q hav(dphi)
// with per-row tables (sin of the row edges, hav of the row's colatitude
// distance) deflated by margins far above the float rounding of the unit
// vectors, so no point that could be (or tie) the nearest is ever skipped:
// the search is exact whatever bound it starts from.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "kernels.h"

namespace phgpu {

// float functions evaluated in double and rounded once (correctly rounded
// except in rare near-halfway cases; glibc's float versions can differ by one
// ulp, so projected coordinates match the reference with high probability).
__device__ __forceinline__ float acos_f(float x) { return (float)acos((double)x); }
__device__ __forceinline__ float atan2_f(float y, float x) { return (float)atan2((double)y, (double)x); }

// One cloud's buffers; the kernels below work on up to two clouds at once
// (blockIdx.y), since one cloud's search leaves the device idle: its time is
// the latency of a few dependent loads per step.
struct CloudView {
  const float4* xyzi;
  const float* refl;
  const float* amb;
  const uint32_t* P_dev;  // when set: the point count in device memory
  int P;
  int n_out_ch;
  float max_sq;
  const float4* grid;
  float4* proj;
  double* range;
  uint32_t* key;
  uint32_t* slot;  // rank of the point among its bin's
  float4* sorted;
  uint32_t *bin_count, *row_count, *bin_start;
  int *row_nxt, *row_prv;
  float *sin_tab, *hav_tab, *stq_tab;
  float* out;
  int32_t* nn_idx;
};
struct CloudPair {
  CloudView c[2];
};

// Projection of every point, its bin and the per-bin and per-row counts.
__global__ void k_project(const __grid_constant__ CloudPair pr, int n2b) {
  chain_begin();
  const CloudView& v = pr.c[blockIdx.y];
  float4* __restrict__ proj = v.proj;
  double* __restrict__ range = v.range;
  uint32_t* __restrict__ key = v.key;
  uint32_t* __restrict__ bin_count = v.bin_count;
  uint32_t* __restrict__ row_count = v.row_count;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (v.P_dev ? (int)*v.P_dev : v.P)) return;
  const float4 p = v.xyzi[i];
  const float sxy = __fadd_rn(__fmul_rn(p.x, p.x), __fmul_rn(p.y, p.y));
  const double dist_xy = (double)sqrtf(sxy);
  const float zz = __fmul_rn(p.z, p.z);
  const double dist = sqrt(__dadd_rn(__dmul_rn(dist_xy, dist_xy), (double)zz));
  const float oz = (float)__ddiv_rn((double)p.z, dist);
  const double tx = (double)acos_f(oz);
  const double ty = fmod(__dadd_rn((double)atan2_f(p.y, p.x), 2.0 * M_PI), 2.0 * M_PI);
  double st, ct, sp, cp;
  sincos(tx, &st, &ct);
  sincos(ty, &sp, &cp);
  const float ox = (float)__dmul_rn(st, cp);
  const float oy = (float)__dmul_rn(st, sp);
  proj[i] = make_float4(ox, oy, oz, 0.0f);
  range[i] = dist;
  // points at the origin or with non-finite coordinates have no direction:
  // they are left out of the search structure
  if (!(isfinite(ox) && isfinite(oy) && isfinite(oz))) {
    key[i] = 0xffffffffu;
    return;
  }
  const double w = M_PI / (double)n2b;  // bin height in theta, half bin width in phi
  const int bi = min(max((int)(tx / w), 0), n2b - 1);
  int bj = (int)floor(ty / (2.0 * w) + 0.5);
  bj = bj >= n2b ? bj - n2b : max(bj, 0);
  const uint32_t b = (uint32_t)(bi * n2b + bj);
  key[i] = b;
  // consecutive points of a scan mostly share bins and rows: one atomic per
  // group of lanes with the same key.  The bin's count before the group is
  // the group's place among the bin's points, so the scatter needs no atomics.
  {
    const unsigned act = __activemask();
    const int lane = threadIdx.x & 31;
    const unsigned pb = __match_any_sync(act, b);
    const int leader = __ffs(pb) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&bin_count[b], (uint32_t)__popc(pb));
    const unsigned pr2 = __match_any_sync(act, bi);
    if (lane == __ffs(pr2) - 1) atomicAdd(&row_count[bi], (uint32_t)__popc(pr2));
    base = __shfl_sync(pb, base, leader);
    v.slot[i] = base + __popc(pb & ((1u << lane) - 1u));
  }
}

// Bin starts and row tables.  Block r: the exclusive scan of row r's n2b bin
// counts offset by the points of rows < r; row_nxt[r] = first non-empty row
// >= r (n2b if none), row_prv[r] = last non-empty row < r (-1 if none).
constexpr int kBinScanThreads = 256;
constexpr int kMaxGridSide = 1024;  // 2B for B <= 512

// Also the row tables of the window bound: sin_tab[r] = sin(r w) - 1e-5
// (clamped at 0) for the row edges r = 0..2B, hav_tab[d] = hav((d - 1/2) w)
// (1 - 1e-4) for the colatitude distance of a row d >= 1 rows away
// (hav_tab[0] = 0), stq_tab[i] = sin((i + 1/2) w) - 1e-5 (clamped at 0) for the
// direction rows, w = pi / 2B.
__global__ void __launch_bounds__(kBinScanThreads) k_bin_scan(int n2b, const __grid_constant__ CloudPair pr) {
  chain_begin();
  const CloudView& v0 = pr.c[blockIdx.y];
  const uint32_t* __restrict__ bin_count = v0.bin_count;
  const uint32_t* __restrict__ row_count = v0.row_count;
  uint32_t* __restrict__ bin_start = v0.bin_start;
  int *__restrict__ row_nxt = v0.row_nxt, *__restrict__ row_prv = v0.row_prv;
  float *__restrict__ sin_tab = v0.sin_tab, *__restrict__ hav_tab = v0.hav_tab, *__restrict__ stq_tab = v0.stq_tab;
  __shared__ uint32_t s_rows[kMaxGridSide];
  __shared__ uint32_t s_w[kBinScanThreads / 32];
  __shared__ uint32_t s_base;
  const int r = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t part = 0;
  for (int q = t; q < n2b; q += kBinScanThreads) {
    const uint32_t v = __ldg(&row_count[q]);
    s_rows[q] = v;
    part += q < r ? v : 0u;
  }
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (lane == 0) s_w[warp] = part;
  __syncthreads();
  const double w = M_PI / (double)n2b;
  if (t == 64) {
    sin_tab[r] = fmaxf((float)sin(r * w) - 1e-5f, 0.0f);
    if (r == n2b - 1) sin_tab[n2b] = 0.0f;
  } else if (t == 96) {
    const double h = sin(0.5 * (r - 0.5) * w);
    hav_tab[r] = r == 0 ? 0.0f : (float)(h * h) * (1.0f - 1e-4f);
  } else if (t == 128) {
    stq_tab[r] = fmaxf((float)sin((r + 0.5) * w) - 1e-5f, 0.0f);
  } else if (t == 160) {
    uint32_t b = 0;
    for (int k = 0; k < kBinScanThreads / 32; ++k) b += s_w[k];
    s_base = b;
  } else if (warp == 0) {  // the next non-empty row, 32 rows a step
    int nx = n2b;
    for (int q = r; q < n2b; q += 32) {
      const unsigned m = __ballot_sync(0xffffffffu, q + lane < n2b && s_rows[q + lane] != 0u);
      if (m) {
        nx = q + __ffs(m) - 1;
        break;
      }
    }
    if (lane == 0) {
      row_nxt[r] = nx;
      if (r == n2b - 1) row_nxt[n2b] = n2b;
    }
  } else if (warp == 1) {  // the previous one
    int pv = -1;
    for (int q = r - 1; q >= 0; q -= 32) {
      const unsigned m = __ballot_sync(0xffffffffu, q - lane >= 0 && s_rows[q - lane] != 0u);
      if (m) {
        pv = q - (__ffs(m) - 1);
        break;
      }
    }
    if (lane == 0) {
      row_prv[r] = pv;
      if (r == n2b - 1) row_prv[n2b] = s_rows[r] ? r : pv;
    }
  }
  __syncthreads();
  // row scan: thread t owns columns [t * per, (t + 1) * per)
  const int per = (n2b + kBinScanThreads - 1) / kBinScanThreads;
  const uint32_t* rc = bin_count + (size_t)r * n2b;
  const int c_lo = min(n2b, t * per), c_hi = min(n2b, (t + 1) * per);
  uint32_t sum = 0;
  for (int c = c_lo; c < c_hi; ++c) sum += __ldg(&rc[c]);
  uint32_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  __syncthreads();
  if (lane == 31) s_w[warp] = incl;
  __syncthreads();
  uint32_t run = s_base + incl - sum;
  for (int k = 0; k < warp; ++k) run += s_w[k];
  uint32_t* bs = bin_start + (size_t)r * n2b;
  for (int c = c_lo; c < c_hi; ++c) {
    bs[c] = run;
    run += __ldg(&rc[c]);
  }
  if (r == n2b - 1 && t == kBinScanThreads - 1) bin_start[(size_t)n2b * n2b] = run;
}

// Counting-sort scatter: sorted[k] = {x, y, z, point index (bits)}.
__global__ void k_bin_scatter(const __grid_constant__ CloudPair pr) {
  chain_begin();
  const CloudView& v = pr.c[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (v.P_dev ? (int)*v.P_dev : v.P)) return;
  const uint32_t k = v.key[i];
  if (k == 0xffffffffu) return;
  const float4 p = v.proj[i];
  v.sorted[v.bin_start[k] + v.slot[i]] = make_float4(p.x, p.y, p.z, __int_as_float(i));
}

__device__ __forceinline__ float ref_dist2(float qx, float qy, float qz, float4 p) {
  const float dx = __fsub_rn(qx, p.x);
  const float dy = __fsub_rn(qy, p.y);
  const float dz = __fsub_rn(qz, p.z);
  float r = __fmul_rn(dx, dx);
  r = __fadd_rn(r, __fmul_rn(dy, dy));
  r = __fadd_rn(r, __fmul_rn(dz, dz));
  return r;
}

// Nearest so far as (squared distance bits, point index): distances are sums
// of squares, never negative, so their bits order like the values and one
// 64-bit minimum takes the smaller distance, the lower index among equals.
typedef unsigned long long NnKey;
constexpr NnKey kNoPoint = ((NnKey)0x7f800000u << 32) | 0x7fffffffu;
__device__ __forceinline__ NnKey nn_key(float d, float idx_bits) {
  return ((NnKey)__float_as_uint(d) << 32) | __float_as_uint(idx_bits);
}
__device__ __forceinline__ float nn_dist(NnKey k) { return __uint_as_float((uint32_t)(k >> 32)); }

// Writes the sampled channels {range, intensity, reflectivity, ambient}
// (float) of the nearest point into out[ch][qi] for ch < n_out_ch and its
// index (or -1) into nn_idx; a match farther than max_sq is dropped.
__device__ __forceinline__ void emit_sample(int qi, int nq, float best, int bidx, float max_sq,
                                            const float4* __restrict__ xyzi, const double* __restrict__ range,
                                            const float* __restrict__ refl, const float* __restrict__ amb,
                                            int n_out_ch, float* __restrict__ out, int32_t* __restrict__ nn_idx) {
  const bool ok = (bidx != 0x7fffffff) && !(best > max_sq);
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (ok) {
    v[0] = (float)range[bidx];
    v[1] = xyzi[bidx].w;
    v[2] = refl ? refl[bidx] : 0.0f;
    v[3] = amb ? amb[bidx] : 0.0f;
  }
  for (int c = 0; c < n_out_ch; ++c) out[(size_t)c * nq + qi] = v[c];
  if (nn_idx) nn_idx[qi] = ok ? bidx : -1;
}


// ---------------------------------------------------------------- row sweep
constexpr float kAngleMargin = 1e-4f;

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Upper bound of sin^2(beta / 2) for the angle beta of a float squared chord
// inflated by kAngleMargin (sin(asin h + m / 2) <= h + m / 2), so float
// rounding of the unit vectors cannot hide a nearer point (the margin's own
// relative term also covers the approximate root's 2^-22); 2 (> 1) when the
// chord bounds nothing.
__device__ __forceinline__ float hav_of_l2(float best) {
  if (!(best < 3.99f)) return 2.0f;
  const float s = 0.5f * sqrt_approx(best) * (1.0f + kAngleMargin) + 0.5f * kAngleMargin;
  return s >= 1.0f ? 2.0f : s * s;
}

// Lanes per direction: a group of kGroup lanes strides over the points of a
// window (coalesced 16-byte loads), then reduces its minima.
constexpr int kGroup = 8;
constexpr int kLongLoads = 4;

// Points [k, e) of the sorted list: lane g takes points g, g + kGroup, ...;
// lane-private minima.  Two points of a lane are in flight (a window holds
// about 46), kLongLoads in long windows: a direction near a pole scans whole
// rows (thousands of points of a scan's outermost beam), and with two in
// flight the slowest such direction alone took 45 us of the kernel's 51.
__device__ __forceinline__ void scan_range(uint32_t k, uint32_t e, int g, float qx, float qy, float qz,
                                           const float4* __restrict__ sorted, NnKey& best) {
  k += g;
  auto step = [&](float4 p) {
    const NnKey key = nn_key(ref_dist2(qx, qy, qz, p), p.w);
    best = key < best ? key : best;
  };
  for (; k + 2 * kLongLoads * kGroup < e; k += kLongLoads * kGroup) {
    float4 p[kLongLoads];
#pragma unroll
    for (int u = 0; u < kLongLoads; ++u) p[u] = __ldg(&sorted[k + u * kGroup]);
#pragma unroll
    for (int u = 0; u < kLongLoads; ++u) step(p[u]);
  }
#pragma unroll 1
  for (; k + kGroup < e; k += 2 * kGroup) {
    const float4 p0 = __ldg(&sorted[k]), p1 = __ldg(&sorted[k + kGroup]);
    step(p0);
    step(p1);
  }
  if (k < e) step(__ldg(&sorted[k]));
}

// Columns c0 .. c0 + len - 1 (mod n2b) of row r (len <= 0: none): one run of
// the sorted points, two where the columns wrap.
struct Window {
  uint32_t k0, e0, k1, e1;
  __device__ __forceinline__ uint32_t points() const { return e0 - k0 + e1 - k1; }
};
__device__ __forceinline__ Window window(int r, int c0, int len, int n2b, const uint32_t* __restrict__ bin_start) {
  Window w{0, 0, 0, 0};
  if (len > 0) {
    c0 = c0 < 0 ? c0 + n2b : (c0 >= n2b ? c0 - n2b : c0);
    const uint32_t* rs = bin_start + (size_t)r * n2b;
    const int over = c0 + len - n2b;
    w.k0 = __ldg(&rs[c0]);
    w.e0 = __ldg(&rs[over > 0 ? n2b : c0 + len]);
    if (over > 0) {
      w.k1 = __ldg(&rs[0]);
      w.e1 = __ldg(&rs[over]);
    }
  }
  return w;
}
__device__ __forceinline__ void scan_window(const Window& w, int g, float qx, float qy, float qz,
                                            const float4* __restrict__ sorted, NnKey& best) {
  scan_range(w.k0, w.e0, g, qx, qy, qz, sorted, best);
  if (w.e1 > w.k1) scan_range(w.k1, w.e1, g, qx, qy, qz, sorted, best);
}

// Minimum over the group; every lane gets it.  The whole warp takes part:
// shuffles with a mask per group would run the warp's four groups one after
// the other up to the next reconvergence (four times the instructions).
__device__ __forceinline__ void group_nn_min(NnKey& best) {
#pragma unroll
  for (int o = kGroup / 2; o > 0; o >>= 1) {
    const NnKey other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other < best ? other : best;
  }
}

// Half-width k (in columns) of the cap window of row r, d rows from the
// direction's own row: column j +- c holds longitudes at least (c - 1/2) 2w
// away from phi_q, and a point of the row within the bound has
//   hav(dphi) <= x^2 = (hb - hav(row distance)) / (min(sin a, sin b) sin t_q)
// (sin is concave, so its minimum over the row's colatitudes [a, b] is at an
// edge).  dphi = 2 asin x takes Abramowitz and Stegun 4.4.45, which is within
// 7e-5 of asin on [0, 1]; the approximate quotient and root are covered by the
// factor 1 + 1e-5 on x^2 (a larger x has a larger asin).  Its error does not
// grow with the window: a looser bound (10 % at x = 1) takes in the middle of a
// cloud far from most directions, which the window of its near edge keeps out
// (100 k points within a degree, B = 256: 13.1 ms so, 3.5 with asinf).  n2b: the
// whole row.
__device__ __forceinline__ int row_window(int r, int d, int n2b, float inv_2w, float stq, float hb,
                                          const float* __restrict__ sin_tab, const float* __restrict__ hav_tab) {
  if (hb >= 1.0f) return n2b;
  const float num = hb - __ldg(&hav_tab[d]);
  const float den = fminf(__ldg(&sin_tab[r]), __ldg(&sin_tab[r + 1])) * stq;
  if (!(num < den)) return n2b;  // the bound reaches every longitude (or a pole row)
  if (num <= 0.0f) return 0;
  const float x = sqrt_approx(__fdividef(num, den) * (1.0f + 1e-5f));
  const float p = fmaf(fmaf(fmaf(-0.0187293f, x, 0.0742610f), x, -0.2121144f), x, 1.5707288f);
  const float e = 3.14159265f - 2.0f * sqrt_approx(fmaxf(1.0f - x, 0.0f)) * p + 2e-4f + kAngleMargin;
  const float kf = fmaf(e, inv_2w, 0.5f);
  return kf >= (float)n2b ? n2b : (int)kf;
}

constexpr int kQueryThreads = 256;
// Points of a wide window from which on it is probed.  A probe is a chain of
// dependent loads of its own: with every wide window probed, sparse clouds and
// ones seen through a narrow opening took longer than with one probe per
// direction (37 points, B = 256: 285 us against 183; now 165).  256 rather than 64
// or 128: 120 k points in a cone of 60 degrees, B = 100: 241, 288 and 276 us, scans of
// full circles within 1 us of one another.
constexpr uint32_t kProbePoints = 256;

// One group of kGroup lanes per direction of the 2B x 2B grid: the
// non-empty rows are visited outward from the direction's own row, nearest
// colatitude first, while their colatitude distance can beat the bound.  A row
// whose window is wide and holds many points is probed at columns j - 1 .. j + 1
// first, which makes the bound finite at the first row and keeps it tight when that row holds
// only stray points (the outermost beam's, split over two rows by rounding: a
// bound from far along such a row had 37 % of the directions of a 128-beam scan
// take the whole next row, 690 points a direction instead of about 60); then
// the columns within the bound's cap are scanned (the probed ones once).  The
// four groups of a warp (neighbouring directions of a row) step through the
// rows together, a group that is done idling.  B = 100, 131 k points, two
// clouds: 80 -> 28 us.
__global__ void __launch_bounds__(kQueryThreads, 6)
k_nn_rows(int n2b, uint32_t mul_n2b, const __grid_constant__ CloudPair pr) {
  chain_begin();
  const CloudView& v = pr.c[blockIdx.y];
  const float4* __restrict__ sorted = v.sorted;
  const uint32_t* __restrict__ bin_start = v.bin_start;
  const int *__restrict__ row_nxt = v.row_nxt, *__restrict__ row_prv = v.row_prv;
  const float *__restrict__ sin_tab = v.sin_tab, *__restrict__ hav_tab = v.hav_tab;
  const int nq = n2b * n2b;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int g = tid % kGroup, t = tid / kGroup;
  if (t >= nq) return;  // whole warps: nq = 4 B^2
  // rows from both poles inwards (0, n - 1, 1, n - 2, ...): the long scans
  // near the poles start first
  const int rank = fast_div(t, mul_n2b), j = t - rank * n2b;
  const int i = (rank & 1) ? n2b - 1 - (rank >> 1) : (rank >> 1);
  const int qi = i * n2b + j;
  const float inv_2w = (float)n2b * (0.5f / 3.14159265358979f);
  const float4 q = __ldg(&v.grid[qi]);
  const float stq = __ldg(&v.stq_tab[i]);
  NnKey best = kNoPoint;
  float hb = 2.0f;
  int up = __ldg(&row_nxt[i]), dn = __ldg(&row_prv[i]);
  // the nearest row not visited yet: r, d rows away; false when there is none
  // or its colatitude distance alone exceeds the bound
  int r, d;
  auto next_row = [&]() -> bool {
    const int du = up < n2b ? up - i : 0x7fffffff, dd = dn >= 0 ? i - dn : 0x7fffffff;
    const bool take_up = du <= dd;
    d = take_up ? du : dd;
    r = take_up ? up : dn;
    if (d == 0x7fffffff || !(__ldg(&hav_tab[d]) <= hb)) return false;
    if (take_up)
      up = __ldg(&row_nxt[up + 1]);
    else
      dn = __ldg(&row_prv[dn]);
    return true;
  };
  const int pw = min(3, n2b);
  bool act = true;
#pragma unroll 1
  for (;;) {
    act = act && next_row();
    if (!__any_sync(0xffffffffu, act)) break;
    int k = act ? row_window(r, d, n2b, inv_2w, stq, hb, sin_tab, hav_tab) : 0;
    bool all = 2 * k + 1 >= n2b;
    int c0 = all ? 0 : j - k, len = act ? (all ? n2b : 2 * k + 1) : 0;
    Window w = window(r, c0, len, n2b, bin_start);
    // a wide window of many points is probed at columns j - 1 .. j + 1 first
    const bool probe = act && k >= 3 && w.points() > kProbePoints;
    if (__any_sync(0xffffffffu, probe)) {
      scan_window(window(r, j - 1, probe ? pw : 0, n2b, bin_start), g, q.x, q.y, q.z, sorted, best);
      __syncwarp();
      group_nn_min(best);
      hb = hav_of_l2(nn_dist(best));
      if (probe) {  // what the probe left: one piece of a whole row, else both sides
        k = row_window(r, d, n2b, inv_2w, stq, hb, sin_tab, hav_tab);
        all = 2 * k + 1 >= n2b;
        c0 = all ? j + 2 : j - k;
        len = all ? n2b - pw : k - 1;
      }
      scan_window(window(r, j + 2, probe && !all ? k - 1 : 0, n2b, bin_start), g, q.x, q.y, q.z, sorted, best);
      w = window(r, c0, len, n2b, bin_start);
    }
    scan_window(w, g, q.x, q.y, q.z, sorted, best);
    __syncwarp();
    group_nn_min(best);
    hb = hav_of_l2(nn_dist(best));
  }
  if (g == 0)
    emit_sample(qi, nq, nn_dist(best), (int)(uint32_t)best, v.max_sq, v.xyzi, v.range, v.refl, v.amb, v.n_out_ch, v.out,
                v.nn_idx);
}

// ---------------------------------------------------------------- launcher

std::atomic<unsigned long long> g_launch_count{0};
thread_local int g_capture_depth = 0;
thread_local bool g_chain_launch = false;

namespace {
int grid_side(int max_queries) {
  int n = (int)sqrt((double)max_queries);
  while ((long long)n * n < max_queries) ++n;
  return n;
}
}  // namespace

size_t sampler_scratch_bytes(int max_points, int max_queries) {
  const int n2b = grid_side(max_queries);
  const size_t nbins = (size_t)n2b * n2b;
  size_t b = (size_t)max_points * sizeof(float4);                // proj
  b += (size_t)max_points * sizeof(double);                      // range
  b += 2 * (size_t)max_points * sizeof(uint32_t);                // key, slot
  b += (size_t)max_points * sizeof(float4);                      // sorted
  b += (nbins + (size_t)n2b) * sizeof(uint32_t);                 // bin counts, row counts
  b += (nbins + 1) * sizeof(uint32_t);                           // bin starts
  b += 2 * (size_t)(n2b + 1) * sizeof(int);                      // row tables
  b += 3 * (size_t)(n2b + 1) * sizeof(float);                    // window bound tables
  return b + 12 * 256;  // carve() rounds each region up to 256 bytes
}

static inline char* carve(char*& p, size_t bytes) {
  char* r = p;
  p += (bytes + 255) & ~(size_t)255;
  return r;
}

cudaError_t launch_sample(const SampleArgs* args, int n_clouds, cudaStream_t st) {
  const int n2b = args[0].n2b;
  if (n_clouds < 1 || n_clouds > 2 || n2b <= 0 || n2b > kMaxGridSide ||
      (size_t)n2b * n2b != (size_t)args[0].n_queries)
    return cudaErrorInvalidValue;
  const size_t nbins = (size_t)n2b * n2b;
  const size_t count_bytes = (nbins + (size_t)n2b) * sizeof(uint32_t);
  CloudPair pr;
  int P = 0;
  for (int i = 0; i < n_clouds; ++i) {
    const SampleArgs& a = args[i];
    if (a.n2b != n2b || a.max_points != args[0].max_points) return cudaErrorInvalidValue;
    CloudView& v = pr.c[i];
    char* p = (char*)a.scratch;
    v.proj = (float4*)carve(p, (size_t)a.max_points * sizeof(float4));
    v.range = (double*)carve(p, (size_t)a.max_points * sizeof(double));
    v.key = (uint32_t*)carve(p, (size_t)a.max_points * sizeof(uint32_t));
    v.slot = (uint32_t*)carve(p, (size_t)a.max_points * sizeof(uint32_t));
    v.sorted = (float4*)carve(p, (size_t)a.max_points * sizeof(float4));
    v.bin_count = (uint32_t*)carve(p, count_bytes);
    v.row_count = v.bin_count + nbins;
    v.bin_start = (uint32_t*)carve(p, (nbins + 1) * sizeof(uint32_t));
    v.row_nxt = (int*)carve(p, (size_t)(n2b + 1) * sizeof(int));
    v.row_prv = (int*)carve(p, (size_t)(n2b + 1) * sizeof(int));
    v.sin_tab = (float*)carve(p, (size_t)(n2b + 1) * sizeof(float));
    v.hav_tab = (float*)carve(p, (size_t)(n2b + 1) * sizeof(float));
    v.stq_tab = (float*)carve(p, (size_t)(n2b + 1) * sizeof(float));
    v.xyzi = a.xyzi;
    v.refl = a.refl;
    v.amb = a.amb;
    v.P_dev = a.n_dev;
    v.P = a.n_points;
    v.n_out_ch = a.n_out_ch;
    v.max_sq = a.max_sq;
    v.grid = a.grid;
    v.out = a.out;
    v.nn_idx = a.nn_idx;
    P = a.n_points > P ? a.n_points : P;
  }
  // both clouds' counts in one pitched fill (its pitch is limited to 2^31 - 1 bytes)
  const ptrdiff_t pitch = n_clouds == 2 ? (char*)pr.c[1].bin_count - (char*)pr.c[0].bin_count : 0;
  cudaError_t e = cudaSuccess;
  if (n_clouds == 2 && pitch >= (ptrdiff_t)count_bytes && pitch < (ptrdiff_t)0x7fffffff) {
    e = cudaMemset2DAsync(pr.c[0].bin_count, (size_t)pitch, 0, count_bytes, 2, st);
  } else {
    for (int i = 0; i < n_clouds && e == cudaSuccess; ++i) e = cudaMemsetAsync(pr.c[i].bin_count, 0, count_bytes, st);
  }
  if (e != cudaSuccess) return e;
  int launched = 0;
  const dim3 gp((P + 255) / 256, n_clouds);
  if (P > 0) {
    launch_kernel(k_project, dim3(gp), dim3(256), 0, st, pr, n2b);
    ++launched;
  }
  launch_kernel(k_bin_scan, dim3(n2b, n_clouds), dim3(kBinScanThreads), 0, st, n2b, pr);
  ++launched;
  if (P > 0) {
    launch_kernel(k_bin_scatter, dim3(gp), dim3(256), 0, st, pr);
    ++launched;
  }
  const size_t q_threads = nbins * kGroup;
  launch_kernel(k_nn_rows, dim3((unsigned)((q_threads + kQueryThreads - 1) / kQueryThreads), n_clouds), dim3(kQueryThreads), 0, st, 
      n2b, fast_div_mul((uint32_t)n2b), pr);
  ++launched;
  count_launches(launched);
  return cudaGetLastError();
}

}  // namespace phgpu
