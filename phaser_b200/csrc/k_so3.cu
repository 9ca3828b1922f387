// Inverse SO(3) transform of the correlation coefficients, |z|^2 and argmax.
//
// Reference behaviour (phaser_core/lib/SOFT/so3_correlate_fftw.c:102-161 and
// soft_fftw.c:1036-1914 with flag = 1, called from
// phaser_core/src/backend/correlation/spherical-correlation.cc:248-279):
//   c(l, m1, m2) = 2 pi sqrt(2/(2l+1)) fhat(l, -m1) (-1)^(m1+m2) conj(hhat(l, -m2))
//   S_{m1 m2}(beta_k) = sum_l c(l, m1, m2) dtilde^l_{m1 m2}(beta_k)
//   z(beta, alpha, gamma) = (B / pi) (1 / 2B) sum S_{m1 m2}(beta) e^{-i(m1 alpha + m2 gamma)}
// where only one member of each pair (m1, m2) / (-m1, -m2) is synthesised
// (the half H = {m1 > 0, m2 != -m1} + {(-m, m)} + {(0, m2 >= 0)}) and the
// other is its conjugate, so z is real.  Output layout [beta][alpha][gamma].
//
// The half spectrum is laid out S[a][b][beta] (a = m1 index in [0, 2B),
// b = m2 >= 0, beta fastest), so a synthesis thread per beta writes
// coalesced runs and both angle transforms read 128-byte beta segments.
//
// FP32 synthesis (k_so3_synth): one block per order class (p, q),
// 0 <= p <= q < B.  Thread k runs the FP64 three-term recurrence of
// dtilde^l_{p q}(beta_k) in l and accumulates in FP32 the four outputs the
// class feeds (so3_common.cuh).  The tensor-core synthesis from a stored
// Wigner table is in k_so3_tc.cu.  Only b = m2 >= 0 is kept (half spectrum);
// the gamma transform is a Hermitian complex-to-real one.
//
// Every kernel takes a batch of requests (grid dimension z or y): requests of
// one (B, bw_out) shape share the tables and plans.
#include <math.h>

#include <vector>

#include "fft_pass.cuh"
#include "kernels.h"
#include "so3_common.cuh"

namespace phgpu {

// KB betas per thread (k = t, t + ceil(n / KB), ...): KB recurrences in flight
// per thread cover the double-precision latency, and the coefficients loaded
// from shared memory serve KB of them.  The host picks the KB that leaves the
// fewest lanes idle (n = 200: 7 betas in 29 of a warp's 32 lanes, where 4 betas
// fill 50 of 64).  A step is three double-precision operations, one conversion
// and four packed multiply-adds, and the issue of these 64-bit operations
// bounds the kernel; two steps are written out, the second in the registers of
// the value it replaces, which takes the moves between them out (16 -> 11.5
// instructions a step).  Four separate FMA pairs, one step and 4 betas for every
// length: B = 150 with padding 10 185 us, now 124; B = 256 1077 -> 860; B = 100
// 46 -> 41.  Packing two betas of a component (no duplicated operand, doubled
// coefficients) takes more registers: 160, 958 and 50 us.
template <int KB>
__device__ __forceinline__ void so3_step(const float4* __restrict__ c, double a, double b, double g, const double (&cb)[KB],
                                         double (&dprev)[KB], const double (&dcur)[KB], float2 (&acc)[KB][4]) {
  const float4 c01 = c[0], c23 = c[1];
#pragma unroll
  for (int u = 0; u < KB; ++u) {
    const float d = (float)dcur[u];
    const float2 dd = make_float2(d, d);
    acc[u][0] = __ffma2_rn(make_float2(c01.x, c01.y), dd, acc[u][0]);
    acc[u][1] = __ffma2_rn(make_float2(c01.z, c01.w), dd, acc[u][1]);
    acc[u][2] = __ffma2_rn(make_float2(c23.x, c23.y), dd, acc[u][2]);
    acc[u][3] = __ffma2_rn(make_float2(c23.z, c23.w), dd, acc[u][3]);
    dprev[u] = wig_step(a, b, g, cb[u], dprev[u], dcur[u]);
  }
}

constexpr int kSynthThreads = 128;

template <int KB>
__global__ void __launch_bounds__(kSynthThreads, KB > 5 ? 4 : 5)
    k_so3_synth(int bw_in, int bw_out, const __grid_constant__ So3Batch bt, const double* __restrict__ btab,
                const double* __restrict__ wtab) {
  chain_begin();
  extern __shared__ __align__(16) double sm[];
  double* fa = sm;                      // [bw_in] pairs {a, b}, then shifts
  double* gs = fa + 2 * bw_in;          // fb * shift
  float2* cv = (float2*)(gs + bw_in + (bw_in & 1));  // [bw_in][4]
  const float2* __restrict__ fz = bt.fused[blockIdx.y];
  float2* __restrict__ S = bt.out[blockIdx.y].S;
  int p, q;
  so3_class(blockIdx.x, &p, &q);
  const int nl = bw_in - q;
  const WigTab W = wig_tab(wtab, bw_in);
  const int b1 = bw_in + 1;
  const int n = 2 * bw_out;
  const int stride = (n + KB - 1) / KB;
  for (int i = threadIdx.x; i < nl; i += blockDim.x) {
    const int l = q + i;
    wig_factors(W, b1, p, q, l, &fa[2 * i], &fa[2 * i + 1], &gs[i]);
    float2 v[4];
    so3_coefs(fz, bw_in, p, q, l, (float)__ldg(&W.wl[l]), v);
#pragma unroll
    for (int u = 0; u < 4; ++u) cv[4 * i + u] = v[u];
  }
  const double lnorm = wig_lnorm(W, p, q);
  __syncthreads();
  for (int k0 = threadIdx.x; k0 < stride; k0 += blockDim.x) {
    double cb[KB], d0[KB], d1[KB];
    float2 acc[KB][4];
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      const int k = min(k0 + u * stride, n - 1);
      cb[u] = __ldg(&btab[k]);
      d0[u] = wig_seed(btab, n, k, lnorm, p, q);
      d1[u] = 0.0;
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = make_float2(0.f, 0.f);
    }
    int i = 0;
#pragma unroll 1
    for (; i + 1 < nl; i += 2) {
      const double2 ab0 = *reinterpret_cast<const double2*>(&fa[2 * i]);
      so3_step<KB>((const float4*)&cv[4 * i], ab0.x, ab0.y, gs[i], cb, d1, d0, acc);
      const double2 ab1 = *reinterpret_cast<const double2*>(&fa[2 * i + 2]);
      so3_step<KB>((const float4*)&cv[4 * i + 4], ab1.x, ab1.y, gs[i + 1], cb, d0, d1, acc);
    }
    if (i < nl) so3_step<KB>((const float4*)&cv[4 * i], 0.0, 0.0, 0.0, cb, d1, d0, acc);
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      const int k = k0 + u * stride;
      if (k < n) so3_store(S, n, p, q, k, acc[u]);
    }
  }
}

void so3_wigner_table(int bw_in, std::vector<double>& tab) {
  tab.assign(wigner_table_entries(bw_in), 0.0);
  const WigTab W = wig_tab(tab.data(), bw_in);
  const int b1 = bw_in + 1;
  double* s1 = const_cast<double*>(W.s1);
  double* r1 = const_cast<double*>(W.r1);
  for (int l = 0; l <= bw_in; ++l)
    for (int m = 0; m < l; ++m) {
      const double v = sqrt((double)l * l - (double)m * m);
      s1[l * b1 + m] = v;
      r1[l * b1 + m] = 1.0 / v;
    }
  for (int l = 0; l <= bw_in; ++l) {
    const double dl = l;
    const_cast<double*>(W.cl)[l] = sqrt((2 * dl + 3) / (2 * dl + 1)) * (dl + 1) * (2 * dl + 1);
    const_cast<double*>(W.el)[l] = l > 0 ? sqrt((2 * dl + 3) / (2 * dl - 1)) * (dl + 1) / dl : 0.0;
    const_cast<double*>(W.il)[l] = l > 0 ? 1.0 / (dl * (dl + 1)) : 0.0;
    const_cast<double*>(W.wl)[l] = 2.0 * M_PI * sqrt(2.0 / (2.0 * dl + 1.0));
    const_cast<double*>(W.lq)[l] = log((2.0 * dl + 1.0) / 2.0);
  }
  for (int k = 0; k < 2 * bw_in + 2; ++k) const_cast<double*>(W.lf)[k] = lgamma((double)k + 1.0);
}

void so3_beta_table(int bw_out, double* tab) {
  const int n = 2 * bw_out;
  for (int k = 0; k < n; ++k) {
    const double beta = M_PI * (2.0 * k + 1.0) / (4.0 * bw_out);
    tab[k] = cos(beta);
    tab[n + k] = log(cos(0.5 * beta));
    tab[2 * n + k] = log(sin(0.5 * beta));
  }
}

// Forward DFT over a (alpha) for one b and a tile of Wt = 2^LOG2W betas
// (8, 16 or 32: a tuned parameter, 16 by default), in place.  The first stage
// reads and the last writes S directly (fft_pass.cuh), so a tile crosses
// shared memory four times instead of eight (with the gamma transform below:
// n = 200 48 -> 37 us, n = 512 757 -> 470).  Per-component butterflies with
// compile-time plans: packed ones round the SO(3) volume differently, and one
// near-tied pair of the 256-pair batched workload then picked another bin under
// the tf32x3 synthesis than under FP32 and the FP64 oracle.
constexpr int kSo3FftAThreads = 320;
template <int NF, int LOG2W>
__global__ void __launch_bounds__(kSo3FftAThreads, NF > 0 ? 4 : 2)
    k_so3_fft_a(int bw_in, int bw_out, const __grid_constant__ So3Batch bt, const __grid_constant__ FftPlan plan) {
  chain_begin();
  extern __shared__ __align__(16) float2 tile[];  // [a][beta tile] | float4 cs[] (runtime plans)
  constexpr int Wt = 1 << LOG2W;
  const int n = NF > 0 ? NF : 2 * bw_out;
  const int Bo = n / 2;
  const int k0 = blockIdx.x * Wt, wt = min(Wt, n - k0);
  float2* S = bt.out[blockIdx.z].S + (size_t)blockIdx.y * n + k0;
  const size_t astride = (size_t)Bo * n;
  const int tid = threadIdx.x, nthr = blockDim.x;
  auto at = [=](int, int t, int i, int m) { return SmemCursor{tile + i * Wt + t, m * Wt, 0}; };
  auto ld = [=](int, int t, int i, int m) {
    const float2* p = S + (size_t)i * astride + t;
    const size_t js = (size_t)m * astride;
    const bool ok = t < wt;
    // rows with |m1| >= bw_in are not synthesised: read them as zero
    return [=](int, int j) {
      const int a = i + j * m;
      return ok && (a < bw_in || a > n - bw_in) ? p[j * js] : make_float2(0.f, 0.f);
    };
  };
  auto sv = [=](int, int t, int i, int m) {
    float2* p = S + (size_t)i * astride + t;
    const size_t js = (size_t)m * astride;
    const bool ok = t < wt;
    return [=](int, int j, float2 v) {
      if (ok) p[j * js] = v;
    };
  };
  const PassMap map{1, LOG2W};
  if constexpr (NF > 0)
    pass_ct<NF, false, 1, true, 0, -1, false>(map, plan.tw, tid, nthr, ld, at, sv);
  else
    pass_rt<false, 1, false>(plan, map, map, map, reinterpret_cast<float4*>(tile + (size_t)n * Wt), tid, nthr, ld, at, sv);
}

// Hermitian complex-to-real transform over gamma, |z|^2 and argmax: one alpha
// row position and kSo3Pairs pairs of betas.  Betas k and k + 1 are inverted by
// one complex transform of Z = X0 + i X1, whose output is x0 + i x1 since both
// spectra are Hermitian: X[b] = conj(u_b), X[n - b] = u_b for 0 < b < n/2; the
// DC term is taken real (its imaginary part only ever reaches the imaginary
// output, which the real transform discards) and the Nyquist term is zero.  A
// pair of betas is one 16-byte load.  The first inverse stage reads S directly
// (neighbouring threads take neighbouring pairs, 256 contiguous bytes), the
// last one's outputs go to the argmax without a shared round trip.
constexpr int kSo3Pairs = 16;
constexpr int kSo3C2rThreads = 320;
template <int NF>
__global__ void __launch_bounds__(kSo3C2rThreads, NF > 0 ? 3 : 2)
    k_so3_c2r(int bw_in, int bw_out, const __grid_constant__ So3Batch bt, const __grid_constant__ FftPlan plan) {
  chain_begin();
  extern __shared__ __align__(16) float2 zrow[];  // [kSo3Pairs][st] | float4 cs[] | int16 pos[n] (runtime plans)
  const int n = NF > 0 ? NF : 2 * bw_out;
  const int Bo = n / 2, st = n | 1;
  const So3Out& o = bt.out[blockIdx.z];
  const int r = blockIdx.y;  // alpha row position of the alpha transform's output
  const int k0 = blockIdx.x * 2 * kSo3Pairs;
  const int np = min(kSo3Pairs, (n - k0) / 2);  // n is even
  const int alpha = pos2freq<NF>(r, plan);
  const float2* Sr = o.S + (size_t)r * Bo * n + k0;
  const int tid = threadIdx.x, nthr = blockDim.x;
  // Z at gamma frequency k of beta pair pk (mir: k > n / 2, mirrored)
  auto zval = [=](int pk, int k, bool mir) -> float2 {
    const int b = mir ? n - k : k;
    if (b >= bw_in || b == Bo) return make_float2(0.f, 0.f);
    const float4 w = __ldg(reinterpret_cast<const float4*>(Sr + (size_t)b * n + 2 * pk));
    if (b == 0) return make_float2(w.x, w.z);
    return mir ? make_float2(w.x - w.w, w.y + w.z)   // u0 + i u1
               : make_float2(w.x + w.w, w.z - w.y);  // conj(u0) + i conj(u1)
  };
  const float K = (float)((1.0 / (double)n) * ((double)Bo / M_PI));
  float* volume = o.volume;
  // per thread: the largest value, the lowest index among equal ones (NaN
  // compares false); a volume whose first value is NaN has its peak there, as
  // for the reference's max_element
  float bv = -1.0f;
  uint32_t bi = 0xffffffffu;
  bool nan_first = false;
  if constexpr (NF > 0) {
    constexpr int cnt = FixedFft<NF>::count;
    constexpr int R = FixedFft<NF>::r[cnt - 1], nb = NF / R;
    for (int it = tid; it < kSo3Pairs * nb; it += nthr) {
      const int pk = it % kSo3Pairs, b = it / kSo3Pairs;
      if (pk >= np) continue;
      float2 x[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const bool below = 2 * (i * nb + nb - 1) < NF, above = 2 * i * nb > NF;
        const int k = b + i * nb;
        x[i] = zval(pk, k, above || (!below && 2 * k > NF));
      }
      dft_small<R, true>(x);
      float2* d = zrow + pk * st + fixed_freq2pos<NF>(b);
#pragma unroll
      for (int i = 0; i < R; ++i) d[i] = x[i];
    }
    __syncthreads();
    const int lwp = 32 - __clz(np - 1);
    auto at = [=](int g, int t, int i, int m) { return SmemCursor{zrow + (g + t) * st + i, m, 0}; };
    pass_ct<NF, true, 1, true, 1, cnt - 1>(PassMap{1, lwp}, plan.tw, tid, nthr, at, at, at);
    if constexpr (cnt > 2) __syncthreads();
    constexpr int R0 = FixedFft<NF>::r[0], m = NF / R0;
    for (int it = tid; it < np * m; it += nthr) {
      const int pk = it / m, j2 = it - pk * m;
      const float2* row = zrow + pk * st + j2;
      float2 x[R0];
#pragma unroll
      for (int j = 0; j < R0; ++j) x[j] = row[j * m];
#pragma unroll
      for (int k = 1; k < R0; ++k) x[k] = cmul(x[k], cconj(__ldg(plan.tw + j2 * k)));
      dft_small<R0, true>(x);
      const uint32_t idx = ((uint32_t)(k0 + 2 * pk) * n + (uint32_t)alpha) * n + j2;
      nan_first |= idx == 0 && isnan(x[0].x);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < R0; ++j) {
          const float v = (h ? x[j].y : x[j].x) * K, v2 = v * v;
          const uint32_t id = idx + h * (uint32_t)(n * n) + j * m;
          if (v2 > bv || (v2 == bv && id < bi)) {
            bv = v2;
            bi = id;
          }
          if (volume) volume[id] = v2;
        }
    }
  } else {
    float4* cs = reinterpret_cast<float4*>(zrow + (size_t)kSo3Pairs * st);
    short* pos = reinterpret_cast<short*>(cs + kMaxGenericRadix);
    for (int k = tid; k < n; k += nthr) pos[k] = (short)freq2pos<NF>(k, plan);
    __syncthreads();
    for (int it = tid; it < kSo3Pairs * (Bo + 1); it += nthr) {
      const int pk = it % kSo3Pairs, b = it / kSo3Pairs;
      if (pk >= np) continue;
      zrow[pk * st + pos[b]] = zval(pk, b, false);
      if (b > 0 && b < Bo) zrow[pk * st + pos[n - b]] = zval(pk, n - b, true);
    }
    __syncthreads();
    const int lwp = 32 - __clz(np - 1);
    auto at = [=](int g, int t, int i, int m) { return SmemCursor{zrow + (g + t) * st + i, m, 0}; };
    auto sv = [=, &bv, &bi, &nan_first](int g, int t, int i, int m) {
      const uint32_t idx = ((uint32_t)(k0 + 2 * (g + t)) * n + (uint32_t)alpha) * n + i;
      return [=, &bv, &bi, &nan_first](int, int j, float2 z) {
        nan_first |= idx == 0 && j == 0 && isnan(z.x);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float v = (h ? z.y : z.x) * K, v2 = v * v;
          const uint32_t id = idx + h * (uint32_t)(n * n) + j * m;
          if (v2 > bv || (v2 == bv && id < bi)) {
            bv = v2;
            bi = id;
          }
          if (volume) volume[id] = v2;
        }
      };
    };
    pass_rt<true, 1, true>(plan, PassMap{1, lwp}, PassMap{1, lwp}, PassMap{np, 0}, cs, tid, nthr, at, at, sv);
  }
  if (nan_first) {
    bv = __int_as_float(0x7fffffff);  // orders above every number
    bi = 0;
  }
  warp_argmax_commit(bi == 0xffffffffu ? 0ull : pack_argmax(bv, bi), o.argmax);
}

static bool so3_fixed_length(int n) {
  bool fixed = false;
  PHGPU_DISPATCH_N(n, fixed = NF > 0);
  return fixed;
}
// Shared memory beyond the tile: the prime-radix scratch of runtime plans.
static size_t so3_prime_scratch(int n) { return so3_fixed_length(n) ? 0 : kMaxGenericRadix * sizeof(float4); }

template <int NF>
static cudaError_t so3_attrs() {
  const int m = 227 * 1024;
  cudaError_t e = cudaFuncSetAttribute(k_so3_fft_a<NF, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_so3_fft_a<NF, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_so3_fft_a<NF, 5>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_so3_c2r<NF>, cudaFuncAttributeMaxDynamicSharedMemorySize, m);
  return e;
}

cudaError_t so3_init_attributes(int n) {
  cudaError_t e = cudaSuccess;
  PHGPU_DISPATCH_N(n, e = so3_attrs<NF>());
  if (e == cudaSuccess) e = so3_tc_init_attributes();
  return e;
}

cudaError_t launch_so3_synth(const So3Args& a, cudaStream_t st) {
  if (a.batch.count < 1 || a.batch.count > kMaxWave) return cudaErrorInvalidValue;
  const int ncls = a.bw_in * (a.bw_in + 1) / 2;
  const int n = 2 * a.bw_out;
  // betas per thread: the largest share of busy lanes, the smaller count where it is as good (fewer registers)
  int kb = 0, thr = 0;
  double best = 0.0;
  for (int c : {2, 4, 5, 7}) {
    const int stride = (n + c - 1) / c;
    const int rounds = (stride + kSynthThreads - 1) / kSynthThreads;
    const int t = ((stride + rounds - 1) / rounds + 31) / 32 * 32;
    const double busy = (double)n / ((double)t * rounds * c);
    if (busy > best + 0.02 && (c > 2 || n <= 64)) {
      best = busy;
      kb = c;
      thr = t;
    }
  }
  const size_t sm = (size_t)(a.bw_in * 3 + 1) * sizeof(double) + (size_t)a.bw_in * 4 * sizeof(float2);
  auto fn = kb == 2 ? k_so3_synth<2> : (kb == 4 ? k_so3_synth<4> : (kb == 5 ? k_so3_synth<5> : k_so3_synth<7>));
  launch_kernel(fn, dim3(ncls, a.batch.count), dim3(thr), sm, st, a.bw_in, a.bw_out, a.batch, a.beta_tab, a.wig_tab);
  count_launches(1);
  return cudaGetLastError();
}

template <int NF>
static void launch_so3_c2r(const So3Args& a, int n, cudaStream_t st) {
  const dim3 g((n + 2 * kSo3Pairs - 1) / (2 * kSo3Pairs), n, a.batch.count);
  size_t sm = (size_t)kSo3Pairs * (n | 1) * sizeof(float2);
  if (NF == 0) sm += so3_prime_scratch(n) + (size_t)n * sizeof(short);  // fits up to n = 1770
  const int thr = NF > 0 ? pass_threads(*a.plan, kSo3Pairs, 1, 160, kSo3C2rThreads)
                         : pass_threads(*a.plan, kSo3Pairs, 1, 128, kSo3C2rThreads, 96, sm);
  launch_kernel(k_so3_c2r<NF>, dim3(g), dim3(thr), sm, st, a.bw_in, a.bw_out, a.batch, *a.plan);
}

template <int NF>
static void launch_so3_fft_a(const So3Args& a, int n, int wt, cudaStream_t st) {
  const dim3 g((n + wt - 1) / wt, a.bw_in, a.batch.count);
  const size_t sm = (size_t)n * wt * sizeof(float2) + so3_prime_scratch(n);
  const int thr = NF > 0 ? pass_threads(*a.plan, wt, 1, 160, kSo3FftAThreads)
                         : pass_threads(*a.plan, wt, 1, 128, kSo3FftAThreads, 96, sm);
  if (wt == 8)
    launch_kernel(k_so3_fft_a<NF, 3>, dim3(g), dim3(thr), sm, st, a.bw_in, a.bw_out, a.batch, *a.plan);
  else if (wt == 32)
    launch_kernel(k_so3_fft_a<NF, 5>, dim3(g), dim3(thr), sm, st, a.bw_in, a.bw_out, a.batch, *a.plan);
  else
    launch_kernel(k_so3_fft_a<NF, 4>, dim3(g), dim3(thr), sm, st, a.bw_in, a.bw_out, a.batch, *a.plan);
}

bool so3_beta_tile_ok(int bw_out, int wt) {
  return (wt == 8 || wt == 16 || wt == 32) &&
         (size_t)2 * bw_out * wt * sizeof(float2) + so3_prime_scratch(2 * bw_out) <= 227u * 1024u;
}

cudaError_t launch_so3_fft(const So3Args& a, cudaStream_t st) {
  if (a.batch.count < 1 || a.batch.count > kMaxWave) return cudaErrorInvalidValue;
  const int n = 2 * a.bw_out;
  const int wt = so3_beta_tile_ok(a.bw_out, a.beta_tile) ? a.beta_tile : 16;
  PHGPU_DISPATCH_N(n, launch_so3_fft_a<NF>(a, n, wt, st); launch_so3_c2r<NF>(a, n, st));
  count_launches(2);
  return cudaGetLastError();
}

}  // namespace phgpu
