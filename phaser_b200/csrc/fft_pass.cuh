// FFT passes whose first stage reads, and whose last stage writes, through a
// caller's functor (global memory, fused arithmetic) instead of through
// shared memory, for columns of a shared tile.
//
// A transform of S stages through shared memory alone moves every element
// 2 S + 2 times between registers and shared memory (load, S in-place stages,
// store); with the first and last stage fused to the global accesses it is
// 2 S - 2 times, and the loads of a whole radix butterfly are in flight per
// thread.  The plans, positions and butterflies are those of fft.cuh: forward
// transforms (decimation in frequency) leave digit-reversed order, inverse
// transforms consume it.
#pragma once

#include "fft.cuh"

namespace phgpu {

// Geometry of one stage: radix R, block length L, m = L / R, nb = n / R
// butterflies per transform, twiddle step n / L.
template <int NF, int S>
struct StageC {
  static constexpr int R = FixedFft<NF>::r[S];
  static constexpr int Lc = fixed_L<NF, S>();
  __device__ __forceinline__ int L() const { return Lc; }
  __device__ __forceinline__ int m() const { return Lc / R; }
  __device__ __forceinline__ int nb() const { return NF / R; }
  __device__ __forceinline__ int twstep() const { return NF / Lc; }
  __device__ __forceinline__ int div_m(int x) const { return S == 0 ? 0 : x / (Lc / R); }  // S = 0: one block
  __device__ __forceinline__ int div_nb(int x) const { return x / (NF / R); }
};
struct StageR {
  int Lv, mv, nbv, tws;
  uint32_t qm, qnb;
  __device__ __forceinline__ StageR(const FftPlan& p, int s)
      : Lv(p.L[s]), mv(p.L[s] / p.radix[s]), nbv(p.n / p.radix[s]), tws(p.n / p.L[s]), qm(p.mul_m[s]),
        qnb(p.mul_nb[s]) {}
  __device__ __forceinline__ int L() const { return Lv; }
  __device__ __forceinline__ int m() const { return mv; }
  __device__ __forceinline__ int nb() const { return nbv; }
  __device__ __forceinline__ int twstep() const { return tws; }
  __device__ __forceinline__ int div_m(int x) const { return fast_div(x, qm); }
  __device__ __forceinline__ int div_nb(int x) const { return fast_div(x, qnb); }
};

// How a stage's transforms map to threads: item = (group * nb + butterfly) *
// 2^lw + column, columns fastest over the threads.  ONE: groups = 1.
struct PassMap {
  int groups, lw;
};

// Cursors: how a stage reaches the elements r0, r0 + m, ... of the NG
// transforms that share one item's butterfly (the channels of one column).
// ld(group, column, r0, m) returns a callable (g, j) -> value and sv(group,
// column, r0, m) a callable (g, j, value), so an item's addresses are formed
// once and its NG * R elements follow at constant strides.
struct SmemCursor {
  float2* p;
  int es;  // between elements r0 + j m and r0 + (j + 1) m
  int gs;  // between transforms g and g + 1
  __device__ __forceinline__ float2 operator()(int g, int j) const { return p[g * gs + j * es]; }
  __device__ __forceinline__ void operator()(int g, int j, float2 v) const { p[g * gs + j * es] = v; }
};

// One radix-R stage of NG * groups * 2^lw transforms.  The NG transforms of an
// item share its index arithmetic and twiddles.  PK: packed butterflies
// (dft_small).
template <int R, bool INV, int NG, bool ONE, bool PK = true, class G, class Ld, class Sv>
__device__ __forceinline__ void pass_stage(const G g, PassMap map, const float2* __restrict__ tw, int tid, int nthr,
                                           Ld ld, Sv sv) {
  const int m = g.m();
  const int nitems = ((ONE ? 1 : map.groups) * g.nb()) << map.lw;
  for (int it = tid; it < nitems; it += nthr) {
    const int t = it & ((1 << map.lw) - 1);
    const int q = it >> map.lw;
    const int grp = ONE ? 0 : g.div_nb(q);
    const int bf = q - grp * g.nb();
    const int blk = g.div_m(bf);
    const int j2 = bf - blk * m;
    const int r0 = blk * g.L() + j2;
    const int ws = g.twstep() * j2;
    [[maybe_unused]] float2 w[R];
    if constexpr (NG > 1) {
      if (m > 1) {
#pragma unroll
        for (int k = 1; k < R; ++k) w[k] = __ldg(tw + ws * k);
      }
    }
    auto twiddle = [&](float2 v, int k) {
      const float2 f = NG > 1 ? w[k] : __ldg(tw + ws * k);
      return cmul(v, INV ? cconj(f) : f);
    };
    const auto lc = ld(grp, t, r0, m);
    const auto sc = sv(grp, t, r0, m);
#pragma unroll
    for (int u = 0; u < NG; ++u) {
      float2 x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = lc(u, j);
      if constexpr (INV) {
        if (m > 1) {
#pragma unroll
          for (int k = 1; k < R; ++k) x[k] = twiddle(x[k], k);
        }
        dft_small<R, true, PK>(x);
      } else {
        dft_small<R, false, PK>(x);
        if (m > 1) {
#pragma unroll
          for (int k = 1; k < R; ++k) x[k] = twiddle(x[k], k);
        }
      }
#pragma unroll
      for (int j = 0; j < R; ++j) sc(u, j, x[j]);
    }
  }
}

// Stage s of a runtime plan (radices with a register butterfly only).
template <bool INV, int NG, class Ld, class Sv>
__device__ __forceinline__ void pass_stage_rt(const FftPlan& p, int s, PassMap map, int tid, int nthr, Ld ld, Sv sv) {
  const StageR g(p, s);
  switch (p.radix[s]) {
    case 2: pass_stage<2, INV, NG, false>(g, map, p.tw, tid, nthr, ld, sv); break;
    case 3: pass_stage<3, INV, NG, false>(g, map, p.tw, tid, nthr, ld, sv); break;
    case 4: pass_stage<4, INV, NG, false>(g, map, p.tw, tid, nthr, ld, sv); break;
    case 5: pass_stage<5, INV, NG, false>(g, map, p.tw, tid, nthr, ld, sv); break;
    case 7: pass_stage<7, INV, NG, false>(g, map, p.tw, tid, nthr, ld, sv); break;
    default: pass_stage<8, INV, NG, false>(g, map, p.tw, tid, nthr, ld, sv); break;
  }
}

// Stage with an odd prime radix above the register butterflies (11..127, e.g.
// 201 = 3 * 67), in place in shared memory (at: a SmemCursor maker).
//
// With s_j = x_j + x_{R-j} and d_j = x_j - x_{R-j} (written in place first),
//   A_k = x_0 + sum_j cos(2 pi j k / R) s_j,   B_k = sum_j sin(2 pi j k / R) d_j,
//   X_k, X_{R-k} = A_k -+ i B_k (forward; +- inverse),   j, k = 1 .. (R-1)/2,
// a quarter of the products of the plain sum, each a packed pair times a real
// constant (one FFMA2).  A work item is kPrimeOuts values of k for kPrimeBfs
// butterflies; items of whole butterflies are summed in rounds of one item
// per thread, since the outputs overwrite the inputs (z pass of N = 201: 1065 us
// with plain complex sums, 388 so).  cs: shared scratch of R
// float4 (cos, cos, sin, sin), filled here.  Every thread must call it; it
// begins after a barrier of the caller's and ends with one.
constexpr int kPrimeOuts = 4;
constexpr int kPrimeBfs = 2;

template <bool INV, int NG, class At>
__device__ __noinline__ void pass_prime(const FftPlan& p, int s, PassMap map, float4* cs, int tid, int nthr, At at) {
  const StageR g(p, s);
  const int R = p.radix[s], h = (R - 1) / 2, m = g.m();
  const int nbf = (map.groups * NG * g.nb()) << map.lw;
  const int rstep = p.n / R;
  // butterfly b of the NG * groups * 2^lw transforms, as a cursor of its own
  auto locate = [=](int b, int& j2) {
    const int t = b & ((1 << map.lw) - 1);
    const int q = b >> map.lw;
    const int gg = g.div_nb(q);
    const int bf = q - gg * g.nb();
    const int blk = g.div_m(bf);
    j2 = bf - blk * m;
    SmemCursor c = at(gg / NG, t, blk * g.L() + j2, m);
    c.p += (gg % NG) * c.gs;
    return c;
  };
  for (int j = tid; j < R; j += nthr) {
    const float2 w = __ldg(&p.tw[rstep * j]);  // (cos, -sin)
    cs[j] = make_float4(w.x, w.x, -w.y, -w.y);
  }
  // sums and differences (after the inverse stage's twiddles)
  for (int it = tid; it < nbf * h; it += nthr) {
    const int j = it / nbf + 1, b = it - (j - 1) * nbf;
    int j2;
    const SmemCursor c = locate(b, j2);
    float2 u = c(0, j), v = c(0, R - j);
    if (INV && m > 1) {
      u = cmul(u, cconj(__ldg(&p.tw[g.twstep() * j2 * j])));
      v = cmul(v, cconj(__ldg(&p.tw[g.twstep() * j2 * (R - j)])));
    }
    c(0, j, cadd(u, v));
    c(0, R - j, csub(u, v));
  }
  __syncthreads();
  const int ng = (h + kPrimeOuts - 1) / kPrimeOuts;
  const int nbg = (nbf + kPrimeBfs - 1) / kPrimeBfs;
  const int per_round = max(1, nthr / ng);
  for (int g0 = 0; g0 < nbg; g0 += per_round) {
    const int nloc = min(per_round, nbg - g0);
    const bool active = tid < nloc * ng;
    const int kg = active ? tid / nloc : 0;
    const int b0 = g0 + tid - kg * nloc;
    float2 A[kPrimeBfs][kPrimeOuts], B[kPrimeBfs][kPrimeOuts], sum[kPrimeBfs];
    SmemCursor cur[kPrimeBfs];
    int j2[kPrimeBfs];
    const int k0 = 1 + kg * kPrimeOuts;
    if (active) {
#pragma unroll
      for (int u = 0; u < kPrimeBfs; ++u) {
        const int b = b0 + u * nbg;
        cur[u] = locate(b < nbf ? b : b0, j2[u]);
        sum[u] = cur[u](0, 0);
#pragma unroll
        for (int i = 0; i < kPrimeOuts; ++i) {
          A[u][i] = sum[u];
          B[u][i] = make_float2(0.f, 0.f);
        }
      }
      int idx[kPrimeOuts], kk[kPrimeOuts];
#pragma unroll
      for (int i = 0; i < kPrimeOuts; ++i) {
        kk[i] = k0 + i <= h ? k0 + i : 0;
        idx[i] = 0;
      }
      for (int j = 1; j <= h; ++j) {
        float2 sj[kPrimeBfs], dj[kPrimeBfs];
#pragma unroll
        for (int u = 0; u < kPrimeBfs; ++u) {
          sj[u] = cur[u](0, j);
          dj[u] = cur[u](0, R - j);
          sum[u] = cadd(sum[u], sj[u]);
        }
#pragma unroll
        for (int i = 0; i < kPrimeOuts; ++i) {
          idx[i] += kk[i];
          if (idx[i] >= R) idx[i] -= R;
          const float4 w = cs[idx[i]];
#pragma unroll
          for (int u = 0; u < kPrimeBfs; ++u) {
            A[u][i] = __ffma2_rn(make_float2(w.x, w.y), sj[u], A[u][i]);
            B[u][i] = __ffma2_rn(make_float2(w.z, w.w), dj[u], B[u][i]);
          }
        }
      }
    }
    __syncthreads();
    if (active) {
#pragma unroll
      for (int u = 0; u < kPrimeBfs; ++u) {
        if (b0 + u * nbg >= nbf) continue;
        if (kg == 0) cur[u](0, 0, sum[u]);
#pragma unroll
        for (int i = 0; i < kPrimeOuts; ++i) {
          const int k = k0 + i;
          if (k > h) continue;
          float2 xk, xr;
          rot_pm<INV>(A[u][i], B[u][i], xk, xr);
          if (!INV && m > 1) {
            xk = cmul(xk, __ldg(&p.tw[g.twstep() * j2[u] * k]));
            xr = cmul(xr, __ldg(&p.tw[g.twstep() * j2[u] * (R - k)]));
          }
          cur[u](0, k, xk);
          cur[u](0, R - k, xr);
        }
      }
    }
    __syncthreads();
  }
}

// Stages [I0, I1) of a transform in execution order (forward: first radix
// first; inverse: last radix first) over NG * groups * 2^lw transforms: stage 0
// reads through ld, the last stage of the plan writes through sv, everything
// between goes through at (shared memory; ld / sv may be at as well).  I1 < 0:
// up to the plan's last stage.  A barrier separates the stages; the caller
// synchronises before reading what sv wrote.  ONE: map.groups = 1.
template <int NF, bool INV, int NG, bool ONE, int I0, int I1, bool PK = true, class Ld, class At, class Sv>
__device__ __forceinline__ void pass_ct(PassMap map, const float2* __restrict__ tw, int tid, int nthr, Ld ld, At at,
                                        Sv sv) {
  constexpr int cnt = FixedFft<NF>::count;
  constexpr int end = I1 < 0 ? cnt : I1;
  if constexpr (I0 < end) {
    constexpr int S = INV ? cnt - 1 - I0 : I0;
    using G = StageC<NF, S>;
    const G g;
    if constexpr (I0 == 0 && cnt == 1) {
      pass_stage<G::R, INV, NG, ONE, PK>(g, map, tw, tid, nthr, ld, sv);
    } else if constexpr (I0 == 0) {
      pass_stage<G::R, INV, NG, ONE, PK>(g, map, tw, tid, nthr, ld, at);
    } else if constexpr (I0 == cnt - 1) {
      pass_stage<G::R, INV, NG, ONE, PK>(g, map, tw, tid, nthr, at, sv);
    } else {
      pass_stage<G::R, INV, NG, ONE, PK>(g, map, tw, tid, nthr, at, at);
    }
    if constexpr (I0 + 1 < end) __syncthreads();
    pass_ct<NF, INV, NG, ONE, I0 + 1, end, PK>(map, tw, tid, nthr, ld, at, sv);
  }
}

// The whole transform on a runtime plan: prime stages work in place in shared
// memory, so a plan that begins (ends) with one is loaded (stored) by a plain
// pass.  `first` maps the loads, `last` the final stores, `mid` the stages
// between (rows of a tile load and store with neighbouring threads along the
// row, but run their shared stages across rows).  LOADED: the data is in
// shared memory already and ld is not called.  cs: shared scratch for
// pass_prime (kMaxGenericRadix float4), unused without prime stages.
template <bool INV, int NG, bool LOADED, class Ld, class At, class Sv>
__device__ __forceinline__ void pass_rt(const FftPlan& p, PassMap first, PassMap mid, PassMap last, float4* cs, int tid,
                                        int nthr, Ld ld, At at, Sv sv) {
  const int cnt = p.nstage;
  auto radix = [&](int i) { return p.radix[INV ? cnt - 1 - i : i]; };
  const bool load = !LOADED && (cnt <= 1 || radix(0) > kMaxRegRadix);
  const bool store = cnt <= 1 || radix(cnt - 1) > kMaxRegRadix;
  if (load) {
    for (int q = tid >> first.lw, t = tid & ((1 << first.lw) - 1); q < first.groups * p.n; q += nthr >> first.lw) {
      const int a = first.groups == 1 ? 0 : q / p.n, i = q - a * p.n;
      const auto c = ld(a, t, i, 1);
      const SmemCursor d = at(a, t, i, 1);
#pragma unroll
      for (int u = 0; u < NG; ++u) d(u, 0, c(u, 0));
    }
    __syncthreads();
  }
  for (int i = 0; i < cnt; ++i) {
    const int s = INV ? cnt - 1 - i : i;
    if (p.radix[s] > kMaxRegRadix) {
      pass_prime<INV, NG>(p, s, mid, cs, tid, nthr, at);
      continue;
    }
    if (!LOADED && i == 0 && !load)
      pass_stage_rt<INV, NG>(p, s, first, tid, nthr, ld, at);
    else if (i == cnt - 1 && !store)
      pass_stage_rt<INV, NG>(p, s, last, tid, nthr, at, sv);
    else
      pass_stage_rt<INV, NG>(p, s, mid, tid, nthr, at, at);
    if (i + 1 < cnt || store) __syncthreads();
  }
  if (store) {
    for (int q = tid >> last.lw, t = tid & ((1 << last.lw) - 1); q < last.groups * p.n; q += nthr >> last.lw) {
      const int a = last.groups == 1 ? 0 : q / p.n, i = q - a * p.n;
      const SmemCursor d = at(a, t, i, 1);
      const auto c = sv(a, t, i, 1);
#pragma unroll
      for (int u = 0; u < NG; ++u) c(u, 0, d(u, 0));
    }
  }
}

// Threads per block (a multiple of 32 in [lo, hi]) of a pass over `cols` items
// per butterfly, each of ng transforms (host).  With regs == 0 (compile-time
// plans) the ones that leave the fewest threads idle in the plan's stages.
// Runtime plans hold 80 to 96 registers a thread and wait for most of their
// time, so theirs is that time over the threads resident on an SM (`regs` a
// thread, `smem` bytes a block): blocks of 5 or 7 warps leave one of the four
// register files short.  The z pass of n = 100 takes 33 us with 128 threads, 46
// with 160, 41 with 256; the fewest idle threads alone took 84 us at n = 110
// and 214 at n = 180, now 58 and 162.
inline int pass_threads(const FftPlan& p, int cols, int ng_item, int lo, int hi, int regs = 0, size_t smem = 0) {
  int best = lo;
  double best_cost = 1e300;
  for (int t = lo; t <= hi; t += 32) {
    double cost = 0.0;
    for (int s = 0; s < p.nstage; ++s) {
      const int R = p.radix[s];
      if (R > kMaxRegRadix) {
        const int h = (R - 1) / 2, ng = (h + kPrimeOuts - 1) / kPrimeOuts;
        const int nbg = (cols * ng_item * (p.n / R) + kPrimeBfs - 1) / kPrimeBfs;
        const int per = t / ng > 0 ? t / ng : 1;
        cost += (double)((nbg + per - 1) / per) * t * h * 4.0 / ng_item;
      } else {
        const int items = cols * (p.n / R);
        cost += (double)((items + t - 1) / t) * t * R;
      }
    }
    if (regs > 0) {
      const int by_regs = 4 * (65536 / 4 / (regs * 32)) / (t / 32), by_smem = (int)((size_t)(228 * 1024) / (smem + 1024));
      const int blocks = by_regs < by_smem ? by_regs : by_smem;
      cost /= (blocks > 0 ? blocks : 1) * t;
    }
    // ties and near-ties of the idle threads: the larger block (fewer rounds between barriers)
    if (cost <= best_cost * (regs > 0 ? 0.9999 : 1.0001)) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}

}  // namespace phgpu
