// Test-only library (built by tests/test_gpu_pass_engine.py, linked against the
// product library for the plans): phgpu_selftest_pass(n, ntrans, inverse, mode,
// order, data) transforms ntrans sequences of length n (complex interleaved,
// natural order, in place in `data`) with the passes of fft_pass.cuh, each
// sequence a column of a shared tile.  mode 0: compile-time plan; 1: runtime plan in radix
// order `order`, first and last stage through global memory; 2: the same on
// data already in shared memory; 3: two sequences of a column in one item.
// Forward = exp(-2 pi i jk/n), inverse = exp(+2 pi i jk/n), both unnormalised.
#include <cuda_runtime.h>

#include <string>

#include "phaser_gpu.h"
#include "fft_pass.cuh"
#include "kernels.h"

namespace phgpu {
bool make_fft_plan(int n, FftPlan* p, float2** d_tw, std::string* err);
bool fft_plan_radices(int n, int order, FftPlan* p);

constexpr int kThreads = 128;
constexpr int kLog2W = 2;

// One block per 2^kLog2W sequences (mode 3: 2^(kLog2W + 1), 2 t and 2 t + 1 in column t).
template <int NF, bool INV, int MODE>
__global__ void __launch_bounds__(kThreads) k_selftest_pass(int n, int ntrans, const float2* __restrict__ in,
                                                            float2* __restrict__ out, const __grid_constant__ FftPlan p) {
  extern __shared__ __align__(16) float2 tile[];  // [NG][n][W] | float4 cs[]
  constexpr int W = 1 << kLog2W, NG = MODE == 3 ? 2 : 1;
  const int slot = n * W, tid = threadIdx.x, first = blockIdx.x * W * NG;
  float4* cs = reinterpret_cast<float4*>(tile + NG * slot);
  auto at = [=](int, int t, int i, int m) { return SmemCursor{tile + i * W + t, m * W, slot}; };
  auto freq = [&](int pos) { return pos2freq<NF>(pos, p); };
  auto ld = [&](int, int t, int i, int m) {
    return [=, &freq](int g, int j) {
      const int k = i + j * m, s = first + NG * t + g;
      return s < ntrans ? in[(size_t)s * n + (INV ? freq(k) : k)] : make_float2(0.f, 0.f);
    };
  };
  auto sv = [&](int, int t, int i, int m) {
    return [=, &freq](int g, int j, float2 v) {
      const int k = i + j * m, s = first + NG * t + g;
      if (s < ntrans) out[(size_t)s * n + (INV ? k : freq(k))] = v;
    };
  };
  const PassMap map{1, kLog2W};
  if constexpr (NF > 0) {
    pass_ct<NF, INV, NG, true, 0, -1>(map, p.tw, tid, kThreads, ld, at, sv);
  } else if constexpr (MODE == 2) {
    for (int e = tid; e < slot; e += kThreads) tile[e] = ld(0, e & (W - 1), e >> kLog2W, 1)(0, 0);
    __syncthreads();
    pass_rt<INV, NG, true>(p, map, map, map, cs, tid, kThreads, at, at, sv);
  } else {
    pass_rt<INV, NG, false>(p, map, map, map, cs, tid, kThreads, ld, at, sv);
  }
}

template <int NF, int MODE>
static cudaError_t run(int n, int ntrans, int inverse, const float2* in, float2* out, const FftPlan& p) {
  const int per = (MODE == 3 ? 2 : 1) << kLog2W;
  const size_t sm = (size_t)per * n * sizeof(float2) + kMaxGenericRadix * sizeof(float4);
  auto fn = inverse ? k_selftest_pass<NF, true, MODE> : k_selftest_pass<NF, false, MODE>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  fn<<<(ntrans + per - 1) / per, kThreads, sm>>>(n, ntrans, in, out, p);
  return cudaGetLastError();
}

}  // namespace phgpu

using namespace phgpu;

extern "C" int phgpu_selftest_pass(int n, int ntrans, int inverse, int mode, int order, float* data) {
  if (n < 1 || n > 1024 || ntrans < 1 || !data || mode < 0 || mode > 3) return PHGPU_ERR_INVALID;
  FftPlan p;
  float2* tw = nullptr;
  std::string err;
  if (!make_fft_plan(n, &p, &tw, &err)) return PHGPU_ERR_INVALID;
  const size_t bytes = sizeof(float2) * (size_t)n * ntrans;
  float2 *in = nullptr, *out = nullptr;
  cudaError_t e = cudaMalloc(&in, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&out, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(in, data, bytes, cudaMemcpyHostToDevice);
  if (mode > 0) fft_plan_radices(n, order, &p);
  if (e == cudaSuccess) {
    e = cudaErrorInvalidValue;
    if (mode == 1) e = run<0, 1>(n, ntrans, inverse, in, out, p);
    if (mode == 2) e = run<0, 2>(n, ntrans, inverse, in, out, p);
    if (mode == 3) e = run<0, 3>(n, ntrans, inverse, in, out, p);
    if (mode == 0) PHGPU_DISPATCH_N(n, if (NF > 0) e = run<NF, 0>(n, ntrans, inverse, in, out, p));
  }
  if (e == cudaSuccess) e = cudaMemcpy(data, out, bytes, cudaMemcpyDeviceToHost);
  cudaFree(in);
  cudaFree(out);
  cudaFree(tw);
  return e == cudaSuccess ? PHGPU_OK : PHGPU_ERR_CUDA;
}
