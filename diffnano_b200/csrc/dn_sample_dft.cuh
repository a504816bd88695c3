// Monitors of the resident runs: running DFTs from stored samples, and what
// monitors add to lambda in the reverse sweep.
#pragma once

#include "dn_common.cuh"

namespace dn {
namespace res {

// ---- monitors ------------------------------------------------------------------
// The march only stores each step's values of a monitor's cells (samples, the
// grid's type); their running DFT is added to the monitor's FP64 sums by a
// kernel of its own after the run, which keeps FP64 arithmetic and its
// registers out of the step every other warp waits for.
//
// sums[f][cell] += sum_t sample[t][cell] phase[t][f]: a block owns 32 cells, its
// warps take every DFT_WARPS-th step, and the partial sums are added in warp
// order (deterministic).
constexpr int DFT_WARPS = 16;
constexpr int DFT_FREQS = 4;  // frequencies per pass
template <typename T>
__device__ __forceinline__ void sample_dft(const T* __restrict__ smp, long long step_stride,
                                           int nsteps, long long ncell,
                                           const double* __restrict__ phase, int nf,
                                           double* __restrict__ acc) {
  __shared__ double2 part[DFT_WARPS][DFT_FREQS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long cell = (long long)blockIdx.x * 32 + lane;
  const bool ok = cell < ncell;
  for (int f0 = 0; f0 < nf; f0 += DFT_FREQS) {
    double2 s[DFT_FREQS];
#pragma unroll
    for (int f = 0; f < DFT_FREQS; ++f) s[f] = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int t = w; t < nsteps; t += DFT_WARPS) {
      const double x = ok ? static_cast<double>(smp[t * step_stride + cell]) : 0.0;
      const double* ph = phase + ((long long)t * nf + f0) * 2;
#pragma unroll
      for (int f = 0; f < DFT_FREQS; ++f)
        if (f0 + f < nf) {
          s[f].x = fma(x, __ldg(ph + 2 * f), s[f].x);
          s[f].y = fma(x, __ldg(ph + 2 * f + 1), s[f].y);
        }
    }
#pragma unroll
    for (int f = 0; f < DFT_FREQS; ++f) part[w][f][lane] = s[f];
    __syncthreads();
    for (int e = threadIdx.x; e < DFT_FREQS * 32; e += blockDim.x) {
      const int f = e / 32, l = e % 32;
      const long long c = (long long)blockIdx.x * 32 + l;
      if (f0 + f < nf && c < ncell) {
        double2 u = make_double2(0.0, 0.0);
#pragma unroll
        for (int v = 0; v < DFT_WARPS; ++v) {
          u.x += part[v][f][l].x;
          u.y += part[v][f][l].y;
        }
        double* a = acc + ((long long)(f0 + f) * ncell + c) * 2;
        a[0] += u.x;
        a[1] += u.y;
      }
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(DFT_WARPS * 32)
    k_sample_dft(const T* smp, long long step_stride, int nsteps, long long ncell,
                 const double* phase, int nf, double* acc, const int* status) {
  if (status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0) return;
  sample_dft<T>(smp, step_stride, nsteps, ncell, phase, nf, acc);
}

// what a monitor adds to lambda before reverse step t: the sum over its
// frequencies of (gradient of the DFT) . phase
template <typename T>
__device__ __forceinline__ T add_of(long long cell, long long ncell, long long t,
                                    const double* __restrict__ phase, int nf,
                                    const double* __restrict__ g) {
  const double* ph = phase + t * nf * 2;
  double s = 0.0;
  for (int f = 0; f < nf; ++f) {
    const double* a = g + ((long long)f * ncell + cell) * 2;
    s = fma(a[0], __ldg(ph + 2 * f), fma(a[1], __ldg(ph + 2 * f + 1), s));
  }
  return static_cast<T>(s);
}

}  // namespace res
}  // namespace dn
