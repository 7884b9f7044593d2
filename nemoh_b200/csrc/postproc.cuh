// Radiation impulse response functions of the post-processor
// (postProcessor/IRF.f90:100-127, Compute_IRF):
//   K(t_i) = 2/pi sum_l 0.5 (B_l cos(w_l t_i) + B_l+1 cos(w_l+1 t_i)) (w_l+1 - w_l)
//   A_inf  = 1/Nw sum_l [A_l + 1/w_l sum_i 0.5 (K_i sin(w_l t_i) + K_i+1 sin(w_l t_i+1)) dt]
// with t_i = i dt. Coefficients are (Nw, Nrad, Nint) with w fastest, K is
// (Ntime, Nrad, Nint) with time fastest. A thread of K owns one time and up to
// IRF_CH radiation/force pairs; a CTA of the added mass owns one frequency and
// IRF_CH pairs and its threads take the times in turn: per pair chunk a cosine is
// evaluated once and the sine of an inner time twice (as either end of a trapezium).
// A serial sum over 1,000 times by one thread per
// frequency was 1,580 us at 40 frequencies x 36 pairs (one CTA per chunk, each
// step behind the last one's latency): now 17 us,
// and K 66 to 24 us with 4 pairs a chunk instead of 16 (1,000 times).
#pragma once
#include "common.cuh"

namespace nb200 {

constexpr int IRF_CH = 4;
constexpr int IRF_THREADS = 128;

// K: a CTA per 128 times and pair chunk, the chunk fastest
__global__ void __launch_bounds__(IRF_THREADS)
    irf_kernel(int nw, const double* __restrict__ w, int npair, const double* __restrict__ damping, int ntime,
               double dt, double* __restrict__ K) {
  const int chunks = (npair + IRF_CH - 1) / IRF_CH;
  const int i = blockIdx.x / chunks * IRF_THREADS + threadIdx.x;
  const int p0 = blockIdx.x % chunks * IRF_CH, np = min(IRF_CH, npair - p0);
  if (i >= ntime) return;
  const double t = i * dt;
  double acc[IRF_CH];
#pragma unroll
  for (int q = 0; q < IRF_CH; ++q) acc[q] = 0.;
  double c0 = cos(w[0] * t);
  for (int l = 0; l < nw - 1; ++l) {
    const double c1 = cos(w[l + 1] * t), dw = w[l + 1] - w[l];
#pragma unroll
    for (int q = 0; q < IRF_CH; ++q) {
      if (q >= np) break;
      const double* B = damping + (size_t)nw * (p0 + q);
      acc[q] = acc[q] + 0.5 * (B[l] * c0 + B[l + 1] * c1) * dw;
    }
    c0 = c1;
  }
  const double PI = 4. * atan(1.0);
#pragma unroll
  for (int q = 0; q < IRF_CH; ++q) {
    if (q >= np) break;
    K[i + (size_t)ntime * (p0 + q)] = acc[q] * 2. / PI;
  }
}

// CM(l, pair) = A_l + (trapezoid of K sin(w_l t)) / w_l: a CTA per frequency and pair chunk
__global__ void __launch_bounds__(IRF_THREADS)
    irf_added_mass_kernel(int nw, const double* __restrict__ w, int npair, const double* __restrict__ added_mass,
                          int ntime, double dt, const double* __restrict__ K, double* __restrict__ cm) {
  __shared__ double red[IRF_THREADS / 32][IRF_CH];
  const int chunks = (npair + IRF_CH - 1) / IRF_CH, tid = threadIdx.x;
  const int l = blockIdx.x / chunks, p0 = blockIdx.x % chunks * IRF_CH, np = min(IRF_CH, npair - p0);
  const double wl = w[l];
  double acc[IRF_CH];
#pragma unroll
  for (int q = 0; q < IRF_CH; ++q) acc[q] = 0.;
  for (int i = tid; i < ntime - 1; i += IRF_THREADS) {
    const double t0 = i * dt, t1 = (i + 1) * dt;
    const double s0 = sin(wl * t0), s1 = sin(wl * t1);
#pragma unroll
    for (int q = 0; q < IRF_CH; ++q) {
      if (q >= np) break;
      const double* Kp = K + (size_t)ntime * (p0 + q);
      acc[q] = acc[q] + 0.5 * (Kp[i] * s0 + Kp[i + 1] * s1) * (t1 - t0);
    }
  }
#pragma unroll
  for (int q = 0; q < IRF_CH; ++q) {
    for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    if (!(tid & 31)) red[tid >> 5][q] = acc[q];
  }
  __syncthreads();
  if (tid >= np) return;
  double s = 0.;
#pragma unroll
  for (int g = 0; g < IRF_THREADS / 32; ++g) s += red[g][tid];
  const size_t e = l + (size_t)nw * (p0 + tid);
  cm[e] = added_mass[e] + s / wl;
}

// A_inf(pair) = sum_l CM(l, pair) / nw, summed in frequency order
__global__ void irf_average_kernel(int nw, int npair, const double* __restrict__ cm, double* __restrict__ ainf) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npair) return;
  double am = 0.;
  for (int l = 0; l < nw; ++l) am = am + cm[l + (size_t)nw * p];
  ainf[p] = am / nw;
}

}  // namespace nb200
