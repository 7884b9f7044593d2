// Kochin function of the solved problems (COMPUTE_KOCHIN.f90:25-152).
//
// H(theta) = 1/(4 pi) sum_J [ ZIGB(J) ZS_J(theta) + ZIGS(J) ZS'_J(theta) ], where
// ZS_J is the analytical integral over panel J of the far-field wave factor,
// an edge sum of (CEP(l+1) - CEP(l)) / (ZJ(l+1) - ZJ(l)) terms with
// ZJ(k) = k0 (z_k - i wbar_k), wbar = (x - XEFF) cos(theta) + (y - YEFF) sin(theta),
// CEP = exp(ZJ) and, in finite depth, CEM = exp(-ZJ - 2 k0 h); ZS' is the same
// for the mirror image of the half mesh (y -> -y). One CTA = 128 panels x one
// direction; each thread builds its panel's ZS (and ZS'), multiplies by the
// source strengths of every problem and the CTA reduces them into H.
// The quantities that decide a branch (wbar, ZJ, ZC = ZJ(l+1) - ZJ(l) and the
// depth switches) are rounded exactly in the reference's order.
#pragma once
#include "common.cuh"

namespace nb200 {

constexpr int KOCHIN_THREADS = 128;
constexpr int KOCHIN_GROUP = 8;   // problems summed between two barriers

// what a panel's direction-independent factors are: node coordinates, k0 z and
// the moduli of CEP and CEM (zero where COMPUTE_KOCHIN.f90 drops them)
struct KochinPanel {
  double x[4], y[4], zre[4], ep[4], em[4];
  double xn, yn, zn, f;   // f: the depth factor over k0
};

NB_HD __forceinline__ void kochin_setup(const double* __restrict__ xyz, const int* __restrict__ m1234,
                                        const double* __restrict__ rows, int nfa, double kwave, double depth, int i,
                                        KochinPanel& P) {
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int k = m1234[4 * i + l] - 1;
    P.x[l] = xyz[3 * k];
    P.y[l] = xyz[3 * k + 1];
    P.zre[l] = XMUL(kwave, xyz[3 * k + 2]);
    P.ep[l] = P.zre[l] < -18. ? 0. : exp(P.zre[l]);
    const double tre = XSUB(-P.zre[l], XMUL(XMUL(2., kwave), depth));
    P.em[l] = (tre < -18.) || (-XMUL(kwave, depth) >= 0.) ? 0. : exp(tre);
  }
  P.xn = rows[3 * nfa + i];
  P.yn = rows[4 * nfa + i];
  P.zn = rows[5 * nfa + i];
  const double kh = XMUL(kwave, depth);
  P.f = (kh > 18.) || (kh <= 0.) ? 1. / kwave : 0.5 * exp(kh) / sinh(kh) / kwave;
}

// ZS of a panel (and ZS' of its mirror half) for the direction (ct, st). CEM's
// phase is CEP's conjugate, so a node takes one sincos; both edge quotients have
// the divisor ZC, so an edge takes one complex division.
NB_HD __forceinline__ void kochin_direction(const KochinPanel& P, int nsymy, double xeff, double yeff, double ct,
                                            double st, double kwave, cplx* zs) {
  for (int half = 0; half <= nsymy; ++half) {
    const double ys = half ? -1. : 1.;
    const cplx ZMS = mk(half ? -P.yn : P.yn, -(P.zn * st));
    const cplx ZNS = mk(P.xn, -(P.zn * ct));
    cplx u[4];
    double zim[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const double wbar = XADD(XMUL(XSUB(P.x[l], xeff), ct), XMUL(XSUB(ys * P.y[l], yeff), st));
      zim[l] = XMUL(kwave, -wbar);
      sincos(zim[l], &u[l].im, &u[l].re);
    }
    cplx acc = mk(0., 0.);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int n = (l + 1) & 3;
      const double dx = P.x[n] - P.x[l], dy = P.y[n] - P.y[l];
      cplx ZCS = half ? ZMS * dx + ZNS * dy : ZMS * dx - ZNS * dy;
      const cplx ZC = mk(XSUB(P.zre[n], P.zre[l]), XSUB(zim[n], zim[l]));
      cplx hs = mk(P.ep[n] * u[n].re, P.ep[n] * u[n].im), hd = mk(P.em[n] * u[n].re, -(P.em[n] * u[n].im));
      const cplx ls = mk(P.ep[l] * u[l].re, P.ep[l] * u[l].im), ld = mk(P.em[l] * u[l].re, -(P.em[l] * u[l].im));
      if (fabs(ZC.im) < 1.E-04 && fabs(ZC.re) < 1.E-04) {
        hs = 0.5 * (hs + ls);
        hd = -0.5 * (hd + ld);
      } else {
        hs = hs - ls;
        hd = hd - ld;
        ZCS = ZCS / ZC;
      }
      const cplx a = ZCS * hs, b = ZCS * hd;
      acc = acc + a + mk(b.re, -b.im);
    }
    zs[half] = (half ? -P.f : P.f) * acc;
  }
}

// both for one panel and one direction
NB_HD __forceinline__ void kochin_panel(const double* __restrict__ xyz, const int* __restrict__ m1234,
                                        const double* __restrict__ rows, int nfa, int nsymy, double kwave,
                                        double depth, double xeff, double yeff, double ct, double st, int i,
                                        cplx* zs) {
  KochinPanel P;
  kochin_setup(xyz, m1234, rows, nfa, kwave, depth, i, P);
  kochin_direction(P, nsymy, xeff, yeff, ct, st, kwave, zs);
}

// Sums of four values over a warp in six shuffles: each step folds pairs of
// values onto half the lanes. Lane 8 k holds the sum of v[k].
__device__ __forceinline__ double warp_sum4(const double* v, int lane) {
  const unsigned all = 0xffffffffu;
  const bool hi = lane & 16, lo = lane & 8;
  const double a = (hi ? v[2] : v[0]) + __shfl_xor_sync(all, hi ? v[0] : v[2], 16);
  const double b = (hi ? v[3] : v[1]) + __shfl_xor_sync(all, hi ? v[1] : v[3], 16);
  double s = (lo ? b : a) + __shfl_xor_sync(all, lo ? a : b, 8);
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(all, s, o);
  return s;
}

// out (ntheta x nprob complex) must be zero; zigb/zigs: nprob x nfa complex.
// The latency of the node and strength loads and of the FP64 chains bounds it (a
// tenth of DRAM, a third of the issue slots), hence the registers for five CTAs
// an SM; the problems are summed in groups, one pair of barriers each. 2,400
// panels x 361 directions x 9 problems: 296 to 182 us (2 CTAs of 168 registers
// 260, 8 CTAs 195; 2 or 4 directions a CTA, their exponentials kept, 190 and 195).
__global__ void __launch_bounds__(KOCHIN_THREADS, 5)
    kochin_kernel(const double* __restrict__ xyz, const int* __restrict__ m1234, const double* __restrict__ rows,
                  int nfa, int nsymy, double kwave, double depth, double xeff, double yeff,
                  const double2* __restrict__ cs, int nprob, const double2* __restrict__ zigb,
                  const double2* __restrict__ zigs, int ntheta, double2* out) {
  constexpr int W = KOCHIN_THREADS / 32;
  __shared__ double red[W][2 * KOCHIN_GROUP];
  const int i = blockIdx.x * KOCHIN_THREADS + threadIdx.x;
  const int t = blockIdx.y;
  cplx zs[2] = {mk(0., 0.), mk(0., 0.)};
  if (i < nfa) kochin_panel(xyz, m1234, rows, nfa, nsymy, kwave, depth, xeff, yeff, cs[t].x, cs[t].y, i, zs);
  const double q = 0.25 / 3.141592653589793;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int p0 = 0; p0 < nprob; p0 += KOCHIN_GROUP) {
    const int np = min(KOCHIN_GROUP, nprob - p0);
#pragma unroll
    for (int pp = 0; pp < KOCHIN_GROUP; pp += 2) {
      if (pp >= np) break;
      double v[4] = {0., 0., 0., 0.};
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (i < nfa && pp + h < np) {
          const double2 b = zigb[(long long)(p0 + pp + h) * nfa + i];
          cplx c = mk(b.x, b.y) * zs[0];
          if (nsymy) {
            const double2 s = zigs[(long long)(p0 + pp + h) * nfa + i];
            c = c + mk(s.x, s.y) * zs[1];
          }
          v[2 * h] = c.re;
          v[2 * h + 1] = c.im;
        }
      const double s = warp_sum4(v, lane);
      if (!(lane & 7)) red[warp][2 * pp + (lane >> 3)] = s;
    }
    __syncthreads();
    if (threadIdx.x < 2 * np) {
      double s = 0.;
#pragma unroll
      for (int w = 0; w < W; ++w) s += red[w][threadIdx.x];
      double2* o = &out[t + (long long)ntheta * (p0 + threadIdx.x / 2)];
      atomicAdd(threadIdx.x & 1 ? &o->y : &o->x, q * s);
    }
    __syncthreads();
  }
}

}  // namespace nb200
