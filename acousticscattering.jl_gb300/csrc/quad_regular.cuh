// Regular 7-point rule of the collocation BEM (device): the FP64 / FP32 precision traits
// and the four Helmholtz kernels of one source panel at one collocation point.  Shared by
// the dense assembly and the hierarchical-matrix kernels so that both evaluate the same
// entries.
#pragma once

#include "bemgpu_internal.h"
#include "quad_math.cuh"

namespace bemgpu {

constexpr int kAsmCols64 = 64;     // FP64 source records per chunk (64 x 256 B = 16 KB)
constexpr int kAsmCols32 = 128;    // FP32 source records per chunk (128 x 128 B = 16 KB)

template <typename R>
struct Prec;
template <>
struct Prec<double> {
  static constexpr int kCols = kAsmCols64;
  static constexpr int kRec = kPanelDoubles;
  __device__ static __forceinline__ void sc(double z, double* s, double* c) { sincos(z, s, c); }
  __device__ static __forceinline__ double rs(double x) { return rsqrt(x); }
  __device__ static __forceinline__ const double* recs(const AsmInst& I) { return I.panels; }
};
template <>
struct Prec<float> {
  static constexpr int kCols = kAsmCols32;
  static constexpr int kRec = kPanelFloats;
  // sin/cos of pi * t with exact argument reduction
  __device__ static __forceinline__ void sc(float z, float* s, float* c) {
    sincospif(z * 0.31830988618379067154f, s, c);
  }
  __device__ static __forceinline__ float rs(float x) { return rsqrtf(x); }
  __device__ static __forceinline__ const float* recs(const AsmInst& I) { return I.panelsf; }
};

template <typename R>
struct Acc {
  cx<R> S, D, K, H;
};

// FP64 phases of a panel's seven points.  FP64 issue (two FMAs per clock and SM) bounds every
// FP64 rule, and a library sine / cosine is about half of a point's work, so it is evaluated
// at the panel's first point (the centroid) only: the others follow by the angle sum with the
// Taylor polynomials of delta = k (r_q - r_0), which the triangle inequality bounds by
// k |y_q - y_0| <= 0.465 k (longest edge).  Terms up to delta^12 (edge k <= 0.53, remainder
// below 3e-17) or delta^18 (edge k <= 1.6); longer panels take the
// library functions.  The Mueller assembly of 2880 panels: 13.0 -> 11.6 ms with both
// wavenumbers sharing the geometry.
constexpr double kPhaseShort = 0.53, kPhaseMid = 1.6;
template <int N>
__device__ __forceinline__ void phase_step(double s0, double c0, double d, double* s, double* c) {
  const double d2 = d * d;
  double ps, pc;
  if (N == 12) {
    ps = -1.0 / 39916800.0;
    pc = 1.0 / 479001600.0;
  } else {
    ps = fma(1.0 / 355687428096000.0, d2, -1.0 / 1307674368000.0);
    ps = fma(ps, d2, 1.0 / 6227020800.0);
    ps = fma(ps, d2, -1.0 / 39916800.0);
    pc = fma(-1.0 / 6402373705728000.0, d2, 1.0 / 20922789888000.0);
    pc = fma(pc, d2, -1.0 / 87178291200.0);
    pc = fma(pc, d2, 1.0 / 479001600.0);
  }
  ps = fma(ps, d2, 1.0 / 362880.0);
  ps = fma(ps, d2, -1.0 / 5040.0);
  ps = fma(ps, d2, 1.0 / 120.0);
  ps = fma(ps, d2, -1.0 / 6.0);
  ps = fma(ps * d2, d, d);
  pc = fma(pc, d2, -1.0 / 3628800.0);
  pc = fma(pc, d2, 1.0 / 40320.0);
  pc = fma(pc, d2, -1.0 / 720.0);
  pc = fma(pc, d2, 1.0 / 24.0);
  pc = fma(pc, d2, -0.5);
  pc = fma(pc, d2, 1.0);
  *c = c0 * pc - s0 * ps;
  *s = s0 * pc + c0 * ps;
}

// The four FP64 kernels of one source panel at NK wavenumbers; the geometry is shared.  N: last
// term of the phase polynomials, 0: library functions.
template <int NK, bool NEED_KH, int N>
__device__ __forceinline__ void panel64(const double* rec, const double x[3], const double nx[3],
                                        const double* k, Acc<double>* a) {
  const double ny0 = rec[3], ny1 = rec[4], ny2 = rec[5];
  const double area = rec[6];
  const double nn = nx[0] * ny0 + nx[1] * ny1 + nx[2] * ny2;
  double r0 = 0.0, s0[NK], c0[NK];
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    const double u0 = rec[8 + 3 * q] - x[0];
    const double u1 = rec[9 + 3 * q] - x[1];
    const double u2 = rec[10 + 3 * q] - x[2];
    const double r2 = u0 * u0 + u1 * u1 + u2 * u2;
    const double ir = rsqrt(r2);
    const double r = r2 * ir;
    const double wir = dRuleW[q] * area * kInv4Pi * ir;
    const double ir2 = ir * ir;
    const double w3 = wir * ir2;
    const double uny = u0 * ny0 + u1 * ny1 + u2 * ny2;
    const double wd = w3 * uny;
    double unx = 0.0, c = 0.0, c3 = 0.0, wk = 0.0;
    if (NEED_KH) {
      unx = u0 * nx[0] + u1 * nx[1] + u2 * nx[2];
      wk = w3 * unx;
      c = unx * uny * ir2;
      c3 = 3.0 * c - nn;
    }
    if (q == 0) r0 = r;
#pragma unroll
    for (int i = 0; i < NK; ++i) {
      const double z = k[i] * r;
      double sn, cs;
      if (N == 0 || q == 0)
        sincos(z, &sn, &cs);
      else
        phase_step<N>(s0[i], c0[i], k[i] * (r - r0), &sn, &cs);
      if (q == 0) {
        s0[i] = sn;
        c0[i] = cs;
      }
      a[i].S.x += wir * cs;
      a[i].S.y += wir * sn;
      // e^{iz} (iz - 1) w / (4 pi r^3)
      const double gx = -cs - z * sn, gy = z * cs - sn;
      a[i].D.x += wd * gx;
      a[i].D.y += wd * gy;
      if (NEED_KH) {
        a[i].K.x -= wk * gx;
        a[i].K.y -= wk * gy;
        // e^{iz} [(nn - c (3 - z^2)) + i z (3c - nn)] w / (4 pi r^3)
        const double br = c * (z * z) - c3, bi = z * c3;
        a[i].H.x += w3 * (cs * br - sn * bi);
        a[i].H.y += w3 * (cs * bi + sn * br);
      }
    }
  }
}
template <int NK, bool NEED_KH>
__device__ __forceinline__ void regular_panel64(const double* rec, const double x[3],
                                                const double nx[3], const double* k,
                                                Acc<double>* a) {
  double kd = k[0] * rec[7];
#pragma unroll
  for (int i = 1; i < NK; ++i) kd = fmax(kd, k[i] * rec[7]);
  if (kd <= kPhaseShort)
    panel64<NK, NEED_KH, 12>(rec, x, nx, k, a);
  else if (kd <= kPhaseMid)
    panel64<NK, NEED_KH, 18>(rec, x, nx, k, a);
  else
    panel64<NK, NEED_KH, 0>(rec, x, nx, k, a);
}

// Full Helmholtz kernels of one source panel (7 points) at one wavenumber.
// (FP64: panel64, whose sums are the same to rounding.)
template <typename R, bool NEED_KH>
__device__ __forceinline__ void regular_panel(const R* rec, const R x[3], const R nx[3], R k,
                                              Acc<R>& a) {
  if constexpr (sizeof(R) == 8) {
    regular_panel64<1, NEED_KH>(rec, x, nx, &k, &a);
    return;
  }
  const R ny0 = rec[3], ny1 = rec[4], ny2 = rec[5];
  const R area = rec[6];
  const R nn = nx[0] * ny0 + nx[1] * ny1 + nx[2] * ny2;
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    const R u0 = rec[8 + 3 * q] - x[0];
    const R u1 = rec[9 + 3 * q] - x[1];
    const R u2 = rec[10 + 3 * q] - x[2];
    const R r2 = u0 * u0 + u1 * u1 + u2 * u2;
    const R ir = Prec<R>::rs(r2);
    const R r = r2 * ir;
    const R z = k * r;
    R sn, cs;
    Prec<R>::sc(z, &sn, &cs);
    const R w = (R)dRuleW[q] * area * (R)kInv4Pi;
    const R wir = w * ir;
    const R ir2 = ir * ir;
    a.S += wir * cx<R>{cs, sn};
    const R uny = u0 * ny0 + u1 * ny1 + u2 * ny2;
    // e^{iz} (iz - 1) w / (4 pi r^3)
    const cx<R> gp = (wir * ir2) * cx<R>{-cs - z * sn, -sn + z * cs};
    a.D += uny * gp;
    if (NEED_KH) {
      const R unx = u0 * nx[0] + u1 * nx[1] + u2 * nx[2];
      a.K -= unx * gp;
      const R c = unx * uny * ir2;
      // e^{iz} [(nn - c (3 - z^2)) + i z (3c - nn)] w / (4 pi r^3)
      const cx<R> br = {nn - c * ((R)3 - z * z), z * ((R)3 * c - nn)};
      a.H += (wir * ir2) * (cx<R>{cs, sn} * br);
    }
  }
}

// The same at two wavenumbers.
template <typename R, bool NEED_KH>
__device__ __forceinline__ void regular_panel2(const R* rec, const R x[3], const R nx[3], R k0,
                                               R k1, Acc<R>& a0, Acc<R>& a1) {
  if constexpr (sizeof(R) == 8) {
    const double k[2] = {k0, k1};
    Acc<double> a[2] = {a0, a1};
    regular_panel64<2, NEED_KH>(rec, x, nx, k, a);
    a0 = a[0];
    a1 = a[1];
  } else {
    regular_panel<R, NEED_KH>(rec, x, nx, k0, a0);
    regular_panel<R, NEED_KH>(rec, x, nx, k1, a1);
  }
}

}  // namespace bemgpu
