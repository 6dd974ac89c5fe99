// Field evaluation at points: the pressure query of the full-3D BEM solution
// (fields/pressure.jl:404-471 of the reference).
//
//   exterior:  u_s(x) = sum_j [ D_j(x) p_j - S_j(x) q_j ]           (scattered traces, k)
//   interior:  u_i(x) = sum_j [ S_j(x) g (q_j + q_inc,j) - D_j(x) (p_j + p_inc,j) ]  (k / h)
//   incident:  e^{ik d.x}
//
// S_j, D_j are the single- and double-layer potentials of the flat panel j with unit
// density: 7-point rule away from the panel, closed-form Laplace parts plus the
// Helmholtz remainders (quad_math.cuh) when x is within eta panel diameters.  The
// region of each point (inside / outside the closed surface) comes from the sum of the
// panels' solid angles (4 pi inside, 0 outside, 2 pi on the surface).  One CTA per
// point, fixed-order reductions, FP64 fields.
//
// Bound by FP64 issue.  The far panels take the shared-phase rule of quad_regular.cuh, the
// interior traces are formed once per call (from kTracesPoints points on), and the region test
// sums FP32 angles (panels within two diameters, or at distances whose cubes FP32 does not
// hold, in FP64), repeated in FP64 when the sum is not clearly 0 or 4 pi:
// 2001 points of a 2880-panel fluid body 6.30 -> 4.5 ms.
#include "bemgpu_internal.h"
#include "pressure.cuh"
#include "quad_math.cuh"
#include "quad_regular.cuh"

namespace bemgpu {

constexpr int kPrThreads = 256;

__device__ __forceinline__ double solid_angle(const double* v, const double* x) {
  double R0[3], R1[3], R2[3], t[3];
  sub3(v, x, R0);
  sub3(v + 3, x, R1);
  sub3(v + 6, x, R2);
  const double r0 = sqrt(dot3(R0, R0)), r1 = sqrt(dot3(R1, R1)), r2 = sqrt(dot3(R2, R2));
  cross3(R1, R2, t);
  const double num = dot3(R0, t);
  const double den = r0 * r1 * r2 + dot3(R0, R1) * r2 + dot3(R0, R2) * r1 + dot3(R1, R2) * r0;
  return 2.0 * atan2(num, den);
}

// Solid angle of a panel in FP32, for the region test: records relative to the point lose nothing
// that matters at a distance of a few panels.  Its products are of the third degree in the
// distances, so it is for panels whose squared distance is within kAngleMin2 and kAngleMax2.
constexpr float kAngleMin2 = 1e-20f, kAngleMax2 = 1e20f;
__device__ __forceinline__ float solid_angle_f(const double* v, const double* x) {
  float R[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int t = 0; t < 3; ++t) R[a][t] = (float)(v[3 * a + t] - x[t]);
  auto dot = [](const float* a, const float* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; };
  const float r0 = sqrtf(dot(R[0], R[0])), r1 = sqrtf(dot(R[1], R[1])), r2 = sqrtf(dot(R[2], R[2]));
  const float t[3] = {R[1][1] * R[2][2] - R[1][2] * R[2][1], R[1][2] * R[2][0] - R[1][0] * R[2][2],
                      R[1][0] * R[2][1] - R[1][1] * R[2][0]};
  const float num = dot(R[0], t);
  const float den =
      r0 * r1 * r2 + dot(R[0], R[1]) * r2 + dot(R[0], R[2]) * r1 + dot(R[1], R[2]) * r0;
  return 2.0f * atan2f(num, den);
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < NT / 32; ++w) t += sh[w];
  __syncthreads();
  if (threadIdx.x == 0) sh[0] = t;
  __syncthreads();
  return sh[0];
}

// Single and double layer of a far panel.
__device__ __forceinline__ void far_layers(const double* rj, const double* x, double k, cd& S,
                                           cd& D) {
  const double none[3] = {0.0, 0.0, 0.0};
  Acc<double> a;
  a.S = a.D = a.K = a.H = cd{0.0, 0.0};
  regular_panel64<1, false>(rj, x, none, &k, &a);
  S = a.S;
  D = a.D;
}

// Interior traces p = p_s + p_inc, q = g (q_s + q_inc).
__device__ __forceinline__ void interior_traces(const PressureInst& P, const double* rj, cd& p,
                                                cd& q) {
  const double* d = P.dir;
  const double ph = P.k * (d[0] * rj[0] + d[1] * rj[1] + d[2] * rj[2]);
  double sn, cs;
  sincos(ph, &sn, &cs);
  const double dn = P.k * (d[0] * rj[3] + d[1] * rj[4] + d[2] * rj[5]);
  p = cd{p.x + cs, p.y + sn};
  q = cd{P.g * (q.x - dn * sn), P.g * (q.y + dn * cs)};
}
__global__ void k_interior_traces(const PressureInst P) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= P.n) return;
  cd p = {P.p[2 * j], P.p[2 * j + 1]}, q = {P.q[2 * j], P.q[2 * j + 1]};
  interior_traces(P, P.panels + j * kPanelDoubles, p, q);
  P.pi[2 * j] = p.x;
  P.pi[2 * j + 1] = p.y;
  P.qi[2 * j] = q.x;
  P.qi[2 * j + 1] = q.y;
}

__global__ void __launch_bounds__(kPrThreads) k_pressure(const PressureInst P) {
  const int64_t ip = blockIdx.x;
  if (ip >= P.npts) return;
  __shared__ double sh[kPrThreads / 32];
  const double x[3] = {P.points[3 * ip], P.points[3 * ip + 1], P.points[3 * ip + 2]};
  const double zero3[3] = {0.0, 0.0, 0.0};
  // region by total solid angle
  const double four_pi = 12.566370614359172954;
  double om = 0.0;
  float omf = 0.f;
  for (int64_t j = threadIdx.x; j < P.n; j += kPrThreads) {
    const double* rj = P.panels + j * kPanelDoubles;
    const float dx = (float)(x[0] - rj[0]), dy = (float)(x[1] - rj[1]), dz = (float)(x[2] - rj[2]);
    const float lim = 2.0f * (float)rj[7], d2 = dx * dx + dy * dy + dz * dz;
    if (!(d2 >= lim * lim && d2 > kAngleMin2 && d2 < kAngleMax2))
      om += solid_angle(P.verts + j * kVertDoubles, x);
    else
      omf += solid_angle_f(P.verts + j * kVertDoubles, x);
  }
  om = block_sum<kPrThreads>(om + (double)omf, sh);
  if (!(fabs(om) < 0.01 * four_pi || fabs(om - four_pi) < 0.01 * four_pi)) {
    om = 0.0;
    for (int64_t j = threadIdx.x; j < P.n; j += kPrThreads)
      om += solid_angle(P.verts + j * kVertDoubles, x);
    om = block_sum<kPrThreads>(om, sh);
  }
  const bool inside = om > 0.5 * four_pi;
  const bool on_surface = fabs(om - 0.5 * four_pi) < 1e-6 * four_pi;
  int region = inside ? 1 : 0;  // 0 exterior, 1 interior
  if (on_surface) region = P.fluid ? 1 : 0;
  if (threadIdx.x == 0) P.region[ip] = on_surface ? 2 : region;
  const double* d = P.dir;
  const double ph_x = P.k * (d[0] * x[0] + d[1] * x[1] + d[2] * x[2]);
  double psn, pcs;
  sincos(ph_x, &psn, &pcs);
  if (P.field == 2) {  // incident only
    if (threadIdx.x == 0) {
      P.out[2 * ip] = pcs;
      P.out[2 * ip + 1] = psn;
    }
    return;
  }
  const bool interior = region == 1;
  if ((interior && !P.fluid) || (P.field == 3 && !interior) ||
      (P.field == 1 && interior)) {
    // the field does not exist at this point: NaN marks it for the host
    if (threadIdx.x == 0) {
      P.out[2 * ip] = NAN;
      P.out[2 * ip + 1] = NAN;
    }
    return;
  }
  const double k = interior ? P.k_int : P.k;
  double acc_r = 0.0, acc_i = 0.0;
  for (int64_t j = threadIdx.x; j < P.n; j += kPrThreads) {
    const double* rj = P.panels + j * kPanelDoubles;
    const double* nT = rj + 3;
    const bool formed = interior && P.pi;
    const double* tp = formed ? P.pi : P.p;
    const double* tq = formed ? P.qi : P.q;
    cd pj = {tp[2 * j], tp[2 * j + 1]}, qj = {tq[2 * j], tq[2 * j + 1]};
    if (interior && !formed) interior_traces(P, rj, pj, qj);
    const double dx = x[0] - rj[0], dy = x[1] - rj[1], dz = x[2] - rj[2];
    const double d2 = dx * dx + dy * dy + dz * dz;
    const double lim = P.eta * rj[7];
    cd S = {0.0, 0.0}, D = {0.0, 0.0};
    if (d2 < lim * lim) {
      double v[9];
#pragma unroll
      for (int t = 0; t < 9; ++t) v[t] = P.verts[j * kVertDoubles + t];
      double S0, D0, K0, H0;
      laplace_parts(v, nT, x, zero3, false, S0, D0, K0, H0);
      Ops o;
      o.S = o.D = o.K = o.H = cd{0.0, 0.0};
#pragma unroll 1
      for (int q = 0; q < 7; ++q) {
        double u[3];
        sub3(rj + 8 + 3 * q, x, u);
        rem_point(k, u, zero3, nT, dRuleW[q] * rj[6], o);
      }
      S = o.S + cd{S0, 0.0};
      D = o.D + cd{D0, 0.0};
    } else {
      far_layers(rj, x, k, S, D);
    }
    cd c = interior ? (S * qj - D * pj) : (D * pj - S * qj);
    acc_r += c.x;
    acc_i += c.y;
  }
  acc_r = block_sum<kPrThreads>(acc_r, sh);
  acc_i = block_sum<kPrThreads>(acc_i, sh);
  if (threadIdx.x == 0) {
    double re = acc_r, im = acc_i;
    if (P.field == 0 && !interior) {  // total exterior = incident + scattered
      re += pcs;
      im += psn;
    }
    P.out[2 * ip] = re;
    P.out[2 * ip + 1] = im;
  }
}

// Single and double layer of panel j (unit density) at x with wavenumber k: closed-form
// Laplace parts plus remainders when x is within eta panel diameters, else the 7-point rule.
__device__ __forceinline__ void panel_layers(const PressureInst& P, int64_t j, const double* x,
                                             double k, cd& S, cd& D) {
  const double zero3[3] = {0.0, 0.0, 0.0};
  const double* rj = P.panels + j * kPanelDoubles;
  const double* nT = rj + 3;
  const double dx = x[0] - rj[0], dy = x[1] - rj[1], dz = x[2] - rj[2];
  const double d2 = dx * dx + dy * dy + dz * dz;
  const double lim = P.eta * rj[7];
  S = D = cd{0.0, 0.0};
  if (d2 < lim * lim) {
    double v[9];
#pragma unroll
    for (int t = 0; t < 9; ++t) v[t] = P.verts[j * kVertDoubles + t];
    double S0, D0, K0, H0;
    laplace_parts(v, nT, x, zero3, false, S0, D0, K0, H0);
    Ops o;
    o.S = o.D = o.K = o.H = cd{0.0, 0.0};
#pragma unroll 1
    for (int q = 0; q < 7; ++q) {
      double u[3];
      sub3(rj + 8 + 3 * q, x, u);
      rem_point(k, u, zero3, nT, dRuleW[q] * rj[6], o);
    }
    S = o.S + cd{S0, 0.0};
    D = o.D + cd{D0, 0.0};
  } else {
    far_layers(rj, x, k, S, D);
  }
}

// Coupled regions (fields/regions.jl:1-65 of the reference): the region of the point by
// the reference's walk over the interfaces (an interface is tested only when its parent
// is the region found so far; the solid angle of its panels tells inside / on / outside),
// then the sum over the interfaces that border the region of S dp - D p (the region
// inside them) or D p - S dp (outside), with the region's wavenumber; in the unbounded
// region the traces are the scattered ones and the total field adds the incident wave.
__global__ void __launch_bounds__(kPrThreads) k_pressure_regions(const PressureInst P) {
  const int64_t ip = blockIdx.x;
  if (ip >= P.npts) return;
  __shared__ double sh[kPrThreads / 32];
  const double x[3] = {P.points[3 * ip], P.points[3 * ip + 1], P.points[3 * ip + 2]};
  const double four_pi = 12.566370614359172954;
  int containing = 0, adj_out = -1, adj_in = -1;
  for (int s = 0; s < P.nsurf; ++s) {
    if (P.parents[s] != containing) continue;  // uniform over the CTA
    double om = 0.0;
    for (int64_t j = P.offsets[s] + threadIdx.x; j < P.offsets[s + 1]; j += kPrThreads)
      om += solid_angle(P.verts + j * kVertDoubles, x);
    om = block_sum<kPrThreads>(om, sh);
    if (fabs(om - 0.5 * four_pi) < 1e-6 * four_pi) {
      adj_out = P.parents[s];
      adj_in = s + 1;
      break;
    }
    if (om > 0.5 * four_pi) containing = s + 1;
  }
  int region, status = 0;
  if (P.requested >= 0) {
    const bool valid = adj_in < 0 ? P.requested == containing
                                  : (P.requested == adj_out || P.requested == adj_in);
    if (!valid) status = kPrBadRegion;
    region = P.requested;
  } else if (adj_in >= 0) {
    region = P.field == 3 ? adj_in : adj_out;
  } else {
    region = containing;
  }
  if (!status && P.field == 1 && region != 0) status = kPrNeedExterior;
  if (!status && P.field == 3 && region == 0) status = kPrNeedFluid;
  const double* d = P.dir;
  double psn, pcs;
  sincos(P.k * (d[0] * x[0] + d[1] * x[1] + d[2] * x[2]), &psn, &pcs);
  if (threadIdx.x == 0) P.region[ip] = status ? -status : region;
  if (status || P.field == 2) {
    if (threadIdx.x == 0) {
      P.out[2 * ip] = status ? NAN : pcs;
      P.out[2 * ip + 1] = status ? NAN : psn;
    }
    return;
  }
  const double k = region == 0 ? P.k : P.kr[region];
  const int64_t n = P.offsets[P.nsurf];
  double acc_r = 0.0, acc_i = 0.0;
  for (int s = 0; s < P.nsurf; ++s) {
    const bool inside = s + 1 == region;
    if (!inside && P.parents[s] != region) continue;
    const double rho = inside ? P.rho[s + 1] : P.rho[P.parents[s]];
    for (int64_t j = P.offsets[s] + threadIdx.x; j < P.offsets[s + 1]; j += kPrThreads) {
      cd pj = {P.xr[2 * j], P.xr[2 * j + 1]};
      cd dp = rho * cd{P.xr[2 * (n + j)], P.xr[2 * (n + j) + 1]};
      if (region == 0) {  // scattered traces
        const double* rj = P.panels + j * kPanelDoubles;
        const double ph = P.k * (d[0] * rj[0] + d[1] * rj[1] + d[2] * rj[2]);
        double sn, cs;
        sincos(ph, &sn, &cs);
        const double dn = P.k * (d[0] * rj[3] + d[1] * rj[4] + d[2] * rj[5]);
        pj = pj - cd{cs, sn};
        dp = dp - cd{-dn * sn, dn * cs};
      }
      cd S, D;
      panel_layers(P, j, x, k, S, D);
      const cd c = inside ? (S * dp - D * pj) : (D * pj - S * dp);
      acc_r += c.x;
      acc_i += c.y;
    }
  }
  acc_r = block_sum<kPrThreads>(acc_r, sh);
  acc_i = block_sum<kPrThreads>(acc_i, sh);
  if (threadIdx.x == 0) {
    double re = acc_r, im = acc_i;
    if (P.field == 0 && region == 0) {
      re += pcs;
      im += psn;
    }
    P.out[2 * ip] = re;
    P.out[2 * ip + 1] = im;
  }
}

void launch_pressure(const Launch& L, const PressureInst& P) {
  if (P.npts <= 0) return;
  if (P.nsurf > 0)
    k_pressure_regions<<<(unsigned)P.npts, kPrThreads, 0, L.stream>>>(P);
  else {
    // the incident field has no traces (a Nystroem solution asks for it and the regions alone)
    if (P.pi && P.field != BEMGPU_FIELD_INCIDENT) {
      k_interior_traces<<<(unsigned)((P.n + 127) / 128), 128, 0, L.stream>>>(P);
      count_launch(1);
    }
    k_pressure<<<(unsigned)P.npts, kPrThreads, 0, L.stream>>>(P);
  }
  count_launch(1);
}

}  // namespace bemgpu
