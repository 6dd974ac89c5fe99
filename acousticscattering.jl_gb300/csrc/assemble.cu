// Assembly, incident-field and far-field kernels of the collocation BEM.
//
// Regular pairs: each CTA owns a tile of kAsmRows collocation points (one per thread)
// and a chunk of source panels whose records (centroid, normal, area, Gauss points)
// are staged in shared memory by one bulk asynchronous copy (TMA engine).  All threads
// of a warp read the same source record (shared-memory broadcast) and write the
// column-major matrix entry of their own row, so every warp store is 32 consecutive
// complex values (256 or 512 contiguous bytes).  The mixed-precision system is stored
// as complex64 (exact for the FP32 rule); the FP64 near values it cannot hold exactly
// keep their rounding error in a sparse correction list.
// Near pairs: one thread per listed pair evaluates the FP64 singular rules and
// overwrites the regular value (stream order guarantees the regular kernel ran first).
#include <cstdio>

#include "bemgpu_internal.h"
#include "quad_math.cuh"
#include "quad_regular.cuh"
#include "tma.cuh"

namespace bemgpu {

constexpr int kAsmRows = 128;      // threads per CTA = collocation points per tile

__device__ __forceinline__ void store_c(void* base, int64_t idx, cd v) {
  reinterpret_cast<double2*>(base)[idx] = make_double2(v.x, v.y);
}
// regular entry: complex64 outputs take the value as computed (exact for the FP32 rule)
template <typename R>
__device__ __forceinline__ void store_r(void* base, bool c64, int64_t idx, cx<R> v) {
  if (c64)
    reinterpret_cast<float2*>(base)[idx] = make_float2((float)v.x, (float)v.y);
  else
    reinterpret_cast<double2*>(base)[idx] = make_double2((double)v.x, (double)v.y);
}
// near entry: complex64 outputs keep the FP64 rounding error as a correction
__device__ __forceinline__ void store_n(void* base, bool c64, double* dnear, int64_t dpos,
                                        int64_t idx, cd v) {
  if (c64) {
    const float2 f = make_float2((float)v.x, (float)v.y);
    reinterpret_cast<float2*>(base)[idx] = f;
    reinterpret_cast<double2*>(dnear)[dpos] = make_double2(v.x - (double)f.x, v.y - (double)f.y);
  } else {
    store_c(base, idx, v);
  }
}

template <typename R, int KIND>
__global__ void __launch_bounds__(kAsmRows) k_assemble_regular(const AsmInst* __restrict__ insts,
                                                               int cols, int* err) {
  constexpr int kCols = Prec<R>::kCols;
  constexpr int kRec = Prec<R>::kRec;
  __shared__ alignas(128) R srec[kCols * kRec];
  __shared__ alignas(8) uint64_t bar;
  const AsmInst& I = insts[blockIdx.z];
  const int64_t n = I.n;
  const int64_t i0 = (int64_t)blockIdx.x * kAsmRows;
  const int64_t j0 = (int64_t)blockIdx.y * cols;
  if (i0 >= n || j0 >= n) return;  // uniform over the CTA
  const int cnt = (int)min((int64_t)cols, n - j0);
  const R* recs = Prec<R>::recs(I);
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t bytes = (uint32_t)(cnt * kRec * sizeof(R));
    mbar_arrive_expect_tx(&bar, bytes);
    bulk_g2s(srec, recs + j0 * kRec, bytes, &bar);
  }
  const int64_t i = i0 + threadIdx.x;
  const bool row_ok = i < n;
  R x[3] = {0, 0, 0}, nx[3] = {0, 0, 1};
  if (row_ok) {
    const R* ri = recs + i * kRec;
    x[0] = ri[0]; x[1] = ri[1]; x[2] = ri[2];
    nx[0] = ri[3]; nx[1] = ri[4]; nx[2] = ri[5];
  }
  const bool ok = mbar_wait(&bar, 0, err);
  if (!ok || !row_ok) return;
  const R ke = (R)I.k_e, ki = (R)I.k_i;
  const int64_t lda = I.lda;
  const int si = KIND == kAsmRegion ? I.surf[i] : 0;
  for (int jj = 0; jj < cnt; ++jj) {
    const int64_t j = j0 + jj;
    if (j == i) continue;  // self pair: near kernel
    const R* rec = srec + jj * kRec;
    if (KIND == kAsmBM || KIND == kAsmCBIE) {
      Acc<R> a;
      a.S = a.D = a.K = a.H = cx<R>{0, 0};
      regular_panel<R, KIND == kAsmBM>(rec, x, nx, ke, a);
      cx<R> m1 = cx<R>{-a.D.x, -a.D.y}, m2 = a.S;
      if (KIND == kAsmBM) {
        const cx<R> al = {(R)I.a_re, (R)I.a_im};
        m1 -= al * a.H;
        m2 += al * a.K;
      }
      store_r(I.out1, (I.c64 & 1) != 0, i + j * lda, m1);
      store_r(I.out2, (I.c64 & 2) != 0, i + j * lda, m2);
    } else if (KIND == kAsmRegion) {
      const RegionTable& RT = *I.region;
      const RegionCoef& C = RT.c[si * kMaxRegions + I.surf[j]];
      cx<R> a11 = {0, 0}, a12 = {0, 0}, a21 = {0, 0}, a22 = {0, 0};
      for (int q = 0; q < C.count; ++q) {
        Acc<R> t;
        t.S = t.D = t.K = t.H = cx<R>{0, 0};
        const R kq = (R)RT.kr[C.kidx[q]];
        if (RT.cbie)
          regular_panel<R, false>(rec, x, nx, kq, t);
        else
          regular_panel<R, true>(rec, x, nx, kq, t);
        const R sg = (R)C.sign[q], rho = (R)C.rho[q];
        if (!RT.cbie) {
          a11 += sg * t.D;
          a12 -= (sg * rho) * t.S;
          a21 += (sg / rho) * t.H;
          a22 -= sg * t.K;
        } else if (C.eq[q] == 0) {
          a11 += sg * t.D;
          a12 -= (sg * rho) * t.S;
        } else {
          a21 += sg * t.D;
          a22 -= (sg * rho) * t.S;
        }
      }
      const bool c64 = (I.c64 & 1) != 0;
      store_r(I.out1, c64, i + j * lda, a11);
      store_r(I.out1, c64, i + (n + j) * lda, a12);
      store_r(I.out1, c64, (n + i) + j * lda, a21);
      store_r(I.out1, c64, (n + i) + (n + j) * lda, a22);
    } else {
      Acc<R> e, t;
      e.S = e.D = e.K = e.H = cx<R>{0, 0};
      t = e;
      constexpr bool kh = (KIND == kAsmMuller);
      regular_panel2<R, kh>(rec, x, nx, ke, ki, e, t);
      // block combinations in the quadrature precision (no FP64 work on the FP32 path)
      const R g = (R)I.g, ginv = (R)(1.0 / I.g);
      cx<R> a11, a12, a21, a22;
      if (KIND == kAsmMuller) {
        a11 = t.D - e.D;
        a12 = e.S - g * t.S;
        a21 = ginv * t.H - e.H;
        a22 = e.K - t.K;
      } else {
        a11 = cx<R>{-e.D.x, -e.D.y};
        a12 = e.S;
        a21 = t.D;
        a22 = cx<R>{-g * t.S.x, -g * t.S.y};
      }
      const bool c64 = (I.c64 & 1) != 0;
      store_r(I.out1, c64, i + j * lda, a11);
      store_r(I.out1, c64, i + (n + j) * lda, a12);
      store_r(I.out1, c64, (n + i) + j * lda, a21);
      store_r(I.out1, c64, (n + i) + (n + j) * lda, a22);
    }
  }
}

template <int KIND, bool F32>
__device__ __forceinline__ Ops near_pair(const double* v, const double* rj, const double* x,
                                         const double* nx, bool self, double k, double S0,
                                         double D0, double K0, double H0) {
  if (F32) return near_ops_f(v, rj, x, nx, self, k, S0, D0, K0, H0);
  return near_ops(v, rj, x, nx, self, k, S0, D0, K0, H0);
}

// F32: remainders in FP32 (mixed-precision assembly); the Laplace parts and the block
// combinations stay FP64.
template <int KIND, bool F32>
__global__ void __launch_bounds__(128) k_assemble_near(const AsmInst* __restrict__ insts) {
  const AsmInst& I = insts[blockIdx.z];
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= I.n_near) return;
  const int64_t i = I.near_i[p], j = I.near_j[p];
  const double* ri = I.panels + i * kPanelDoubles;
  const double* rj = I.panels + j * kPanelDoubles;
  double v[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) v[t] = I.verts[j * kVertDoubles + t];
  double x[3] = {ri[0], ri[1], ri[2]}, nx[3] = {ri[3], ri[4], ri[5]};
  const bool self = (i == j);
  const double4 lp = reinterpret_cast<const double4*>(I.near_lap)[p];
  const double S0 = lp.x, D0 = lp.y, K0 = lp.z, H0 = lp.w;
  const int64_t n = I.n, lda = I.lda;
  const double delta = self ? 1.0 : 0.0;
  if (KIND == kAsmBM || KIND == kAsmCBIE) {
    Ops o = near_pair<KIND, F32>(v, rj, x, nx, self, I.k_e, S0, D0, K0, H0);
    cd m1 = cd{0.5 * delta - o.D.x, -o.D.y};
    cd m2 = o.S;
    if (KIND == kAsmBM) {
      cd al = {I.a_re, I.a_im};
      m1 -= al * o.H;
      m2 += al * (o.K + cd{0.5 * delta, 0.0});
    }
    const int64_t dst = I.near_dst ? I.near_dst[p] : i + j * lda;
    store_n(I.out1, (I.c64 & 1) != 0, I.dnear, p, dst, m1);
    store_n(I.out2, (I.c64 & 2) != 0, I.dnear2, p, dst, m2);
  } else if (KIND == kAsmRegion) {
    const RegionTable& RT = *I.region;
    const RegionCoef& C = RT.c[I.surf[i] * kMaxRegions + I.surf[j]];
    cd a11, a12 = {0.0, 0.0}, a21, a22 = {0.0, 0.0};
    if (RT.cbie) {  // 1/2 I in both equation rows (one per region of the interface)
      a11 = cd{0.5 * delta, 0.0};
      a21 = cd{0.5 * delta, 0.0};
    } else {
      a11 = cd{delta, 0.0};
      a22 = cd{delta, 0.0};
      a21 = cd{0.0, 0.0};
    }
    for (int q = 0; q < C.count; ++q) {
      const Ops o = near_pair<KIND, F32>(v, rj, x, nx, self, RT.kr[C.kidx[q]], S0, D0, K0, H0);
      const double sg = C.sign[q], rho = C.rho[q];
      if (!RT.cbie) {
        a11 += sg * o.D;
        a12 -= (sg * rho) * o.S;
        a21 += (sg / rho) * o.H;
        a22 -= sg * o.K;
      } else if (C.eq[q] == 0) {
        a11 += sg * o.D;
        a12 -= (sg * rho) * o.S;
      } else {
        a21 += sg * o.D;
        a22 -= (sg * rho) * o.S;
      }
    }
    const bool c64 = (I.c64 & 1) != 0;
    const int64_t nn = I.n_near;
    store_n(I.out1, c64, I.dnear, p, i + j * lda, a11);
    store_n(I.out1, c64, I.dnear, nn + p, i + (n + j) * lda, a12);
    store_n(I.out1, c64, I.dnear, 2 * nn + p, (n + i) + j * lda, a21);
    store_n(I.out1, c64, I.dnear, 3 * nn + p, (n + i) + (n + j) * lda, a22);
  } else {
    Ops e = near_pair<KIND, F32>(v, rj, x, nx, self, I.k_e, S0, D0, K0, H0);
    Ops t = near_pair<KIND, F32>(v, rj, x, nx, self, I.k_i, S0, D0, K0, H0);
    const double g = I.g;
    cd a11, a12, a21, a22;
    if (KIND == kAsmMuller) {
      a11 = cd{delta - e.D.x + t.D.x, -e.D.y + t.D.y};
      a12 = e.S - g * t.S;
      a21 = cd{t.H.x / g - e.H.x, t.H.y / g - e.H.y};
      a22 = cd{delta + e.K.x - t.K.x, e.K.y - t.K.y};
    } else {
      a11 = cd{0.5 * delta - e.D.x, -e.D.y};
      a12 = e.S;
      a21 = cd{0.5 * delta + t.D.x, t.D.y};
      a22 = cd{-g * t.S.x, -g * t.S.y};
    }
    const bool c64 = (I.c64 & 1) != 0;
    const int64_t nn = I.n_near;
    store_n(I.out1, c64, I.dnear, p, i + j * lda, a11);
    store_n(I.out1, c64, I.dnear, nn + p, i + (n + j) * lda, a12);
    store_n(I.out1, c64, I.dnear, 2 * nn + p, (n + i) + j * lda, a21);
    store_n(I.out1, c64, I.dnear, 3 * nn + p, (n + i) + (n + j) * lda, a22);
  }
}

// Laplace parts of the near pairs: computed once per mesh, reused by every wavenumber.
__global__ void k_near_laplace(const double* __restrict__ panels, const double* __restrict__ verts,
                               const int32_t* __restrict__ near_i,
                               const int32_t* __restrict__ near_j, int64_t n_near, double* out) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_near) return;
  const int64_t i = near_i[p], j = near_j[p];
  const double* ri = panels + i * kPanelDoubles;
  const double* rj = panels + j * kPanelDoubles;
  double v[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) v[t] = verts[j * kVertDoubles + t];
  double x[3] = {ri[0], ri[1], ri[2]}, nx[3] = {ri[3], ri[4], ri[5]};
  double S0, D0, K0, H0;
  laplace_parts(v, rj + 3, x, nx, i == j, S0, D0, K0, H0);
  reinterpret_cast<double4*>(out)[p] = make_double4(S0, D0, K0, H0);
}

void launch_near_laplace(const Launch& L, const double* panels, const double* verts,
                         const int32_t* near_i, const int32_t* near_j, int64_t n_near,
                         double* out) {
  if (n_near <= 0) return;
  k_near_laplace<<<(unsigned)((n_near + 127) / 128), 128, 0, L.stream>>>(panels, verts, near_i,
                                                                         near_j, n_near, out);
  count_launch(1);
}

// ------------------------------------------------------------------ launch wrappers
template <typename R>
static void launch_regular_t(const Launch& L, const AsmInst* d, int ninst, int64_t nmax,
                             int kind) {
  // source panels per CTA: the staging buffer's, halved until the grid has about four CTAs per
  // SM (a 320-panel body in 64-column CTAs of FP64 is 15 CTAs: 1.16 ms, 0.14 ms in
  // 4-column CTAs)
  int cols = Prec<R>::kCols;
  const int64_t row_tiles = (nmax + kAsmRows - 1) / kAsmRows;
  while (cols > 4 && row_tiles * ((nmax + cols - 1) / cols) * ninst < 4 * (int64_t)device_sm_count())
    cols /= 2;
  dim3 grid((unsigned)row_tiles, (unsigned)((nmax + cols - 1) / cols), (unsigned)ninst);
  switch (kind) {
    case kAsmBM: k_assemble_regular<R, kAsmBM><<<grid, kAsmRows, 0, L.stream>>>(d, cols, L.err_flag); count_launch(1); break;
    case kAsmCBIE: k_assemble_regular<R, kAsmCBIE><<<grid, kAsmRows, 0, L.stream>>>(d, cols, L.err_flag); count_launch(1); break;
    case kAsmMuller: k_assemble_regular<R, kAsmMuller><<<grid, kAsmRows, 0, L.stream>>>(d, cols, L.err_flag); count_launch(1); break;
    case kAsmRegion: k_assemble_regular<R, kAsmRegion><<<grid, kAsmRows, 0, L.stream>>>(d, cols, L.err_flag); count_launch(1); break;
    default: k_assemble_regular<R, kAsmFluidCBIE><<<grid, kAsmRows, 0, L.stream>>>(d, cols, L.err_flag); count_launch(1); break;
  }
}

void launch_assemble_regular(const Launch& L, const AsmInst* d_inst, int ninst, int64_t nmax,
                             int kind, bool fp32) {
  if (nmax <= 0 || ninst <= 0) return;
  if (fp32)
    launch_regular_t<float>(L, d_inst, ninst, nmax, kind);
  else
    launch_regular_t<double>(L, d_inst, ninst, nmax, kind);
}

template <bool F32>
static void launch_near_t(const Launch& L, const AsmInst* d_inst, int ninst, int64_t max_near,
                          int kind) {
  dim3 grid((unsigned)((max_near + 127) / 128), 1, (unsigned)ninst);
  switch (kind) {
    case kAsmBM: k_assemble_near<kAsmBM, F32><<<grid, 128, 0, L.stream>>>(d_inst); break;
    case kAsmCBIE: k_assemble_near<kAsmCBIE, F32><<<grid, 128, 0, L.stream>>>(d_inst); break;
    case kAsmMuller: k_assemble_near<kAsmMuller, F32><<<grid, 128, 0, L.stream>>>(d_inst); break;
    case kAsmRegion: k_assemble_near<kAsmRegion, F32><<<grid, 128, 0, L.stream>>>(d_inst); break;
    default: k_assemble_near<kAsmFluidCBIE, F32><<<grid, 128, 0, L.stream>>>(d_inst); break;
  }
  count_launch(1);
}

void launch_assemble_near(const Launch& L, const AsmInst* d_inst, int ninst, int64_t max_near,
                          int kind, bool fp32) {
  if (max_near <= 0 || ninst <= 0) return;
  if (fp32)
    launch_near_t<true>(L, d_inst, ninst, max_near, kind);
  else
    launch_near_t<false>(L, d_inst, ninst, max_near, kind);
}

// ------------------------------------------------------------------ incident traces
// p = e^{ik d.c}, q = ik (d.n) p at every collocation point (core/incident.jl:64-76).
__global__ void k_incident(const WaveInst* __restrict__ insts) {
  const WaveInst& W = insts[blockIdx.z];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= W.n || r >= W.nrhs) return;
  const double* rec = W.panels + i * kPanelDoubles;
  const double* d = W.dirs + 3 * r;
  const double ph = W.k * (d[0] * rec[0] + d[1] * rec[1] + d[2] * rec[2]);
  double sn, cs;
  sincos(ph, &sn, &cs);
  const double dn = W.k * (d[0] * rec[3] + d[1] * rec[4] + d[2] * rec[5]);
  const int64_t o = 2 * (i + r * W.ldp);
  W.p[o] = cs;
  W.p[o + 1] = sn;
  W.q[o] = -dn * sn;
  W.q[o + 1] = dn * cs;
}

void launch_incident(const Launch& L, const WaveInst* d_inst, int ninst, int64_t nmax,
                     int32_t max_rhs) {
  if (nmax <= 0 || ninst <= 0 || max_rhs <= 0) return;
  dim3 grid((unsigned)((nmax + 255) / 256), (unsigned)max_rhs, (unsigned)ninst);
  k_incident<<<grid, 256, 0, L.stream>>>(d_inst); count_launch(1);
}

// ------------------------------------------------------------------ far field
// f(xh) = -(1/4pi) sum_j area_j (ik xh.n_j p_j + q_j) sum_g W_g e^{-ik xh.y_jg}
// (solvers/bem/full.jl:509-519).
//
// Bound by FP64 issue (two FMAs per clock and SM), so the work per (panel, direction) is
// what counts.  The seven phases of a panel are one sine / cosine at the centroid times a
// power series: the Gauss points of the 7-point rule lie on the lines from the centroid c to
// the vertices, y - c = lambda (v_m - c), so with t_m = k xh.(y_{4+m} - c), t_0 + t_1 + t_2 = 0,
//   sum_g W_g e^{-ik xh.(y_g - c)} = sum_n c_n (-i)^n P_n,  P_n = t_0^n + t_1^n + t_2^n,
// where c_n = (W_1 rho^n + W_4) / n! (rho: ratio of the two orbits' lambda) and the power
// sums obey P_n = m_2 P_{n-2} + e_3 P_{n-3} (Newton's identities without e_1).  Terms up to
// n = 11 (|t| <= 0.232) or 17 (|t| <= 0.743) leave a remainder below 3e-17; longer panels
// take six more sines and cosines.  Per pair about 80 FP64 instructions instead of about
// 230: 6000 directions of 5120 panels 13.0 -> 5.6 ms on a GB300, one direction of 1280
// panels 20 -> 9 us.
//
// Many directions (>= kFarMany): thread = direction, the panels of a chunk staged in shared
// memory and read by broadcast, no reductions.  Few: thread = panel, one warp per 32 panels,
// which spreads one direction over more SMs.  The lines' crossover is not critical: at 32
// directions both take about the same time.  A second kernel adds the chunk sums.  Every
// sum has a fixed order, so the result does not depend on what else runs on the GPU.
constexpr int kFarChunk = 128;  // panels per chunk, thread = direction
constexpr int kFarFew = 32;     // panels per chunk, thread = panel
constexpr int kFarMany = 32;    // directions from which a thread takes a direction
constexpr int kFarThreads = 128;
constexpr double kFarT11 = 0.232, kFarT17 = 0.743;

size_t far_field_scratch(int64_t n, int32_t ndir, int32_t nrhs) {
  const int64_t per = ndir >= kFarMany ? kFarChunk : kFarFew;
  const int64_t chunks = (n + per - 1) / per;
  return (size_t)chunks * (size_t)ndir * (size_t)nrhs * 2 * sizeof(double);
}

// c_n of the panel phase series, sign of (-i)^n included (even: real, odd: imaginary part)
constexpr double far_coef(int n) {
  // 1 - 3 b of the two orbits (b: the repeated barycentric coordinate)
  constexpr double l1 = 1.0 - 3.0 * kRuleB[1][1], l2 = 1.0 - 3.0 * kRuleB[4][1];
  double r = 1.0, f = 1.0;
  for (int i = 1; i <= n; ++i) {
    r *= l1 / l2;
    f *= (double)i;
  }
  const double s = (n % 4 == 0 || n % 4 == 3) ? 1.0 : -1.0;
  return s * (kRuleW[1] * r + kRuleW[4]) / f;
}

__constant__ double dFarCoef[18] = {
    far_coef(0),  far_coef(1),  far_coef(2),  far_coef(3),  far_coef(4),  far_coef(5),
    far_coef(6),  far_coef(7),  far_coef(8),  far_coef(9),  far_coef(10), far_coef(11),
    far_coef(12), far_coef(13), far_coef(14), far_coef(15), far_coef(16), far_coef(17)};

// One panel's values staged for all directions of a chunk (areas folded into p and q).
struct FarPanel {
  double c[3], n[3], e0[3], e1[3];  // k c, k n, k (y_4 - c), k (y_5 - c)
  double pr, pi, qr, qi;
};

__device__ __forceinline__ void far_panel(const WaveInst& W, int r, int64_t j, FarPanel& F,
                                          double& tmax) {
  const double* rec = W.panels + j * kPanelDoubles;
  const double k = W.k, area = rec[6];
  double m[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    F.c[a] = k * rec[a];
    F.n[a] = k * rec[3 + a];
    const double d0 = k * (rec[8 + 12 + a] - rec[a]), d1 = k * (rec[8 + 15 + a] - rec[a]);
    F.e0[a] = d0;
    F.e1[a] = d1;
    m[0] += d0 * d0;
    m[1] += d1 * d1;
    m[2] += (d0 + d1) * (d0 + d1);
  }
  tmax = fmax(m[0], fmax(m[1], m[2]));  // squared bound of |t_m| over all directions
  const int64_t o = 2 * (j + r * W.ldp);
  F.pr = area * W.p[o];
  F.pi = area * W.p[o + 1];
  F.qr = area * W.q[o];
  F.qi = area * W.q[o + 1];
}

// Adds the panel's contribution for the unit direction x; N: last term of the series, 0: by
// sines and cosines.
template <int N>
__device__ __forceinline__ void far_add(const FarPanel& F, const double x[3], double& ar,
                                        double& ai) {
  const double ph = x[0] * F.c[0] + x[1] * F.c[1] + x[2] * F.c[2];
  const double kxn = x[0] * F.n[0] + x[1] * F.n[1] + x[2] * F.n[2];
  const double t0 = x[0] * F.e0[0] + x[1] * F.e0[1] + x[2] * F.e0[2];
  const double t1 = x[0] * F.e1[0] + x[1] * F.e1[1] + x[2] * F.e1[2];
  double fr = 1.0, fi = 0.0;
  if (N > 0) {
    const double s = t0 + t1, m2 = t0 * s + t1 * t1, e3 = -(t0 * t1) * s;
    double pa = 0.0, pb = 2.0 * m2, pc = 3.0 * e3;  // P_{n-3}, P_{n-2}, P_{n-1} before n = 4
    fr += dFarCoef[2] * pb;
    fi += dFarCoef[3] * pc;
#pragma unroll
    for (int n = 4; n <= N; ++n) {
      const double pn = n == 4 ? m2 * pb : m2 * pb + e3 * pa;
      if (n % 2 == 0)
        fr += dFarCoef[n] * pn;
      else
        fi += dFarCoef[n] * pn;
      pa = pb;
      pb = pc;
      pc = pn;
    }
  } else {
    constexpr double rho = (1.0 - 3.0 * kRuleB[1][1]) / (1.0 - 3.0 * kRuleB[4][1]);
    constexpr double w0 = kRuleW[0], w1 = kRuleW[1], w4 = kRuleW[4];
    fr = w0;
#pragma unroll 1
    for (int m = 0; m < 3; ++m) {
      const double t = m == 0 ? t0 : m == 1 ? t1 : -(t0 + t1);
      double s1, c1, s2, c2;
      sincos(rho * t, &s1, &c1);
      sincos(t, &s2, &c2);
      fr += w1 * c1 + w4 * c2;
      fi -= w1 * s1 + w4 * s2;
    }
  }
  double sn, cs;
  sincos(ph, &sn, &cs);
  // (i kxn p + q) f e^{-i ph}
  const double br = F.qr - kxn * F.pi, bi = F.qi + kxn * F.pr;
  const double gr = br * fr - bi * fi, gi = br * fi + bi * fr;
  ar += gr * cs + gi * sn;
  ai += gi * cs - gr * sn;
}

// thread = direction: grid (directions / 128, chunks, instance x rhs)
__global__ void __launch_bounds__(kFarThreads) k_far_field_many(WaveInst w0,
                                                                const WaveInst* insts,
                                                                int max_rhs) {
  const WaveInst& W = insts ? insts[blockIdx.z / max_rhs] : w0;
  const int r = (int)(blockIdx.z % max_rhs);
  const int64_t nchunks = (W.n + kFarChunk - 1) / kFarChunk, chunk = blockIdx.y;
  const int64_t d0 = (int64_t)blockIdx.x * kFarThreads;
  if (r >= W.nrhs || chunk >= nchunks || d0 >= W.ndir) return;  // uniform over the CTA
  __shared__ FarPanel sp[kFarChunk];
  const int64_t j0 = chunk * kFarChunk;
  const int cnt = (int)min((int64_t)kFarChunk, W.n - j0);
  double tm = 0.0;
  if (threadIdx.x < cnt) far_panel(W, r, j0 + threadIdx.x, sp[threadIdx.x], tm);
  const bool over11 = __syncthreads_or(!(tm <= kFarT11 * kFarT11));
  const bool over17 = __syncthreads_or(!(tm <= kFarT17 * kFarT17));
  const int64_t d = d0 + threadIdx.x;
  if (d >= W.ndir) return;
  const double* xh = W.dirs + 3 * ((int64_t)r * W.ndir + d);
  const double x[3] = {xh[0], xh[1], xh[2]};
  double ar = 0.0, ai = 0.0;
  if (!over11)
    for (int j = 0; j < cnt; ++j) far_add<11>(sp[j], x, ar, ai);
  else if (!over17)
    for (int j = 0; j < cnt; ++j) far_add<17>(sp[j], x, ar, ai);
  else
    for (int j = 0; j < cnt; ++j) far_add<0>(sp[j], x, ar, ai);
  double* o = W.part + 2 * (((int64_t)r * W.ndir + d) * nchunks + chunk);
  o[0] = ar;
  o[1] = ai;
}

// thread = panel: grid (direction x rhs, groups of 4 chunks, instance), a warp per chunk
__global__ void __launch_bounds__(kFarThreads) k_far_field_few(WaveInst w0,
                                                               const WaveInst* insts) {
  const WaveInst& W = insts ? insts[blockIdx.z] : w0;
  const int64_t dr = blockIdx.x;
  const int64_t nchunks = (W.n + kFarFew - 1) / kFarFew;
  const int64_t chunk = (int64_t)blockIdx.y * (kFarThreads / 32) + (threadIdx.x >> 5);
  if (dr >= (int64_t)W.ndir * W.nrhs || chunk >= nchunks) return;  // uniform per warp
  const int r = (int)(dr / W.ndir);
  const double* xh = W.dirs ? W.dirs + 3 * dr : W.dir1;
  const double x[3] = {xh[0], xh[1], xh[2]};
  const int lane = threadIdx.x & 31;
  const int64_t j = chunk * kFarFew + lane;
  double ar = 0.0, ai = 0.0, tm = 0.0;
  FarPanel F;
  if (j < W.n) far_panel(W, r, j, F, tm);
  const bool over11 = __any_sync(0xffffffffu, !(tm <= kFarT11 * kFarT11));
  const bool over17 = __any_sync(0xffffffffu, !(tm <= kFarT17 * kFarT17));
  if (j < W.n) {
    if (!over11)
      far_add<11>(F, x, ar, ai);
    else if (!over17)
      far_add<17>(F, x, ar, ai);
    else
      far_add<0>(F, x, ar, ai);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    ar += __shfl_down_sync(0xffffffffu, ar, off);
    ai += __shfl_down_sync(0xffffffffu, ai, off);
  }
  if (lane == 0) {
    double* o = W.part + 2 * (dr * nchunks + chunk);
    o[0] = ar;
    o[1] = ai;
  }
}

// one warp per (direction, rhs): its chunk sums, lane-strided, then a shuffle tree
__global__ void __launch_bounds__(kFarThreads) k_far_field_finish(WaveInst w0,
                                                                  const WaveInst* insts, int per) {
  const WaveInst& W = insts ? insts[blockIdx.z] : w0;
  const int64_t dr = (int64_t)blockIdx.x * (kFarThreads / 32) + (threadIdx.x >> 5);
  if (dr >= (int64_t)W.ndir * W.nrhs) return;
  const int64_t nchunks = (W.n + per - 1) / per;
  const double2* part = reinterpret_cast<const double2*>(W.part) + dr * nchunks;
  double tr = 0.0, ti = 0.0;
  for (int64_t c = threadIdx.x & 31; c < nchunks; c += 32) {
    const double2 v = part[c];
    tr += v.x;
    ti += v.y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    tr += __shfl_down_sync(0xffffffffu, tr, off);
    ti += __shfl_down_sync(0xffffffffu, ti, off);
  }
  if ((threadIdx.x & 31) == 0) {
    W.out[2 * dr] = -tr * kInv4Pi;
    W.out[2 * dr + 1] = -ti * kInv4Pi;
  }
}

static void far_field(const Launch& L, const WaveInst& w0, const WaveInst* d_inst, int ninst,
                      int32_t max_rhs, int32_t max_dirs, int64_t max_n) {
  if (ninst <= 0 || max_dirs <= 0 || max_rhs <= 0 || max_n <= 0) return;
  const int64_t dr = (int64_t)max_dirs * max_rhs;
  const bool many = max_dirs >= kFarMany;
  const int per = many ? kFarChunk : kFarFew;
  const int64_t chunks = (max_n + per - 1) / per;
  if (many)
    k_far_field_many<<<dim3((unsigned)((max_dirs + kFarThreads - 1) / kFarThreads),
                            (unsigned)chunks, (unsigned)(ninst * max_rhs)),
                       kFarThreads, 0, L.stream>>>(w0, d_inst, max_rhs);
  else
    k_far_field_few<<<dim3((unsigned)dr, (unsigned)((chunks + 3) / 4), (unsigned)ninst),
                      kFarThreads, 0, L.stream>>>(w0, d_inst);
  k_far_field_finish<<<dim3((unsigned)((dr + 3) / 4), 1, (unsigned)ninst), kFarThreads, 0,
                       L.stream>>>(w0, d_inst, per);
  count_launch(2);
}

void launch_far_field(const Launch& L, const WaveInst* d_inst, int ninst, int32_t max_rhs,
                      int32_t max_dirs, int64_t max_n) {
  far_field(L, WaveInst{}, d_inst, ninst, max_rhs, max_dirs, max_n);
}

void launch_far_field_one(const Launch& L, const WaveInst& w) {
  far_field(L, w, nullptr, 1, w.nrhs, w.ndir, w.n);
}

}  // namespace bemgpu
