// Matrix-vector work around the factorisation: equilibration (solvers/bem/full.jl:388-394,
// solvers/bem/fluid_system.jl:202-216), scaled low-precision copies, products with the
// complex128 system (right-hand sides, residuals, componentwise denominators), the
// backward-error statistics of fluid_system.jl:241-262 and the correction steps of
// fluid_system.jl:229-239.
//
// Column-major matrices are swept with one thread per row (consecutive threads read
// consecutive rows of a column: coalesced), and the columns are split into vec_chunks(n)
// chunks whose partial results are combined by a second kernel in a fixed order, so
// every reduction here is deterministic.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "bemgpu_internal.h"
#include "gemm_oz.cuh"
#include "linalg.cuh"
#include "refine.cuh"

namespace bemgpu {

__device__ __forceinline__ cd ldc(const void* base, int64_t idx) {
  double2 v = reinterpret_cast<const double2*>(base)[idx];
  return {v.x, v.y};
}
__device__ __forceinline__ void stc(void* base, int64_t idx, cd v) {
  reinterpret_cast<double2*>(base)[idx] = make_double2(v.x, v.y);
}
__device__ __forceinline__ double cabs(cd a) { return hypot(a.x, a.y); }
// The nearest float of a (ties away from zero; below the normal range 0), by integer
// instructions: a conversion instruction of a double takes a turn of the FP64 pipe, and four of
// them per entry were half of the pipe's work in the products of complex128 systems.
__device__ __forceinline__ float near_float(double a) {
  const uint32_t hi = (uint32_t)__double2hiint(a) & 0x7fffffffu, lo = (uint32_t)__double2loint(a);
  if (hi < 0x38100000u) return 0.f;                       // |a| < 2^-126
  if (hi >= 0x47f00000u)                                  // |a| >= 2^128, infinity, NaN
    return hi > 0x7ff00000u || (hi == 0x7ff00000u && lo) ? NAN : INFINITY;
  return __uint_as_float(__funnelshift_l(lo, hi - 0x38000000u, 3) + ((lo >> 28) & 1u));
}
// Magnitude for scales, norms and componentwise denominators: single precision is
// ample there (relative 1e-7), and GB300 issues FP64 at a small fraction of FP32.
__device__ __forceinline__ float fabs_c(cd a) {
  const float x = near_float(a.x), y = near_float(a.y);
  return sqrtf(fmaf(x, x, y * y));
}

__device__ __forceinline__ void chunk_range(int64_t n, int ch, int nch, int64_t* j0, int64_t* j1) {
  int64_t w = (n + nch - 1) / nch;
  *j0 = min(n, (int64_t)ch * w);
  *j1 = min(n, *j0 + w);
}

// Element access of the system: complex128, or complex64 for compact instances (a32).
__device__ __forceinline__ float2 ldf(const void* base, int64_t idx) {
  return reinterpret_cast<const float2*>(base)[idx];
}
template <bool A32>
struct Entry {
  using T = cd;
  static __device__ __forceinline__ T at(const VecInst& V, int64_t idx) { return ldc(V.A, idx); }
  static __device__ __forceinline__ float mag(T a) { return fabs_c(a); }
};
template <>
struct Entry<true> {
  using T = float2;
  static __device__ __forceinline__ T at(const VecInst& V, int64_t idx) { return ldf(V.A, idx); }
  static __device__ __forceinline__ float mag(T a) { return sqrtf(fmaf(a.x, a.x, a.y * a.y)); }
};
// Row-wise products of a system whose digit products were good enough (VecInst::gate).
__device__ __forceinline__ bool closed(const VecInst& V) { return V.gate && *V.gate <= V.gate_cap; }
template <bool A32>
__device__ __forceinline__ float mag_at(const VecInst& V, int64_t idx) {
  return Entry<A32>::mag(Entry<A32>::at(V, idx));
}

// ---------------------------------------------------------------- equilibration
template <bool A32>
__device__ __forceinline__ void rowstats_body(const VecInst& V) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  int64_t j0, j1;
  if (blockIdx.y >= vec_chunks(V.n)) return;
  chunk_range(V.n, blockIdx.y, vec_chunks(V.n), &j0, &j1);
  using E = Entry<A32>;
  float mx = 0.f, sm32 = 0.f;
  double sm = 0.0;
  auto take = [&](typename E::T v) {
    const float a = E::mag(v);
    mx = fmaxf(mx, a);
    sm32 += a;
  };
  constexpr int kB = A32 ? 16 : 8;  // columns loaded before the first is used
  for (int64_t jf = j0; jf < j1; jf += 256) {  // fold into FP64 every 256 terms
    const int64_t jf1 = min(j1, jf + 256);
    int64_t j = jf;
    for (; j + kB <= jf1; j += kB) {
      typename E::T a[kB];
#pragma unroll
      for (int q = 0; q < kB; ++q) a[q] = E::at(V, i + (j + q) * V.lda);
#pragma unroll
      for (int q = 0; q < kB; ++q) take(a[q]);
    }
    for (; j < jf1; ++j) take(E::at(V, i + j * V.lda));
    sm += sm32;
    sm32 = 0.f;
  }
  V.part[2 * (blockIdx.y * V.n + i)] = mx;
  V.part[2 * (blockIdx.y * V.n + i) + 1] = sm;
}
__global__ void k_rowstats(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.z];
  if (V.a32)
    rowstats_body<true>(V);
  else
    rowstats_body<false>(V);
}

__global__ void k_rowstats_finish(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.y];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  double mx = 0.0, sm = 0.0;
  const int chunks = vec_chunks(V.n);
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) {
    mx = fmax(mx, V.part[2 * (c * V.n + i)]);
    sm += V.part[2 * (c * V.n + i) + 1];
  }
  mx = fmax(mx, V.norm_floor);  // the reference's norm_floor (full.jl:388-394)
  V.rows[i] = (mx == 0.0) ? 1.0 : mx;
  V.rows_inv[i] = (float)(1.0 / V.rows[i]);
  V.rowsum[i] = sm;
}

// columns[j] = max_i |A_ij / rows_i|, one warp per column
template <bool A32>
__device__ __forceinline__ void colmax_body(const VecInst& V) {
  const int64_t j = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= V.n) return;
  float mx = 0.f;
  const int64_t n = V.n, base = j * V.lda;
  int64_t i = lane;
  constexpr int kB = 8;
  for (; i + 32 * (kB - 1) < n; i += 32 * kB) {
    typename Entry<A32>::T a[kB];
    float w[kB];
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      a[q] = Entry<A32>::at(V, base + i + 32 * q);
      w[q] = V.rows_inv[i + 32 * q];
    }
#pragma unroll
    for (int q = 0; q < kB; ++q) mx = fmaxf(mx, Entry<A32>::mag(a[q]) * w[q]);
  }
  for (; i < n; i += 32) mx = fmaxf(mx, mag_at<A32>(V, base + i) * V.rows_inv[i]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, off));
  if (lane == 0) {
    const double cm = fmax((double)mx, V.norm_floor);
    V.cols[j] = (cm == 0.0) ? 1.0 : cm;
  }
}
__global__ void k_colmax(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.y];
  if (V.a32)
    colmax_body<true>(V);
  else
    colmax_body<false>(V);
}

__global__ void k_cols_inv(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.y];
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < V.n) {
    V.cols_inv[j] = 1.0 / V.cols[j];
    if (V.cols_inv32) V.cols_inv32[j] = (float)V.cols_inv[j];
    if (V.rows_inv) V.rows_inv[j] = (float)(1.0 / V.rows[j]);  // rows may have been reset
  }
}

// out_ij = A_ij / rows_i / cols_j (complex64 or complex128); partial row sums of |out|.
// The complex64 copy scales in FP32 by the FP32 reciprocals (a rounding-level change of
// the scaling that the refinement, which uses the FP64 scales, absorbs).
template <bool A32>
__device__ __forceinline__ void scale_copy_body(const VecInst& V) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V.n) return;
  int64_t j0, j1;
  if (blockIdx.y >= vec_chunks(V.n)) return;
  chunk_range(V.n, blockIdx.y, vec_chunks(V.n), &j0, &j1);
  double sm = 0.0;
  float sm32 = 0.f;
  int cnt = 0;
  bool bad = false;
  if (V.out_single) {
    const float ri = V.rows_inv[i];
    constexpr int kB = 8;
    for (int64_t jb = j0; jb < j1; jb += kB) {
      const int nb = (int)min((int64_t)kB, j1 - jb);
      float2 a[kB];
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        if (q < nb) {
          if (A32) {
            a[q] = ldf(V.A, i + (jb + q) * V.lda);
          } else {
            const cd d = ldc(V.A, i + (jb + q) * V.lda);
            a[q] = make_float2((float)d.x, (float)d.y);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        if (q < nb) {
          const float fs = ri * V.cols_inv32[jb + q];
          const float2 f = make_float2(a[q].x * fs, a[q].y * fs);
          reinterpret_cast<float2*>(V.out)[i + (jb + q) * V.n] = f;
          bad |= !(isfinite(f.x) && isfinite(f.y));
          sm32 += sqrtf(fmaf(f.x, f.x, f.y * f.y));
        }
      }
      cnt += nb;
      if (cnt >= 256) {  // fold into FP64 every 256 terms
        sm += sm32;
        sm32 = 0.f;
        cnt = 0;
      }
    }
    sm += sm32;
  } else {
    const double ri = 1.0 / V.rows[i];
    for (int64_t j = j0; j < j1; ++j) {
      cd a;
      if (A32) {
        const float2 f = ldf(V.A, i + j * V.lda);
        a = cd{(double)f.x, (double)f.y};
      } else {
        a = ldc(V.A, i + j * V.lda);
      }
      const double sc = ri * V.cols_inv[j];
      cd v = {a.x * sc, a.y * sc};
      stc(V.out, i + j * V.n, v);
      bad |= !(isfinite(v.x) && isfinite(v.y));
      sm += fabs_c(v);
    }
  }
  V.part[blockIdx.y * V.n + i] = sm;
  if (bad) atomicExch(V.flag, 1);
}
__global__ void k_scale_copy(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.z];
  if (V.a32)
    scale_copy_body<true>(V);
  else
    scale_copy_body<false>(V);
}

// stats[0] = max_i rowsum_i (||A||_inf), stats[1] = max_i sum_c part (||scaled||_inf)
constexpr int kNormT = 1024;
__global__ void __launch_bounds__(kNormT) k_norms_finish(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.x];
  __shared__ double s0[kNormT], s1[kNormT];
  double m0 = 0.0, m1 = 0.0;
  const int chunks = vec_chunks(V.n);
  for (int64_t i = threadIdx.x; i < V.n; i += kNormT) {
    double t = 0.0;
#pragma unroll 8
    for (int c = 0; c < chunks; ++c) t += V.part[c * V.n + i];
    m0 = fmax(m0, V.rowsum[i]);
    m1 = fmax(m1, t);
  }
  s0[threadIdx.x] = m0;
  s1[threadIdx.x] = m1;
  __syncthreads();
  for (int s = kNormT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      s0[threadIdx.x] = fmax(s0[threadIdx.x], s0[threadIdx.x + s]);
      s1[threadIdx.x] = fmax(s1[threadIdx.x], s1[threadIdx.x + s]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    V.stats[0] = s0[0];
    V.stats[1] = s1[0];
  }
}

// ---------------------------------------------------------------- compact storage helpers
// out += near corrections (scaled unless unit); one thread per (near pair, block)
__global__ void k_near_add(const VecInst* __restrict__ insts, int unit) {
  const VecInst& V = insts[blockIdx.z];
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (!V.a32 || p >= V.n_near || b >= V.nbc * V.nbc) return;
  const int br = b / V.nbc, bc = b % V.nbc;
  const int64_t row = br * V.n_mesh + V.near_i[p], col = bc * V.n_mesh + V.near_j[p];
  const cd d = ldc(V.dnear, (int64_t)b * V.n_near + p);
  const double sc = unit ? 1.0 : (1.0 / V.rows[row]) * V.cols_inv[col];
  const int64_t o = row + col * V.n;
  cd v = ldc(V.out, o);
  stc(V.out, o, cd{v.x + d.x * sc, v.y + d.y * sc});
}

__global__ void k_expand_a32(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.z];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!V.a32 || i >= V.n) return;
  for (int64_t j = blockIdx.y; j < V.n; j += gridDim.y) {
    const float2 f = ldf(V.A, i + j * V.lda);
    stc(V.out, i + j * V.n, cd{(double)f.x, (double)f.y});
  }
}

// x split for the compact products: hi = fl32(x), lo = fl32(x - hi), every part twice (the paired
// instructions take it for two rows)
__global__ void k_split_x(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.z];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (!V.a32 || i >= V.n || r >= V.nrhs || closed(V)) return;
  const cd x = ldc(V.x, i + (int64_t)r * V.ldx);
  const float hr = (float)x.x, hi = (float)x.y;
  const float lr = (float)(x.x - (double)hr), li = (float)(x.y - (double)hi);
  float4* xs = V.xs + 2 * (i + (int64_t)r * V.n);
  xs[0] = make_float4(hr, hr, hi, hi);
  xs[1] = make_float4(lr, lr, li, li);
  V.xa[i + (int64_t)r * V.n] = sqrtf(fmaf(hr, hr, hi * hi));
}

// ---------------------------------------------------------------- products
// Compact products in FP32 pair arithmetic.  A complex64 entry times the split x
// (hi + lo): each product a * hi is exact as p + e (round-to-nearest product and its FMA
// error), p enters a (s, t) pair by TwoSum (s + t carries the sum exactly up to the FP32
// rounding of t), and e and a * lo go into t.  Every 32 columns (128 real products) the
// pair is folded into FP64, so t holds at most that many terms' errors.  What is left is
// the FP32 rounding of t: for an exact solution the computed residual stays below about
// 6e-14 of |b| + |A||x| in every row of small Burton-Miller and Mueller systems, where a
// dominant diagonal block carries most of a row (median about 3e-15; an operation-by-
// operation emulation on the CPU), under the refinement's 1e-13 acceptance, at a small
// fraction of the FP64 instruction count of the complex128 path.  The intrinsics keep the
// compiler from contracting or reassociating the error-free steps.
// Two rows go through the paired FP32 instructions, which round each half as the single ones do.
// a - b and -a through products with -1, which are exact: one instruction each.
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 f2_neg(float2 a) {
  return __fmul2_rn(a, make_float2(-1.f, -1.f));
}
struct FPair {
  float2 s, t;
};
// a += u v, nu = -u
__device__ __forceinline__ void pair_add_prod(FPair& a, float2 u, float2 nu, float2 v) {
  const float2 p = __fmul2_rn(u, v);
  const float2 e = __ffma2_rn(nu, v, p);  // -(the product's error)
  const float2 s = __fadd2_rn(a.s, p);
  const float2 bb = f2_sub(s, a.s);
  const float2 err = __fadd2_rn(f2_sub(a.s, f2_sub(s, bb)), f2_sub(p, bb));
  a.s = s;
  a.t = __fadd2_rn(a.t, f2_sub(err, e));
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

template <int NR>
__device__ __forceinline__ void gemv_body(const VecInst& V, int grp0, int with_abs) {
  constexpr int kGemvR = NR;  // right-hand sides per pass of this instantiation
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int ch = blockIdx.y % kMaxChunks, grp = grp0 + blockIdx.y / kMaxChunks;
  if (ch >= vec_chunks(V.n, V.nrhs)) return;
  const int r0 = grp * kGemvR;
  if (i >= V.n || r0 >= V.nrhs) return;
  const int nr = min(kGemvR, V.nrhs - r0);
  int64_t j0, j1;
  chunk_range(V.n, ch, vec_chunks(V.n, V.nrhs), &j0, &j1);
  cd acc[kGemvR];
  float aacc[kGemvR];
#pragma unroll
  for (int r = 0; r < kGemvR; ++r) {
    acc[r] = cd{0.0, 0.0};
    aacc[r] = 0.f;
  }
  constexpr int kBatch = 4;  // columns loaded before the first is used
  for (int64_t jb = j0; jb < j1; jb += kBatch) {
    const int cnt = (int)min((int64_t)kBatch, j1 - jb);
    cd a[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      a[q] = q < cnt ? ldc(V.A, i + (jb + q) * V.lda) : cd{0.0, 0.0};
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      if (q < cnt) {
        const float aa = with_abs ? fabs_c(a[q]) : 0.f;
#pragma unroll
        for (int r = 0; r < kGemvR; ++r) {
          if (r < nr) {
            const cd x = ldc(V.x, jb + q + (int64_t)(r0 + r) * V.ldx);
            acc[r].x = fma(a[q].x, x.x, fma(-a[q].y, x.y, acc[r].x));
            acc[r].y = fma(a[q].x, x.y, fma(a[q].y, x.x, acc[r].y));
            if (with_abs) aacc[r] = fmaf(aa, fabs_c(x), aacc[r]);
          }
        }
      }
    }
  }
  // part layout: [chunk][rhs][row] x (re, im, abs)
#pragma unroll
  for (int r = 0; r < kGemvR; ++r) {
    if (r < nr) {
      int64_t o = 3 * (((int64_t)ch * V.nrhs + r0 + r) * V.n + i);
      V.part[o] = acc[r].x;
      V.part[o + 1] = acc[r].y;
      V.part[o + 2] = (double)aacc[r];
    }
  }
}

// Compact instances: a thread takes two rows (T apart: coalesced) as the halves of the paired
// instructions.  Its columns come through a ring of its own in shared memory, kA32Stages groups of
// kA32Cols ahead by asynchronous copies, so that no thread waits for another one: with the loads in
// registers the kernel waited for them half of the time, 1.69 ms for four systems of 10240
// unknowns (3.4 GB, 0.53 ms of reading); now 1.23 ms, of which the issue of about 54 instructions
// per entry (14 of them for |A||x|) is half.  The sums are folded into FP64 every kFold columns.
// T (64 or 128) is a launch shape of the autotuner; it does not change any row's arithmetic.
constexpr int kA32Cols = 4, kA32Stages = 4;
constexpr int a32_smem(int threads) { return kA32Stages * kA32Cols * 2 * 8 * threads; }

template <int NR, bool ABS, int T>
__global__ void __launch_bounds__(T, (NR == 1 ? 640 : 512) / T)
    k_gemv_a32(const VecInst* __restrict__ insts, int grp0) {
  constexpr int kFold = 32, kRows = 2;
  const VecInst& V = insts[blockIdx.z];
  if (!V.a32 || closed(V)) return;
  extern __shared__ __align__(16) unsigned char a32_ring[];
  const int64_t n = V.n, lda = V.lda;
  const int64_t i0 = (int64_t)blockIdx.x * (kRows * T) + threadIdx.x;
  const int ch = blockIdx.y % kMaxChunks, grp = grp0 + blockIdx.y / kMaxChunks;
  if (ch >= vec_chunks(n, V.nrhs)) return;
  const int r0 = grp * NR;
  if (i0 >= n || r0 >= V.nrhs) return;
  const int nr = min(NR, V.nrhs - r0);
  int64_t j0, j1;
  chunk_range(n, ch, vec_chunks(n, V.nrhs), &j0, &j1);
  const int cols = (int)(j1 - j0), groups = cols / kA32Cols;  // whole groups
  const float2* A[kRows];  // rows past the last: the first one again
#pragma unroll
  for (int h = 0; h < kRows; ++h)
    A[h] = reinterpret_cast<const float2*>(V.A) + (i0 + T * h < n ? i0 + T * h : i0) + j0 * lda;
  // column q, row h of group g: ring[((g % kA32Stages) kA32Cols + q) kRows + h][thread]
  float2* ring = reinterpret_cast<float2*>(a32_ring) + threadIdx.x;
  const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring);
  constexpr uint32_t kGroup = kA32Cols * kRows * T;  // entries
  int fetched = 0;
  uint32_t to = 0, from = 0;
  auto fetch = [&]() {
    if (fetched < groups) {
      const uint32_t at = ring_at + to * 8;
#pragma unroll
      for (int q = 0; q < kA32Cols; ++q)
#pragma unroll
        for (int h = 0; h < kRows; ++h) {
          cp_async8(at + (kRows * q + h) * T * 8, A[h]);
          A[h] += lda;
        }
    }
    ++fetched;
    to = to == (kA32Stages - 1) * kGroup ? 0 : to + kGroup;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int g = 0; g < kA32Stages - 1; ++g) fetch();
  const float4* xs[NR];
  const float* xa[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int64_t rr = (int64_t)(r0 + (r < nr ? r : 0)) * n + j0;
    xs[r] = V.xs + 2 * rr;
    xa[r] = V.xa + rr;
  }
  cd acc[kRows][NR];
  float aacc[kRows][NR];
#pragma unroll
  for (int h = 0; h < kRows; ++h)
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      acc[h][r] = cd{0.0, 0.0};
      aacc[h][r] = 0.f;
    }
  FPair re[NR], im[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) re[r] = im[r] = FPair{};
  // column c past xs and xa
  auto column = [&](float2 a0, float2 a1, int c) {
    const float2 ax = make_float2(a0.x, a1.x), ay = make_float2(a0.y, a1.y);
    const float2 nax = f2_neg(ax), nay = f2_neg(ay);
    float m0 = 0.f, m1 = 0.f;
    if (ABS) {
      m0 = sqrtf(fmaf(a0.x, a0.x, a0.y * a0.y));
      m1 = sqrtf(fmaf(a1.x, a1.x, a1.y * a1.y));
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const float4 hi = xs[r][2 * c], lo = xs[r][2 * c + 1];  // (re re, im im)
      const float2 hr = make_float2(hi.x, hi.y), hm = make_float2(hi.z, hi.w);
      const float2 lr = make_float2(lo.x, lo.y), lm = make_float2(lo.z, lo.w);
      // re += a.x x.re - a.y x.im ; im += a.x x.im + a.y x.re
      pair_add_prod(re[r], ax, nax, hr);
      pair_add_prod(re[r], nay, ay, hm);
      pair_add_prod(im[r], ax, nax, hm);
      pair_add_prod(im[r], ay, nay, hr);
      re[r].t = __ffma2_rn(ax, lr, __ffma2_rn(nay, lm, re[r].t));
      im[r].t = __ffma2_rn(ax, lm, __ffma2_rn(ay, lr, im[r].t));
      if (ABS) {
        const float xm = xa[r][c];
        aacc[0][r] = fmaf(m0, xm, aacc[0][r]);
        aacc[1][r] = fmaf(m1, xm, aacc[1][r]);
      }
    }
  };
  auto fold = [&]() {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      acc[0][r].x += (double)re[r].s.x + (double)re[r].t.x;
      acc[0][r].y += (double)im[r].s.x + (double)im[r].t.x;
      acc[1][r].x += (double)re[r].s.y + (double)re[r].t.y;
      acc[1][r].y += (double)im[r].s.y + (double)im[r].t.y;
      re[r] = im[r] = FPair{};
    }
  };
  for (int g = 0; g < groups; ++g) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kA32Stages - 2) : "memory");
    const float2* at = ring + from;
    from = from == (kA32Stages - 1) * kGroup ? 0 : from + kGroup;
#pragma unroll
    for (int q = 0; q < kA32Cols; ++q) column(at[(2 * q) * T], at[(2 * q + 1) * T], q);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      xs[r] += 2 * kA32Cols;
      xa[r] += kA32Cols;
    }
    fetch();  // into the group read before this one
    if ((g + 1) % (kFold / kA32Cols) == 0) fold();
  }
  for (int c = 0; c < cols - groups * kA32Cols; ++c) {  // A stands behind the whole groups
    column(*A[0], *A[1], c);
    A[0] += lda;
    A[1] += lda;
  }
  fold();
  // part layout: [chunk][rhs][row] x (re, im, abs)
#pragma unroll
  for (int h = 0; h < kRows; ++h) {
    const int64_t i = i0 + T * h;
    if (i >= n) break;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      if (r < nr) {
        const int64_t o = 3 * (((int64_t)ch * V.nrhs + r0 + r) * n + i);
        V.part[o] = acc[h][r].x;
        V.part[o + 1] = acc[h][r].y;
        V.part[o + 2] = (double)aacc[h][r];
      }
    }
  }
}

template <int NR, bool ABS, int T>
void gemv_a32(const Launch& L, const VecInst* d, int ninst, int64_t nmax, int grp0, int groups) {
  static PerDeviceOnce attr;
  attr.call([] {
    cudaFuncSetAttribute(k_gemv_a32<NR, ABS, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         a32_smem(T));
  });
  constexpr int rows = 2 * T;
  k_gemv_a32<NR, ABS, T><<<dim3((unsigned)((nmax + rows - 1) / rows),
                                (unsigned)(kMaxChunks * groups), (unsigned)ninst),
                           T, a32_smem(T), L.stream>>>(d, grp0);
}
template <int NR, bool ABS>
void gemv_a32(const Launch& L, const VecInst* d, int ninst, int64_t nmax, int grp0, int groups,
              int rows) {
  if (rows == 1)
    gemv_a32<NR, ABS, 64>(L, d, ninst, nmax, grp0, groups);
  else
    gemv_a32<NR, ABS, 128>(L, d, ninst, nmax, grp0, groups);
}

// partial y = A x (and |A||x|) over a column chunk, up to kGemvR right-hand sides
// per pass (rhs group = grp0 + blockIdx.y / kMaxChunks).
template <int NR>
__global__ void __launch_bounds__(256) k_gemv_part(const VecInst* __restrict__ insts, int grp0,
                                                   int with_abs) {
  const VecInst& V = insts[blockIdx.z];
  if (V.a32 || closed(V)) return;
  gemv_body<NR>(V, grp0, with_abs);
}

// Lane s of the eight threads of a row: its share of the row's near corrections (FP64, every
// eighth pair) times x, added to t.
__device__ __forceinline__ void near_product(const VecInst& V, int64_t i, int r, int s, cd& t) {
  const int br = i >= V.n_mesh ? 1 : 0;
  const int64_t im_ = i - br * V.n_mesh;
  const int32_t p1 = V.near_ptr[im_ + 1];
  for (int32_t p = V.near_ptr[im_] + s; p < p1; p += 8) {
    const int64_t j = V.near_j[p];
    for (int bc = 0; bc < V.nbc; ++bc) {
      const cd d = ldc(V.dnear, (int64_t)(br * V.nbc + bc) * V.n_near + p);
      const cd x = ldc(V.x, j + bc * V.n_mesh + (int64_t)r * V.ldx);
      t.x = fma(d.x, x.x, fma(-d.y, x.y, t.x));
      t.y = fma(d.x, x.y, fma(d.y, x.x, t.y));
    }
  }
}
__device__ __forceinline__ double row8_sum(double v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// mode 0: y = A x.  mode 1: y = b - A x, den = |b| + |A||x|.  Compact instances add the near
// corrections of the row.  Eight threads per row (a chunk sum and a list of about 30 pairs is a
// chain of dependent loads: 41 us for 1280 rows with one thread, 12 us with eight), their
// shares added by a fixed tree.
__global__ void k_gemv_finish(const VecInst* __restrict__ insts, int mode) {
  const VecInst& V = insts[blockIdx.z];
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int r = blockIdx.y, s = threadIdx.x & 7;
  if (r >= V.nrhs || closed(V)) return;
  const bool on = i < V.n;
  double re = 0.0, im = 0.0, ab = 0.0;
  if (on) {
    const int chunks = vec_chunks(V.n, V.nrhs);
    for (int c = s; c < chunks; c += 8) {
      const int64_t o = 3 * (((int64_t)c * V.nrhs + r) * V.n + i);
      re += V.part[o];
      im += V.part[o + 1];
      ab += V.part[o + 2];
    }
    if (V.a32) {
      cd t = {re, im};
      near_product(V, i, r, s, t);
      re = t.x;
      im = t.y;
    }
  }
  re = row8_sum(re);
  im = row8_sum(im);
  ab = row8_sum(ab);
  if (!on || s != 0) return;
  const int64_t yo = i + (int64_t)r * V.ldy;
  if (mode == 0) {
    stc(V.y, yo, cd{re, im});
  } else {
    cd b = ldc(V.b, i + (int64_t)r * V.ldb);
    stc(V.y, yo, cd{b.x - re, b.y - im});
    V.den[yo] = cabs(b) + ab;
  }
}

// ---------------------------------------------------------------- many right-hand sides
// kexp[j]: the largest FP64 exponent field (0: none) of the finite x_jr over the vectors r, 32
// unknowns per CTA, eight threads each
__global__ void __launch_bounds__(256) k_wide_scale(const VecInst V, int32_t* __restrict__ kexp) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t j = (int64_t)blockIdx.x * 32 + tx;
  int mx = 0;
  if (j < V.n)
    for (int r = ty; r < V.nrhs; r += 8) {
      const cd x = ldc(V.x, j + (int64_t)r * V.ldx);
      const int ex = (__double2hiint(x.x) >> 20) & 0x7FF, ey = (__double2hiint(x.y) >> 20) & 0x7FF;
      if (ex != 0x7FF) mx = max(mx, ex);
      if (ey != 0x7FF) mx = max(mx, ey);
    }
  __shared__ int sh[8][32];
  sh[ty][tx] = mx;
  __syncthreads();
  if (ty == 0 && j < V.n) {
    for (int u = 1; u < 8; ++u) mx = max(mx, sh[u][tx]);
    kexp[j] = mx;
  }
}

void launch_wide_scale(const Launch& L, const VecInst& v, int32_t* kexp) {
  k_wide_scale<<<(unsigned)((v.n + 31) / 32), 256, 0, L.stream>>>(v, kexp);
  count_launch(1);
}

// The digit products' error bound.  With one exponent per row of A and per vector in a block of
// 128 columns, the error of y_ir is a few times 2^-56 E_ir, E_ir = sum over the blocks of
// 2^(aexp + bexp), about 16 max|a| max|x| of the block (up to 8 times for entries of mixed signs
// and 30 for equal ones, whose E is about |A||x|; random, Burton-Miller and fluid systems of up
// to 640 unknowns on the CPU).  Entries with E above a multiple of |A||x| (large x meet small a)
// are listed for k_wide_redo.  The multiple: 32 for right-hand sides, whose E stays below it for
// bodies of 560 to 20480 panels; 64 for residuals of complex128 systems (up to 1 % of the
// entries of rigid bodies are above it, those in the shadow of a direction); 256 for those of
// compact ones (one entry in 64000), which leaves errors below 3e-14 of |A||x|, half of what
// the paired FP32 products may reach.
__device__ __forceinline__ double wide_spread(const VecInst& V, int mode) {
  return mode == 0 ? 32.0 : V.a32 ? 256.0 : 64.0;
}
constexpr int kChkRows = 128, kChkN = 8;
__device__ __forceinline__ float chk_pow2(int e) {  // 2^e of e <= 0, not below 2^-63
  return __int_as_float((max(e, -63) + 127) << 23);
}
__global__ void __launch_bounds__(kChkRows) k_wide_check(const VecInst V, const WideCheck K,
                                                         int mode) {
  constexpr int kSeg = 16;  // blocks of the vectors' exponents at a time
  const int64_t i = (int64_t)blockIdx.x * kChkRows + threadIdx.x;
  const int g0 = blockIdx.y * kChkN;
  const bool on = i < K.m;
  __shared__ float sb[kSeg][kChkN];
  __shared__ int smax[kChkN];
  if (threadIdx.x < kChkN) {
    int mx = kOzNone;
    if (g0 + threadIdx.x < V.nrhs)
      for (int b = 0; b < K.kb; ++b) mx = max(mx, K.bexp[b * K.bs + g0 + threadIdx.x]);
    smax[threadIdx.x] = mx;
  }
  int amax = kOzNone;
  if (on)
    for (int b = 0; b < K.kb; ++b) amax = max(amax, K.aexp[b * K.as + i]);
  float sum[kChkN];
#pragma unroll
  for (int g = 0; g < kChkN; ++g) sum[g] = 0.f;
  for (int b0 = 0; b0 < K.kb; b0 += kSeg) {
    __syncthreads();
    for (int e = threadIdx.x; e < kSeg * kChkN; e += kChkRows) {
      const int b = b0 + e / kChkN, g = e % kChkN;
      const bool some = b < K.kb && g0 + g < V.nrhs && smax[g] != kOzNaN;
      sb[e / kChkN][g] = some ? chk_pow2(K.bexp[b * K.bs + g0 + g] - smax[g]) : 0.f;
    }
    __syncthreads();
    if (on && amax != kOzNaN)
      for (int b = b0; b < min(K.kb, b0 + kSeg); ++b) {
        const float fa = chk_pow2(K.aexp[b * K.as + i] - amax);
#pragma unroll
        for (int g = 0; g < kChkN; ++g) sum[g] = fmaf(fa, sb[b - b0][g], sum[g]);
      }
  }
  if (!on || amax == kOzNaN) return;
#pragma unroll
  for (int g = 0; g < kChkN; ++g) {
    if (g0 + g >= V.nrhs || smax[g] == kOzNaN) continue;
    const double den = V.den[K.r0 + i + (int64_t)(g0 + g) * V.ldy];
    if (isfinite(den) && scalbn((double)sum[g], amax + smax[g]) > wide_spread(V, mode) * den) {
      const int at = atomicAdd(K.count, 1);
      if (at < K.cap) K.list[at] = make_int2((int)(K.r0 + i), g0 + g);
    }
  }
}

void launch_wide_check(const Launch& L, const VecInst& v, const WideCheck& k, int mode) {
  k_wide_check<<<dim3((unsigned)((k.m + kChkRows - 1) / kChkRows),
                      (unsigned)((v.nrhs + kChkN - 1) / kChkN)),
                 kChkRows, 0, L.stream>>>(v, k, mode);
  count_launch(1);
}

// The listed entries of y in FP64, one warp each.  The list's order varies, its entries do not
// depend on one another.
template <bool A32>
__global__ void __launch_bounds__(256) k_wide_redo(const VecInst V, const WideCheck K, int mode) {
  const int count = *K.count;
  if (count > K.cap) return;  // the row-wise products do them all
  const int lane = threadIdx.x & 31;
  for (int e = blockIdx.x * 8 + (threadIdx.x >> 5); e < count; e += gridDim.x * 8) {
    const int2 at = K.list[e];
    const int64_t i = at.x, n = V.n;
    const double* x = V.x + 2 * (int64_t)at.y * V.ldx;
    cd t = {0.0, 0.0};
    constexpr int kB = 8;
    for (int64_t j0 = lane; j0 < n; j0 += 32 * kB) {
      typename Entry<A32>::T a[kB];
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        const int64_t j = j0 + 32 * q;
        a[q] = j < n ? Entry<A32>::at(V, i + j * V.lda) : typename Entry<A32>::T{};
      }
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        const int64_t j = j0 + 32 * q;
        const cd v = j < n ? ldc(x, j) : cd{0.0, 0.0};
        t.x = fma((double)a[q].x, v.x, fma(-(double)a[q].y, v.y, t.x));
        t.y = fma((double)a[q].x, v.y, fma((double)a[q].y, v.x, t.y));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
      t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
    }
    if (lane == 0) {
      const cd b = mode == 1 ? ldc(V.b, i + (int64_t)at.y * V.ldb) : cd{0.0, 0.0};
      stc(V.y, i + (int64_t)at.y * V.ldy, cd{b.x - t.x, b.y - t.y});
    }
  }
}

void launch_wide_redo(const Launch& L, const VecInst& v, const WideCheck& k, int mode) {
  const unsigned grid =
      (unsigned)std::min<int64_t>((k.cap + 7) / 8, 4 * (int64_t)device_sm_count());
  if (v.a32)
    k_wide_redo<true><<<grid, 256, 0, L.stream>>>(v, k, mode);
  else
    k_wide_redo<false><<<grid, 256, 0, L.stream>>>(v, k, mode);
  count_launch(1);
}

// |x| of every vector in FP32 (ld n)
__global__ void k_wide_mag(const VecInst V, float* __restrict__ xa) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i < V.n) xa[i + (int64_t)r * V.n] = fabs_c(ldc(V.x, i + (int64_t)r * V.ldx));
}

// den = |A||x| (mode 1: + |b|) in FP32 magnitudes (as the row-wise products): 64 x 96 tiles, 4 x 6
// entries per thread, K-chunks of 16 with the next chunk in registers as it was loaded (a
// magnitude taken at the load would wait for it).  FP32-issue bound, one FMA per matrix entry and
// vector, two of them in a paired instruction: 2.1 ms for 20480 unknowns and 181 vectors at the
// single rate, 11 ms before the pairs, the late magnitudes and the odd row stride of sX, 5.3 ms
// with them.  FP32 sums of kWaFold columns are added in FP64 (the row-wise products': n / 8 to n
// / 32 columns).
constexpr int kWaM = 64, kWaN = 96, kWaK = 16, kWaFold = 2048;
template <bool A32>
__global__ void __launch_bounds__(256) k_wide_abs(const VecInst V, const float* __restrict__ xa,
                                                  int mode) {
  using E = Entry<A32>;
  const int64_t r0 = (int64_t)blockIdx.x * kWaM, n = V.n;
  const int g0 = blockIdx.y * kWaN;
  __shared__ alignas(16) float sA[kWaK][kWaM];
  __shared__ alignas(16) float sX[kWaK][kWaN + 2];  // 2 more: the 16 columns of a store apart
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  constexpr int kA = kWaM * kWaK / 256, kX = kWaN * kWaK / 256;
  typename E::T na[kA];
  float nx[kX];
  float2 acc[4][3];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) acc[a][b] = make_float2(0.f, 0.f);
  auto load = [&](int64_t k) {
#pragma unroll
    for (int e = 0; e < kA; ++e) {
      const int t = tid + 256 * e;
      const int64_t r = r0 + t % kWaM, c = k + t / kWaM;
      na[e] = r < n && c < n ? E::at(V, r + c * V.lda) : typename E::T{};
    }
#pragma unroll
    for (int e = 0; e < kX; ++e) {
      const int t = tid + 256 * e;
      const int64_t c = k + t % kWaK;
      const int g = g0 + t / kWaK;
      nx[e] = g < V.nrhs && c < n ? xa[c + (int64_t)g * n] : 0.f;
    }
  };
  // the sums so far into den, the first time with |b|
  auto fold = [&](bool first) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 6; ++b) {
        const int64_t r = r0 + tx * 4 + a;
        const int g = g0 + ty * 6 + b;
        if (r < n && g < V.nrhs) {
          double* at = V.den + r + (int64_t)g * V.ldy;
          const double old =
              !first ? *at : mode == 1 ? cabs(ldc(V.b, r + (int64_t)g * V.ldb)) : 0.0;
          *at = old + (double)(b & 1 ? acc[a][b / 2].y : acc[a][b / 2].x);
        }
      }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) acc[a][b] = make_float2(0.f, 0.f);
  };
  load(0);
  for (int64_t k = 0; k < n; k += kWaK) {
    if (k > 0 && k % kWaFold == 0) fold(k == kWaFold);
#pragma unroll
    for (int e = 0; e < kA; ++e)
      sA[(tid + 256 * e) / kWaM][(tid + 256 * e) % kWaM] = E::mag(na[e]);
#pragma unroll
    for (int e = 0; e < kX; ++e) sX[(tid + 256 * e) % kWaK][(tid + 256 * e) / kWaK] = nx[e];
    __syncthreads();
    if (k + kWaK < n) load(k + kWaK);
#pragma unroll
    for (int kk = 0; kk < kWaK; ++kk) {
      const float4 av = *reinterpret_cast<const float4*>(&sA[kk][tx * 4]);
      const float2* xp = reinterpret_cast<const float2*>(&sX[kk][ty * 6]);
      const float2 xv[3] = {xp[0], xp[1], xp[2]};
      const float ar[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
          acc[a][b] = __ffma2_rn(make_float2(ar[a], ar[a]), xv[b], acc[a][b]);
    }
    __syncthreads();
  }
  fold(n <= kWaFold);
}

void launch_wide_abs(const Launch& L, const VecInst& v, float* xa, int mode) {
  k_wide_mag<<<dim3((unsigned)((v.n + 255) / 256), (unsigned)v.nrhs), 256, 0, L.stream>>>(v, xa);
  const dim3 g((unsigned)((v.n + kWaM - 1) / kWaM), (unsigned)((v.nrhs + kWaN - 1) / kWaN));
  if (v.a32)
    k_wide_abs<true><<<g, 256, 0, L.stream>>>(v, xa, mode);
  else
    k_wide_abs<false><<<g, 256, 0, L.stream>>>(v, xa, mode);
  count_launch(2);
}

__global__ void k_wide_finish(const VecInst V, int mode) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int r = blockIdx.y, s = threadIdx.x & 7;
  const bool on = i < V.n;
  cd t = {0.0, 0.0};
  if (on && V.a32) near_product(V, i, r, s, t);
  t.x = row8_sum(t.x);
  t.y = row8_sum(t.y);
  if (!on || s != 0) return;
  const int64_t yo = i + (int64_t)r * V.ldy;
  const cd y = ldc(V.y, yo) - t;
  stc(V.y, yo, mode == 0 ? cd{-y.x, -y.y} : y);
}

void launch_wide_finish(const Launch& L, const VecInst& v, int mode) {
  k_wide_finish<<<dim3((unsigned)((v.n + 31) / 32), (unsigned)v.nrhs), 256, 0, L.stream>>>(v, mode);
  count_launch(1);
}

// Per right-hand side statistics of a residual r (in y), denominators den, solution x,
// rhs b and row scales:  [0] max|r|  [1] max |r|/den (0/0 = 0, r/0 = inf)  [2] max|x|
// [3] max|b|  [4] sum|r|^2  [5] sum|b|^2  [6] sum|r/rows|^2  [7] sum|b/rows|^2
// [8] nonfinite flag.  The hypots make it FP64-bound (about 250 instructions a row), so the
// rows of a right-hand side are shared by stat_split(n) CTAs whose results, left in the products'
// scratch, the second kernel combines in order: 0.6 ms a pass for one system of 8960 unknowns
// with one CTA, 32 us so.
constexpr int kMaxStatSplit = 16;
__host__ __device__ inline int stat_split(int64_t n) {
  return n < 512 ? 1 : n >= 256 * kMaxStatSplit ? kMaxStatSplit : (int)(n / 256);
}
__device__ __forceinline__ bool stat_is_sum(int t) { return t >= 4 && t <= 7; }

__global__ void __launch_bounds__(256) k_resid_stats(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.y];
  const int r = blockIdx.x, split = stat_split(V.n), z = blockIdx.z;
  if (r >= V.nrhs || z >= split) return;
  int64_t j0, j1;
  chunk_range(V.n, z, split, &j0, &j1);
  double v[kStats];
#pragma unroll
  for (int t = 0; t < kStats; ++t) v[t] = 0.0;
  for (int64_t i = j0 + threadIdx.x; i < j1; i += 256) {
    const int64_t o = i + (int64_t)r * V.ldy;
    cd rr = ldc(V.y, o);
    cd bb = ldc(V.b, i + (int64_t)r * V.ldb);
    cd xx = ldc(V.x, i + (int64_t)r * V.ldx);
    double ar = cabs(rr), ab = cabs(bb), ax = cabs(xx);
    double den = V.den ? V.den[o] : 0.0;
    double ratio = (den == 0.0) ? (ar == 0.0 ? 0.0 : INFINITY) : ar / den;
    double rw = V.rows ? V.rows[i] : 1.0;
    v[0] = fmax(v[0], ar);
    v[1] = fmax(v[1], ratio);
    v[2] = fmax(v[2], ax);
    v[3] = fmax(v[3], ab);
    v[4] += ar * ar;
    v[5] += ab * ab;
    v[6] += (ar / rw) * (ar / rw);
    v[7] += (ab / rw) * (ab / rw);
    if (!(isfinite(rr.x) && isfinite(rr.y) && isfinite(den) && isfinite(xx.x) && isfinite(xx.y)))
      v[8] = 1.0;
  }
  __shared__ double sh[kStats][256];
#pragma unroll
  for (int t = 0; t < kStats; ++t) sh[t][threadIdx.x] = v[t];
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
#pragma unroll
      for (int t = 0; t < kStats; ++t) {
        double a = sh[t][threadIdx.x], b = sh[t][threadIdx.x + s];
        sh[t][threadIdx.x] = stat_is_sum(t) ? a + b : fmax(a, b);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < kStats)
    V.part[((int64_t)r * split + z) * kStats + threadIdx.x] = sh[threadIdx.x][0];
}

// ---------------------------------------------------------------- correction steps

__global__ void k_stats_finish(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.y];
  const int r = blockIdx.x, t = threadIdx.x, split = stat_split(V.n);
  if (r >= V.nrhs || t >= kStats) return;
  double v = 0.0;
  for (int z = 0; z < split; ++z) {
    const double a = V.part[((int64_t)r * split + z) * kStats + t];
    v = stat_is_sum(t) ? v + a : fmax(v, a);
  }
  V.stats[(int64_t)r * kStats + t] = v;
}

// The maxima of |v_i / rows_i| over each CTA's rows of the vectors in y (v = b or residual); NaN
// where one isn't finite.  Split as the statistics, for the same reason: 88 us for one system of
// 8960 unknowns with one CTA, 11 us so.
__global__ void __launch_bounds__(256) k_scaled_absmax(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.y];
  const int r = blockIdx.x, split = stat_split(V.n), z = blockIdx.z;
  if (r >= V.nrhs || z >= split) return;
  int64_t j0, j1;
  chunk_range(V.n, z, split, &j0, &j1);
  double m = 0.0;
  bool bad = false;
  for (int64_t i = j0 + threadIdx.x; i < j1; i += 256) {
    cd a = ldc(V.y, i + (int64_t)r * V.ldy);
    double s = V.rows ? V.rows[i] : 1.0;
    double t = hypot(a.x / s, a.y / s);
    if (!isfinite(t)) bad = true;
    m = fmax(m, t);
  }
  __shared__ double sh[256];
  bad = __syncthreads_or(bad);
  sh[threadIdx.x] = m;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) V.part[(int64_t)r * split + z] = bad ? NAN : sh[0];
}

// work (getrs input, complex64 or complex128, ld n) = (v / rows) / mag, mag the largest of
// k_scaled_absmax's maxima
__global__ void k_corr_prep(const VecInst* __restrict__ insts) {
  const VecInst& V = insts[blockIdx.z];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= V.n || r >= V.nrhs) return;
  const int split = stat_split(V.n);
  double mag = 0.0;
  bool bad = false;
  for (int z = 0; z < split; ++z) {
    const double m = V.part[(int64_t)r * split + z];
    bad = bad || isnan(m);
    mag = fmax(mag, m);
  }
  if (bad) mag = NAN;
  if (i == 0) V.stats[(int64_t)r * kStats] = mag;  // for the way back
  cd a = ldc(V.y, i + (int64_t)r * V.ldy);
  double s = V.rows ? V.rows[i] : 1.0;
  cd w = {0.0, 0.0};
  if (mag > 0.0 && isfinite(mag)) w = cd{a.x / s / mag, a.y / s / mag};
  const int64_t o = i + (int64_t)r * V.n;
  if (V.out_single)
    reinterpret_cast<float2*>(V.out)[o] = make_float2((float)w.x, (float)w.y);
  else
    stc(V.out, o, w);
}

// value = work * mag / cols;  mode 0: x = value;  mode 1: x += value (flag if changed)
__global__ void k_corr_apply(const VecInst* __restrict__ insts, int mode) {
  const VecInst& V = insts[blockIdx.z];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= V.n || r >= V.nrhs) return;
  if (V.active && !V.active[r]) return;
  const double mag = V.stats[(int64_t)r * kStats];
  const int64_t o = i + (int64_t)r * V.n;
  cd w;
  if (V.out_single) {
    float2 f = reinterpret_cast<const float2*>(V.out)[o];
    w = {(double)f.x, (double)f.y};
  } else {
    w = ldc(V.out, o);
  }
  const double c = V.cols ? V.cols[i] : 1.0;
  cd val;
  if (!isfinite(mag))
    val = cd{NAN, NAN};
  else if (mag == 0.0)
    val = cd{0.0, 0.0};
  else
    val = cd{w.x * mag / c, w.y * mag / c};
  double* X = const_cast<double*>(V.x);
  const int64_t xo = i + (int64_t)r * V.ldx;
  if (mode == 0) {
    stc(X, xo, val);
  } else {
    cd x = ldc(X, xo);
    cd nx = {x.x + val.x, x.y + val.y};
    if (nx.x != x.x || nx.y != x.y) V.changed[r] = 1;
    stc(X, xo, nx);
  }
}

// ---------------------------------------------------------------- launch wrappers
void launch_equilibrate(const Launch& L, const VecInst* d, int ninst, int64_t nmax) {
  dim3 g1((unsigned)((nmax + 255) / 256), kMaxChunks, (unsigned)ninst);
  k_rowstats<<<g1, 256, 0, L.stream>>>(d); count_launch(1);
  k_rowstats_finish<<<dim3((unsigned)((nmax + 255) / 256), (unsigned)ninst), 256, 0, L.stream>>>(d); count_launch(1);
  k_colmax<<<dim3((unsigned)((nmax + 7) / 8), (unsigned)ninst), 256, 0, L.stream>>>(d); count_launch(1);
}

void launch_scale_copy(const Launch& L, const VecInst* d, int ninst, int64_t nmax) {
  k_cols_inv<<<dim3((unsigned)((nmax + 255) / 256), (unsigned)ninst), 256, 0, L.stream>>>(d);
  count_launch(1);
  dim3 g1((unsigned)((nmax + 255) / 256), kMaxChunks, (unsigned)ninst);
  k_scale_copy<<<g1, 256, 0, L.stream>>>(d); count_launch(1);
  k_norms_finish<<<ninst, kNormT, 0, L.stream>>>(d); count_launch(1);
}

void launch_gemv(const Launch& L, const VecInst* d, int ninst, int64_t nmax, int32_t max_rhs,
                 int mode, int rows) {
  // compact and complex128 instances by their own instantiations (each skips the others);
  // one right-hand side gets a single-rhs instantiation
  const int nr = max_rhs == 1 ? 1 : kGemvR;
  const int groups = (max_rhs + nr - 1) / nr;
  dim3 g0((unsigned)((nmax + 255) / 256), (unsigned)max_rhs, (unsigned)ninst);
  k_split_x<<<g0, 256, 0, L.stream>>>(d); count_launch(1);
  // chunks and groups share the grid's second dimension: as many groups per launch as it holds
  constexpr int kMaxGroups = 65535 / kMaxChunks;
  for (int q0 = 0; q0 < groups; q0 += kMaxGroups) {
    const int q = std::min(kMaxGroups, groups - q0);
    const dim3 g1((unsigned)((nmax + 255) / 256), (unsigned)(kMaxChunks * q), (unsigned)ninst);
    if (nr == 1) {
      if (mode == 1)
        gemv_a32<1, true>(L, d, ninst, nmax, q0, q, rows);
      else
        gemv_a32<1, false>(L, d, ninst, nmax, q0, q, rows);
      k_gemv_part<1><<<g1, 256, 0, L.stream>>>(d, q0, mode == 1);
    } else {
      if (mode == 1)
        gemv_a32<kGemvR, true>(L, d, ninst, nmax, q0, q, rows);
      else
        gemv_a32<kGemvR, false>(L, d, ninst, nmax, q0, q, rows);
      k_gemv_part<kGemvR><<<g1, 256, 0, L.stream>>>(d, q0, mode == 1);
    }
    count_launch(2);
  }
  dim3 g2((unsigned)((nmax + 31) / 32), (unsigned)max_rhs, (unsigned)ninst);
  k_gemv_finish<<<g2, 256, 0, L.stream>>>(d, mode); count_launch(1);
}

void launch_near_add(const Launch& L, const VecInst* d, int ninst, int64_t max_near,
                     int unit_scales) {
  if (max_near <= 0 || ninst <= 0) return;
  k_near_add<<<dim3((unsigned)((max_near + 255) / 256), 4, (unsigned)ninst), 256, 0, L.stream>>>(
      d, unit_scales);
  count_launch(1);
}

void launch_expand_a32(const Launch& L, const VecInst* d, int ninst, int64_t nmax) {
  if (nmax <= 0 || ninst <= 0) return;
  k_expand_a32<<<dim3((unsigned)((nmax + 255) / 256), 256, (unsigned)ninst), 256, 0, L.stream>>>(d);
  count_launch(1);
}

void launch_resid_stats(const Launch& L, const VecInst* d, int ninst, int32_t max_rhs) {
  k_resid_stats<<<dim3((unsigned)max_rhs, (unsigned)ninst, kMaxStatSplit), 256, 0, L.stream>>>(d);
  k_stats_finish<<<dim3((unsigned)max_rhs, (unsigned)ninst), 32, 0, L.stream>>>(d);
  count_launch(2);
}

void launch_corr_prep(const Launch& L, const VecInst* d, int ninst, int64_t nmax,
                      int32_t max_rhs) {
  k_scaled_absmax<<<dim3((unsigned)max_rhs, (unsigned)ninst, kMaxStatSplit), 256, 0, L.stream>>>(
      d); count_launch(1);
  k_corr_prep<<<dim3((unsigned)((nmax + 255) / 256), (unsigned)max_rhs, (unsigned)ninst), 256, 0,
                L.stream>>>(d); count_launch(1);
}

void launch_corr_apply(const Launch& L, const VecInst* d, int ninst, int64_t nmax,
                       int32_t max_rhs, int mode) {
  k_corr_apply<<<dim3((unsigned)((nmax + 255) / 256), (unsigned)max_rhs, (unsigned)ninst), 256, 0,
                 L.stream>>>(d, mode); count_launch(1);
}

}  // namespace bemgpu
