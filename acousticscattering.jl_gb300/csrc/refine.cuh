// Descriptors and launch declarations of the matrix-vector kernels in refine.cu.
#pragma once

#include "bemgpu_internal.h"

namespace bemgpu {

// Column chunks of the row-wise sweeps, by the system's own order: a thread takes a row, so
// small systems need more chunks to fill the GPU (1280 unknowns: 24 CTAs with 8 chunks, 76 us
// a residual; 19 us with 32).  Products of many right-hand sides fill it by these, and their
// partial sums are a chunk's worth of memory per right-hand side: 8 chunks.
constexpr int kMaxChunks = 32;
constexpr int kManyChunksRhs = 16;
__host__ __device__ inline int vec_chunks(int64_t n, int32_t nrhs = 1) {
  return nrhs >= kManyChunksRhs || n > 5120 ? 8 : n <= 2560 ? 32 : 16;
}
constexpr int kGemvR = 4;    // right-hand sides per gemv pass
constexpr int kStats = 9;    // residual statistics per right-hand side

struct VecInst {
  const void* A;     // complex128 matrix, column-major
  int64_t n;         // order
  int64_t lda;
  double* rows;      // row scales (n), or null for unit scales
  double* cols;      // column scales (n), or null
  double* rowsum;    // row sums of |A| (n)
  double* cols_inv;  // 1 / cols (n), filled by the scaled-copy launch
  float* rows_inv;   // 1 / rows (n), filled by the row-statistics launch
  double* part;      // scratch: vec_chunks(n, nrhs) * nrhs * n * 3 doubles
  void* out;         // scaled copy / correction work buffer (ld n)
  int32_t out_single;
  int32_t nrhs;
  int32_t* flag;     // nonfinite conversion flag
  const double* x;   // complex128 vectors (n x nrhs, ld ldx)
  int64_t ldx;
  const double* b;   // complex128 right-hand sides
  int64_t ldb;
  double* y;         // complex128 output / input vectors
  int64_t ldy;
  double* den;       // componentwise denominators (n x nrhs, ld ldy)
  double* stats;     // kStats doubles per right-hand side
  int32_t* active;   // per rhs: still refining (null = all)
  int32_t* changed;  // per rhs: last correction changed x
  // Compact system storage (mixed precision with FP32 regular pairs): A is complex64,
  // exact for every regular pair, and the near pairs carry an FP64 correction
  // dnear = a64 - (complex128)(complex64)a64, so A64 = A + the sparse corrections.
  int32_t a32;
  int32_t nbc;               // block columns of the near pattern: 1 (n x n) or 2 (2n x 2n)
  int64_t n_mesh, n_near;
  const int32_t* near_ptr;   // CSR row pointers over the mesh's near pairs (n_mesh + 1)
  const int32_t* near_i;
  const int32_t* near_j;
  const double* dnear;       // corrections, complex128 [block][n_near], block = nbc br + bc
  float4* xs;                // x split as FP32, every part twice: (hi.re, hi.im), (lo.re, lo.im)
  float* xa;                 // |x| in FP32, n x nrhs
  float* cols_inv32;         // 1 / cols in FP32 (n)
  double norm_floor;         // equilibration: lower bound of the row and column scales
  const int32_t* gate;       // or null: the row-wise products do nothing unless *gate > gate_cap
  int32_t gate_cap;
};

#ifdef __CUDACC__
void launch_equilibrate(const Launch& L, const VecInst* d, int ninst, int64_t nmax);
void launch_scale_copy(const Launch& L, const VecInst* d, int ninst, int64_t nmax);
// mode 0: y = A x; mode 1: y = b - A x and den = |b| + |A||x|.  rows: CTAs of 128 (1) or
// 256 (2) rows in the compact-storage product (results identical)
void launch_gemv(const Launch& L, const VecInst* d, int ninst, int64_t nmax, int32_t max_rhs,
                 int mode, int rows = 2);
// Products of one system with many vectors (api.cu:wide_product).  scale: kexp[j] = largest
// exponent field of x_j over the vectors (n values); abs: den = |A||x| (mode 1: + |b|), xa: n x
// nrhs scratch; check: entries whose digit product may be off by more than its share of den, at
// most cap of them listed; redo: those entries in FP64; finish: the end of a product whose sum
// the tensor-core kernel left in y (mode 0: y = -A x without the near corrections, mode 1:
// y = b - A x without them).
constexpr int kWideRhs = 16;  // right-hand sides of a system from which they are used
struct WideCheck {
  const int32_t* aexp;  // exponents of rows [r0, r0 + m) of A and of the vectors, kb blocks
  const int32_t* bexp;
  int64_t r0, m;
  int64_t as, bs;       // entries of a block of aexp, bexp
  int32_t kb, cap;
  int32_t* count;       // entries found so far (more than cap: the row-wise products take over)
  int2* list;           // (row, vector)
};
void launch_wide_scale(const Launch& L, const VecInst& v, int32_t* kexp);
void launch_wide_abs(const Launch& L, const VecInst& v, float* xa, int mode);
void launch_wide_check(const Launch& L, const VecInst& v, const WideCheck& k, int mode);
void launch_wide_redo(const Launch& L, const VecInst& v, const WideCheck& k, int mode);
void launch_wide_finish(const Launch& L, const VecInst& v, int mode);
// compact instances: out (complex128, ld n) += the near corrections, each scaled by
// 1 / (rows_i cols_j) (unit_scales = 0) or unscaled (unit_scales = 1)
void launch_near_add(const Launch& L, const VecInst* d, int ninst, int64_t max_near,
                     int unit_scales);
// compact instances: out (complex128, ld n) = complex128(A)
void launch_expand_a32(const Launch& L, const VecInst* d, int ninst, int64_t nmax);
void launch_resid_stats(const Launch& L, const VecInst* d, int ninst, int32_t max_rhs);
void launch_corr_prep(const Launch& L, const VecInst* d, int ninst, int64_t nmax,
                      int32_t max_rhs);
void launch_corr_apply(const Launch& L, const VecInst* d, int ninst, int64_t nmax,
                       int32_t max_rhs, int mode);
#endif

}  // namespace bemgpu
