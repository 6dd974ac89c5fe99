// Shared constants and launch declarations of the dense linear-algebra kernels.
#pragma once

#include "bemgpu_internal.h"
#include "quad_math.cuh"

namespace bemgpu {

constexpr int kPanelNB = 32;  // LU panel width (columns factored per getf2 launch)

// Factors the panel [k0, k0 + nb) of every instance; nmax: largest order, nact: instances
// with rows left (the launch shape; the factor does not depend on it).  Returns whether the
// interchanges were applied to the panel's own columns (if not, they are the caller's).
// shape: a launch shape other than the one chosen by size (bemgpu_debug_panel).
struct PanelShape {
  int cluster = 0;         // CTAs per instance, a power of two up to 16 (0: by size)
  bool streaming = false;  // the kernel that keeps the panel in global memory
};
bool launch_getf2(const Launch& L, const MatInst* d, int ninst, int nact, int64_t nmax, int64_t k0,
                  int nb, int prec, const PanelShape& shape = {});
// row interchanges k0 .. k0 + nb - 1 on columns [c_lo, c_hi) \ [s_lo, s_hi)
void launch_laswp(const Launch& L, const MatInst* d, int ninst, int64_t k0, int nb, int64_t c_lo,
                  int64_t c_hi, int64_t s_lo, int64_t s_hi, int prec);
// U12 = L11^{-1} A12 of the panel at k0 on columns [c_lo, c_hi)
void launch_trsm_panel(const Launch& L, const MatInst* d, int ninst, int64_t k0, int64_t c_lo,
                       int64_t c_hi, int prec);
// rows [k0 + nb, n) x columns [c_lo, c_hi) -= L21 U12 (SIMT)
void launch_gemm_update(const Launch& L, const MatInst* d, int ninst, int64_t k0, int nb,
                        int64_t nmax, int64_t c_lo, int64_t c_hi, int prec);
// Triangular solves (trsv.cu).  Bytes of the inverted diagonal blocks of a factor
// (MatInst.dinv), and their computation.
size_t tri_inv_bytes(int64_t n, int prec);
void launch_tri_inv(const Launch& L, const MatInst* d, int ninst, int64_t nmax, int prec);
// Solves with the factor in place on MatInst.x; MatInst.y is a second buffer.  trans 0:
// A x = b, swaps 0 leaving out the row interchanges (MatInst.perm otherwise); trans 1:
// (LU)^H x = b, without interchanges.  The instances of one launch agree on many =
// many_rhs(nrhs), which selects the path by each system's own right-hand sides.
bool many_rhs(int32_t nrhs);
void launch_getrs(const Launch& L, const MatInst* d, int ninst, int64_t nmax, int32_t max_rhs,
                  int trans, int prec, int swaps, bool many);
// out[i] (kLinvB x kLinvB complex64, column-major) = -(L11^{-1} - I) of the unit lower
// block at (k0, k0) of instance i (complex64 factors).
void launch_linv_neg(const Launch& L, const MatInst* d, int ninst, int64_t k0, float2* const* outs);
// The same for complex128 factors.
void launch_linv_neg_c128(const Launch& L, const MatInst* d, int ninst, int64_t k0,
                          double2* const* outs);
// Row permutation of each factor from its pivots.
void launch_make_perm(const Launch& L, const MatInst* d, int ninst, int64_t nmax);

}  // namespace bemgpu
