// Descriptors and launch declarations of the complex128 tensor-core update (gemm_oz.cu).
#pragma once

#include "bemgpu_internal.h"

namespace bemgpu {

constexpr int kOzK = 128;        // K of one exact accumulation (gemm_oz.cu); longer K in blocks
constexpr int kOzMaxInst = 256;  // instances per GEMM launch (more are split by the wrapper)

// One operand panel to cut into digit slices.
struct OzPackInst {
  const void* a;   // complex128 column-major matrix
  int64_t lda;
  int64_t r0;      // first operand row (side A: matrix row; side B: matrix column)
  int64_t k0;      // first K index (side A: matrix column; side B: matrix row)
  int64_t rows;    // operand rows (M or N extent); 0: nothing to do
  int32_t kk;      // K extent
  int32_t single;  // 1: complex64 matrix
  void* out;       // slice images, oz_pack_bytes(rows, kk, side)
  int32_t* exps;   // exponent of every operand row and block of kOzK columns, block by block:
                   // oz_exps(rows, side) values each
  int32_t* kexp;   // or null: an exponent field (of FP64, 1..2046) per K index, by which side A is
                   // multiplied and side B divided (relative to 1023, the field of one); 0: side
                   // A takes the column as zeros
};
// Stored exponents of a row with a NaN or an infinity, and of one without nonzero entries.
constexpr int32_t kOzNaN = INT32_MAX, kOzNone = -101021;

// One C -= A B update: C block rows [c_r0, c_r0 + m), columns [c_c0, c_c0 + n).
struct OzGemmInst {
  const void* apack;
  const void* bpack;
  const int32_t* aexp;
  const int32_t* bexp;
  void* c;         // complex128 column-major
  int64_t ldc;
  int64_t c_r0, c_c0;
  int64_t m, n;    // 0: nothing to do
  int32_t kk;
  int32_t n_first;  // 1: neighbouring CTAs take neighbouring columns (A larger than L2)
  const int32_t* gate;  // or null: nothing to do when *gate > gate_cap (one instance per launch)
  int32_t gate_cap;
};

enum OzSide { kOzA = 0, kOzB = 1 };
size_t oz_pack_bytes(int64_t rows, int kk, OzSide side);
size_t oz_exps(int64_t rows, OzSide side);
int64_t oz_tiles(int64_t m, int64_t n);  // tiles of one update

#ifdef __CUDACC__
// kexp of side B: kexp[k] = max(kexp[k], largest field of the operand's finite entries at k) over
// its rows (zeros before the first call)
void launch_oz_kexp(const Launch& L, const OzPackInst* d, int ninst, int64_t max_rows, int max_kk);
// side A: element (r, k) at r + k lda, single: the complex64 instances (the others are
// skipped); side B: at k + r lda, complex128
void launch_oz_pack(const Launch& L, const OzPackInst* d, int ninst, int64_t max_rows, int max_kk,
                    OzSide side, bool single = false);
// tiles[i]: oz_tiles of instance i (host array), for the grid of each launch
void launch_oz_gemm(const Launch& L, const OzGemmInst* d, int ninst, const int64_t* tiles);
#endif

}  // namespace bemgpu
