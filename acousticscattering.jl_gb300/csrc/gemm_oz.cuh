// Descriptors and launch declarations of the complex128 tensor-core update (gemm_oz.cu).
#pragma once

#include "bemgpu_internal.h"

namespace bemgpu {

constexpr int kOzK = 128;        // largest K of one update (exact accumulation, gemm_oz.cu)
constexpr int kOzMaxInst = 256;  // instances per GEMM launch (more are split by the wrapper)

// One operand panel to cut into digit slices.
struct OzPackInst {
  const void* a;   // complex128 column-major matrix
  int64_t lda;
  int64_t r0;      // first operand row (side A: matrix row; side B: matrix column)
  int64_t k0;      // first K index (side A: matrix column; side B: matrix row)
  int64_t rows;    // operand rows (M or N extent); 0: nothing to do
  int32_t kk;      // K extent, at most kOzK
  int32_t pad;
  void* out;       // slice images, oz_pack_bytes(rows, kk, side)
  int32_t* exps;   // exponent of every operand row (oz_exps(rows, side) values)
};

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
  int32_t pad;
};

enum OzSide { kOzA = 0, kOzB = 1 };
size_t oz_pack_bytes(int64_t rows, int kk, OzSide side);
size_t oz_exps(int64_t rows, OzSide side);
int64_t oz_tiles(int64_t m, int64_t n);  // tiles of one update

#ifdef __CUDACC__
// side A: element (r, k) at r + k lda; side B: at k + r lda
void launch_oz_pack(const Launch& L, const OzPackInst* d, int ninst, int64_t max_rows,
                    OzSide side);
// tiles[i]: oz_tiles of instance i (host array), for the grid of each launch
void launch_oz_gemm(const Launch& L, const OzGemmInst* d, int ninst, const int64_t* tiles);
#endif

}  // namespace bemgpu
