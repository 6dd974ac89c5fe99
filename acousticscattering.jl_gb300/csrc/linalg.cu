// Batched dense complex linear algebra for the BEM systems (complex128 and complex64).
//
// Every kernel takes a device array of MatInst descriptors and handles all instances
// of a batch in one launch (blockIdx.z or blockIdx.y selects the instance); instances
// whose order is exhausted at the current step return at once, so batches of uneven
// size share one launch sequence.
//
// LU: right-looking blocked partial pivoting (LAPACK zgetrf semantics: pivot = first
// row of largest |re| + |im| in the column, P A = L U with unit lower L):
//   getf2   panel of kPanelNB columns, one thread-block cluster per instance;
//   laswp   the panel's row interchanges applied to the columns outside it;
//   trsm    U12 = L11^{-1} A12, one warp per column of A12;
//   gemm    A22 -= L21 U12 (SIMT tile kernel; the complex64 factor of the mixed path
//           uses the tensor-core kernel in gemm_tc.cu instead).
// The triangular solves are in trsv.cu.
#include <cfloat>
#include <climits>
#include <cstdio>

#include "bemgpu_internal.h"
#include <algorithm>

#include "linalg.cuh"

namespace bemgpu {

// ------------------------------------------------------------------ helpers
template <typename R>
__device__ __forceinline__ cx<R> ld(const void* base, int64_t idx) {
  if constexpr (sizeof(R) == 8) {
    double2 v = reinterpret_cast<const double2*>(base)[idx];
    return {v.x, v.y};
  } else {
    float2 v = reinterpret_cast<const float2*>(base)[idx];
    return {v.x, v.y};
  }
}
template <typename R>
__device__ __forceinline__ void st(void* base, int64_t idx, cx<R> v) {
  if constexpr (sizeof(R) == 8)
    reinterpret_cast<double2*>(base)[idx] = make_double2(v.x, v.y);
  else
    reinterpret_cast<float2*>(base)[idx] = make_float2(v.x, v.y);
}
template <typename R>
__device__ __forceinline__ R cabs1(cx<R> a) {
  return fabs(a.x) + fabs(a.y);
}
template <typename R>
__device__ __forceinline__ cx<R> cinv(cx<R> a) {
  R s = fmax(fabs(a.x), fabs(a.y));
  R ar = a.x / s, ai = a.y / s;
  R d = (ar * ar + ai * ai) * s;
  return {ar / d, -ai / d};
}
// ------------------------------------------------------------------ getf2, streaming
// The panel factorisation for more rows than k_getf2_reg below holds: the panel stays in global
// memory (L2).  Column c is brought up to date only
// when it is reached (U[0:c, c] by one warp from the finished L11 rows cached in shared
// memory, then a[r, c] -= sum_j L[r, j] u_j for the rows below), and the pivot search is
// fused into that pass, as is the scaling of column c - 1 by its pivot's reciprocal.
// A cluster of CTAs shares an instance's rows (fixed ownership: row k0 + g + t CS T belongs to
// cluster thread g), exchanging the pivot candidates through distributed shared memory.  Two
// cluster barriers per column order the global writes of one CTA before the reads of the other.
// Every entry takes the operations of k_getf2_reg in the same order, so both give the same
// factor.
constexpr int kRegMaxCS = 16;   // CTAs per cluster at most
constexpr int kGetf2T = 1024;
constexpr int kLLBatch = 16;  // L values per row in flight

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// The two halves of the barrier, for work in between.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_smem(const void* p, unsigned rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_peer_f32(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int32_t ld_peer_s32(uint32_t a) {
  int32_t v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
template <typename V>
__device__ __forceinline__ void better32(V& bv, int32_t& bi, V ov, int32_t oi) {
  if (ov > bv || (ov == bv && oi < bi)) {
    bv = ov;
    bi = oi;
  }
}
__device__ __forceinline__ double ld_peer_f64(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
template <typename R>
__device__ __forceinline__ R ld_peer_real(uint32_t a) {
  if constexpr (sizeof(R) == 8)
    return ld_peer_f64(a);
  else
    return ld_peer_f32(a);
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// x -= a b and a b, the one form every panel kernel uses
__device__ __forceinline__ void cfnma(cx<float>& x, cx<float> a, cx<float> b) {
  x.x = __fmaf_rn(a.y, b.y, __fmaf_rn(-a.x, b.x, x.x));
  x.y = __fmaf_rn(-a.y, b.x, __fmaf_rn(-a.x, b.y, x.y));
}
__device__ __forceinline__ void cfnma(cx<double>& x, cx<double> a, cx<double> b) {
  x.x = __fma_rn(a.y, b.y, __fma_rn(-a.x, b.x, x.x));
  x.y = __fma_rn(-a.y, b.x, __fma_rn(-a.x, b.y, x.y));
}
__device__ __forceinline__ cx<float> cmul(cx<float> a, cx<float> b) {
  return {__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x))};
}
__device__ __forceinline__ cx<double> cmul(cx<double> a, cx<double> b) {
  return {__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x))};
}
// reciprocal with one division: scaled by a power of two so that the squares neither
// overflow nor vanish
__device__ __forceinline__ cx<double> cinv_fast(cx<double> a) {
  const int e = (max(__double2hiint(a.x) & 0x7FFFFFFF, __double2hiint(a.y) & 0x7FFFFFFF)) >> 20;
  if (e < 2 || e > 2044) return cinv(a);
  const double sc = __hiloint2double((2046 - e) << 20, 0);
  const double x = a.x * sc, y = a.y * sc;
  const double q = sc / (x * x + y * y);
  return {x * q, -y * q};
}
__device__ __forceinline__ cx<float> cinv_fast(cx<float> a) { return cinv(a); }

template <typename R, int T, int BATCH>
__global__ void __launch_bounds__(T) k_getf2_ll(const MatInst* __restrict__ insts, int64_t k0,
                                                int nb) {
  using C = cx<R>;
  const unsigned rank = cluster_rank(), cs = cluster_size();
  const MatInst& M = insts[blockIdx.x / cs];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;  // the whole cluster (one instance) leaves together
  const int nbe = (int)min((int64_t)nb, n - k0);
  const int64_t lda = M.lda;
  void* A = M.a;
  __shared__ C sL[kPanelNB][kPanelNB + 1];  // finished L11 rows
  __shared__ C su[kPanelNB];                // U[0:c, c]
  __shared__ R w_val[T / 32];
  __shared__ int32_t w_idx[T / 32];         // rows as int32 (orders below 2^31)
  __shared__ R c_val;                       // this CTA's pivot candidate
  __shared__ int32_t c_idx;
  __shared__ C s_inv;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int64_t g = (int64_t)rank * T + tid;
  const int64_t stride = (int64_t)cs * T;
  C inv_prev = {(R)1, (R)0};
  for (int c = 0; c < nbe; ++c) {
    const int64_t col = k0 + c;
    // (1) u = L11[0:c, 0:c]^{-1} a[k0:k0+c, col] (identical in every CTA)
    if (wid == 0) {
      C x = {(R)0, (R)0};
      if (lane < c) x = ld<R>(A, (k0 + lane) + col * lda);
      for (int i = 0; i + 1 < c; ++i) {
        C ui;
        ui.x = __shfl_sync(0xffffffffu, x.x, i);
        ui.y = __shfl_sync(0xffffffffu, x.y, i);
        if (lane > i && lane < c) cfnma(x, sL[lane][i], ui);
      }
      if (lane < c) su[lane] = x;  // stored after the first cluster barrier (peers read
                                   // the original values of these rows first)
    }
    __syncthreads();
    // (2) rows >= col: finish L[., c - 1], update column c, pivot candidate
    R best = (R)-1;
    int32_t bidx = INT32_MAX;
    int64_t r = k0 + g;
    if (r < col) r += ((col - r + stride - 1) / stride) * stride;
    for (; r < n; r += stride) {
      C acc = ld<R>(A, r + col * lda);
      for (int j0 = 0; j0 < c; j0 += BATCH) {
        C lv[BATCH];
#pragma unroll
        for (int e = 0; e < BATCH; ++e) {
          lv[e] = C{(R)0, (R)0};
          if (j0 + e < c) lv[e] = ld<R>(A, r + (k0 + j0 + e) * lda);
        }
#pragma unroll
        for (int e = 0; e < BATCH; ++e) {
          if (j0 + e < c) {
            if (j0 + e == c - 1) {
              lv[e] = cmul(lv[e], inv_prev);
              st<R>(A, r + (k0 + j0 + e) * lda, lv[e]);
            }
            cfnma(acc, lv[e], su[j0 + e]);
          }
        }
      }
      st<R>(A, r + col * lda, acc);
      better32(best, bidx, cabs1(acc), (int32_t)r);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const R ov = __shfl_down_sync(0xffffffffu, best, off);
      const int32_t oi = __shfl_down_sync(0xffffffffu, bidx, off);
      better32(best, bidx, ov, oi);
    }
    if (lane == 0) {
      w_val[wid] = best;
      w_idx[wid] = bidx;
    }
    __syncthreads();
    if (wid == 0) {  // the CTA's candidate: a shuffle tree over the 32 warps' candidates
      R bv = lane < T / 32 ? w_val[lane] : (R)-1;
      int32_t bi = lane < T / 32 ? w_idx[lane] : INT32_MAX;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const R ov = __shfl_xor_sync(0xffffffffu, bv, off);
        const int32_t oi = __shfl_xor_sync(0xffffffffu, bi, off);
        better32(bv, bi, ov, oi);
      }
      if (lane == 0) {
        c_val = bv;
        c_idx = bi;
      }
    }
    // (3) pivot of the cluster: only warp 0 needs it (the U row, the interchange over the
    // panel's <= 32 columns, the singular marker and the pivot's reciprocal are its work)
    cluster_sync_all();
    R pv = (R)-1;
    int32_t piv32 = INT32_MAX;
    if (wid == 0) {  // one lane per CTA of the cluster, all peer loads in flight
      if (lane < (int)cs) {
        if ((unsigned)lane != rank) {
          pv = ld_peer_real<R>(peer_smem(&c_val, (unsigned)lane));
          piv32 = ld_peer_s32(peer_smem(&c_idx, (unsigned)lane));
        } else {
          pv = c_val;
          piv32 = c_idx;
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {  // every lane gets the cluster's pivot
        const R ov = __shfl_xor_sync(0xffffffffu, pv, off);
        const int32_t oi = __shfl_xor_sync(0xffffffffu, piv32, off);
        better32(pv, piv32, ov, oi);
      }
    }
    int64_t piv = piv32;
    if (piv >= n) piv = col;  // no candidate rows (cannot happen for col < n)
    const bool nonzero = pv > (R)0;
    if (rank == 0) {
      if (tid < c) st<R>(A, (k0 + tid) + col * lda, su[tid]);
      if (tid == 0) {
        M.ipiv[col] = (int32_t)piv;
        if (!nonzero && *M.info == 0) *M.info = (int32_t)(col + 1);
      }
      if (piv != col && tid < nbe) {  // interchange over the panel's columns
        const int64_t cc = k0 + tid;
        const C a = ld<R>(A, col + cc * lda), b = ld<R>(A, piv + cc * lda);
        st<R>(A, col + cc * lda, b);
        st<R>(A, piv + cc * lda, a);
      }
    }
    cluster_sync_all();
    // (4) reciprocal of the pivot; cache the finished row of L11
    if (tid < c) sL[c][tid] = ld<R>(A, col + (k0 + tid) * lda);
    if (tid == 0) s_inv = nonzero ? cinv_fast(ld<R>(A, col + col * lda)) : C{(R)1, (R)0};
    __syncthreads();
    inv_prev = s_inv;
  }
  // scale the last column below its pivot
  const int64_t colL = k0 + nbe - 1;
  int64_t r = k0 + g;
  if (r <= colL) r += ((colL + 1 - r + stride - 1) / stride) * stride;
  for (; r < n; r += stride) st<R>(A, r + colL * lda, cmul(ld<R>(A, r + colL * lda), inv_prev));
}

// ------------------------------------------------------------------ getf2, in registers
// The panel factorisation of both precisions up to kRegRows rows per thread: a cluster of
// CTAs holds the panel's rows in registers, W columns at a time (a sub-panel), and never
// moves them: a row keeps its place and remembers its position under the interchanges
// (implicit pivoting; the launcher's caller applies the interchanges to the panel's columns
// with everybody else's).  Bound by the latency of a column step, so a step has one CTA
// barrier and one cluster barrier: the CTA's candidate (value, position, reciprocal and the
// row's remaining entries) is pushed by its owner's warp into every CTA's shared memory
// before the cluster barrier, after which each CTA picks the winner among the copies it
// holds and updates its rows from registers.  Sub-panels are left-looking: the rows' finished
// L values come back from global memory (L2) and the pivot rows' U values are solved by every
// CTA.  Every entry takes its updates a -= l_j u_j one by one in the order of j with the same
// four FMAs whatever W, the cluster size and the rows per thread, so factors do not depend
// on the batch.  Measured, one instance of 8960 unknowns, complex64: 7.0 us a column with the
// streaming kernel above, see the launcher for this one's; complex128 (FP64 issue: two FMAs
// per clock and SM beside the latency) of 5760 unknowns: 27 us a column before.
__device__ __forceinline__ void st_peer_b32(uint32_t a, uint32_t v) {
  asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// Ordered key of a pivot candidate: |re| + |im| as bits, 0 for a NaN (never a candidate).
struct PivKey {
  uint32_t hi, lo;   // value bits (lo: 0 for complex64)
  int32_t pos;       // position under the interchanges, INT32_MAX: no candidate
  int32_t phys;      // row
};
__device__ __forceinline__ void key_of(cx<float> a, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(cabs1(a));
  lo = 0u;
}
__device__ __forceinline__ void key_of(cx<double> a, uint32_t& hi, uint32_t& lo) {
  const double v = cabs1(a);
  hi = (uint32_t)__double2hiint(v);
  lo = (uint32_t)__double2loint(v);
}
__device__ __forceinline__ bool key_nan(const PivKey& k, float) { return k.hi > 0x7F800000u; }
__device__ __forceinline__ bool key_nan(const PivKey& k, double) {
  return k.hi > 0x7FF00000u || (k.hi == 0x7FF00000u && k.lo != 0u);
}
__device__ __forceinline__ bool key_better(const PivKey& a, const PivKey& b) {
  if (a.pos == INT32_MAX) return false;
  if (b.pos == INT32_MAX) return true;
  if (a.hi != b.hi) return a.hi > b.hi;
  if (a.lo != b.lo) return a.lo > b.lo;
  return a.pos < b.pos;
}
// best candidate of a warp, in every lane; returns the lane that holds it (-1: none)
template <typename R>
__device__ __forceinline__ int warp_best(PivKey& k) {
  const bool cand = k.pos != INT32_MAX;
  const uint32_t any = __ballot_sync(0xffffffffu, cand);
  if (!any) return -1;
  uint32_t h = cand ? k.hi : 0u;
  const uint32_t mh = __reduce_max_sync(0xffffffffu, h);
  bool in = cand && k.hi == mh;
  if (sizeof(R) == 8) {
    const uint32_t ml = __reduce_max_sync(0xffffffffu, in ? k.lo : 0u);
    in = in && k.lo == ml;
    k.lo = ml;
  }
  k.hi = mh;
  const int32_t mp = __reduce_min_sync(0xffffffffu, in ? k.pos : INT32_MAX);
  const int src = __ffs(__ballot_sync(0xffffffffu, in && k.pos == mp)) - 1;
  k.pos = mp;
  k.phys = __shfl_sync(0xffffffffu, k.phys, src);
  return src;
}
__device__ __forceinline__ cx<float> shfl_c(cx<float> v, int src) {
  return {__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}
__device__ __forceinline__ cx<double> shfl_c(cx<double> v, int src) {
  return {__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}
__device__ __forceinline__ void st_peer_c(uint32_t a, cx<float> v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void st_peer_c(uint32_t a, cx<double> v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}

template <typename R, int W>
struct alignas(16) PivSlot {
  PivKey key;
  cx<R> inv;
  cx<R> row[W];
};

// T: threads per CTA at most (complex128 sub-panels of 16 columns need the registers of a
// CTA of 256)
template <typename R, int W, int RPT, int T_>
__global__ void __launch_bounds__(T_) k_getf2_reg(const MatInst* __restrict__ insts, int64_t k0,
                                                     int nb, int share) {
  using C = cx<R>;
  // Columns whose code is unrolled.  All 16 of a sub-panel are 80 KB of instructions that run twice
  // in a launch: a quarter of the cycles waited for them.  Four at a time: 61 to 53 us a panel of
  // a factorisation of 1280 unknowns on average.  With more than two rows per thread the registers
  // that take turns cost more.
  constexpr int kU = RPT > 2 || W <= 4 ? W : 4;
  const unsigned rank = cluster_rank(), cs = cluster_size();
  const MatInst& M = insts[blockIdx.x / cs];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;  // the whole cluster (one instance) leaves together
  // a CTA's shared memory exists for its peers once it has started: every CTA says so here and
  // waits for the others before its first store to a peer, with the panel's loads in between
  cluster_arrive();
  const int nbe = (int)min((int64_t)nb, n - k0);
  const int64_t lda = M.lda;
  void* A = M.a;
  __shared__ PivSlot<R, W> slot[2][kRegMaxCS];
  __shared__ PivKey s_key[T_ / 32];
  __shared__ C sL[kPanelNB][kPanelNB + 1];  // L rows of the pivots of finished sub-panels
  __shared__ C sU[W][kPanelNB];             // U rows of this sub-panel's columns
  __shared__ int32_t s_phys[kPanelNB];      // row of every pivot
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int T = blockDim.x, nw = T >> 5;
  // this CTA's rows: share of them from k0 + rank share on, T at a time
  const int64_t stride = T;
  const int64_t g = k0 + (int64_t)rank * share + tid;
  int32_t pos[RPT], fz[RPT];  // position; step at which the row became a pivot (nb: not yet)
#pragma unroll
  for (int t = 0; t < RPT; ++t) {
    pos[t] = (int32_t)(g + t * stride);
    fz[t] = tid + t * T < share && g + t * stride < n ? kPanelNB : -1;  // -1: no row
  }
  for (int s0 = 0; s0 < nbe; s0 += W) {
    const int wn = min(W, nbe - s0);
    C a[RPT][W];
#pragma unroll
    for (int t = 0; t < RPT; ++t)
#pragma unroll
      for (int w = 0; w < W; ++w)
        a[t][w] = fz[t] >= 0 && w < wn ? ld<R>(A, (g + t * stride) + (k0 + s0 + w) * lda) : C{0, 0};
    if (s0 == 0) cluster_wait();  // every peer has started
    if (s0 > 0) {
      // U rows of the finished pivots in these columns
      for (int e = tid; e < s0 * s0; e += T) {
        const int j = e % s0, i = e / s0;
        if (i < j) sL[j][i] = ld<R>(A, s_phys[j] + (k0 + i) * lda);
      }
      for (int w = wid; w < wn; w += nw) {
        if (lane < s0) sU[w][lane] = ld<R>(A, s_phys[lane] + (k0 + s0 + w) * lda);
      }
      __syncthreads();
      for (int w = wid; w < wn; w += nw) {
        C x = lane < s0 ? sU[w][lane] : C{0, 0};
        for (int i = 0; i + 1 < s0; ++i) {
          const C ui = shfl_c(x, i);
          if (lane > i && lane < s0) cfnma(x, sL[lane][i], ui);
        }
        __syncwarp();
        if (lane < s0) sU[w][lane] = x;
      }
      __syncthreads();
      constexpr int kB = sizeof(R) == 4 ? 8 : 4;  // L values in flight (s0 is a multiple)
#pragma unroll
      for (int t = 0; t < RPT; ++t) {
        const int lim = min(fz[t], s0);
        for (int j0 = 0; j0 < lim; j0 += kB) {
          C l[kB];
#pragma unroll
          for (int e = 0; e < kB; ++e)
            if (j0 + e < lim) l[e] = ld<R>(A, (g + t * stride) + (k0 + j0 + e) * lda);
#pragma unroll
          for (int e = 0; e < kB; ++e)
            if (j0 + e < lim) {
#pragma unroll
              for (int w = 0; w < W; ++w)
                if (w < wn) cfnma(a[t][w], l[e], sU[w][j0 + e]);
            }
        }
      }
    }
    // kU columns at a time, after which the columns move up by kU places (back where they were
    // after W of them)
#pragma unroll 1
    for (int w0 = 0; w0 < W; w0 += kU) {
#pragma unroll
      for (int w = 0; w < kU; ++w) {
        if (w0 + w >= wn) break;  // uniform over the cluster
        const int c = s0 + w0 + w;
        const int32_t col = (int32_t)(k0 + c);
        PivSlot<R, W>* sl = slot[c & 1];
        // this thread's, the warp's and the CTA's candidate
        PivKey best = {0u, 0u, INT32_MAX, 0};
#pragma unroll
        for (int t = 0; t < RPT; ++t) {
          PivKey k;
          key_of(a[t][w], k.hi, k.lo);
          k.pos = fz[t] == kPanelNB ? pos[t] : INT32_MAX;
          k.phys = (int32_t)(g + t * stride);
          if (!key_nan(k, R{}) && key_better(k, best)) best = k;
        }
        warp_best<R>(best);
        if (lane == 0) s_key[wid] = best;
        __syncthreads();
        best = lane < nw ? s_key[lane] : PivKey{0u, 0u, INT32_MAX, 0};
        const int bw = warp_best<R>(best);  // warp of the CTA's candidate
        // its owner's warp pushes it to every CTA, lane i to CTA i
        if (wid == max(bw, 0)) {
          int own = -1;  // this thread's row that is the candidate
#pragma unroll
          for (int t = 0; t < RPT; ++t)
            if (bw >= 0 && fz[t] == kPanelNB && pos[t] == best.pos) own = t;
          const uint32_t who = __ballot_sync(0xffffffffu, own >= 0);
          const int src = who ? __ffs(who) - 1 : 0;
          const uint32_t dst = peer_smem(&sl[rank], (unsigned)min(lane, (int)cs - 1));
          const bool send = lane < (int)cs;
          if (send) {
            st_peer_b32(dst, best.hi);
            st_peer_b32(dst + 4, best.lo);
            st_peer_b32(dst + 8, (uint32_t)best.pos);
            st_peer_b32(dst + 12, (uint32_t)best.phys);
          }
#pragma unroll
          for (int q = w; q < W; ++q) {
            if (q / kU * kU >= wn - w0) break;  // columns that are left, rounded up to kU
            C v = a[0][q];
#pragma unroll
            for (int t = 1; t < RPT; ++t)
              if (own == t) v = a[t][q];
            v = shfl_c(v, src);
            if (q == w) v = (best.hi | best.lo) != 0u && bw >= 0 ? cinv_fast(v) : C{(R)1, (R)0};
            if (send) st_peer_c(dst + 16 + (q == w ? 0 : 1 + q) * (uint32_t)sizeof(C), v);
          }
        }
        cluster_sync_all();
        // the cluster's pivot; the slots of step c are free again after the barrier of c + 1
        best = lane < (int)cs ? sl[lane].key : PivKey{0u, 0u, INT32_MAX, 0};
        const int win = max(warp_best<R>(best), 0);
        // no candidate (only NaNs): the row at the diagonal position, marked singular
        const int32_t piv = best.pos == INT32_MAX ? col : best.pos;
        const bool nonzero = best.pos != INT32_MAX && (best.hi | best.lo) != 0u;
        const C inv = sl[win].inv;
        if (rank == 0 && tid == 0) {
          M.ipiv[col] = piv;
          if (!nonzero && *M.info == 0) *M.info = col + 1;
        }
        if (tid == 0) s_phys[c] = best.pos != INT32_MAX ? best.phys : col;
#pragma unroll
        for (int t = 0; t < RPT; ++t) {
          if (fz[t] == kPanelNB) {
            if (pos[t] == piv) {
              fz[t] = c;
              pos[t] = col;
            } else {
              if (pos[t] == col) pos[t] = piv;
              const C l = cmul(a[t][w], inv);
              a[t][w] = l;
#pragma unroll
              for (int q = w + 1; q < W; ++q) {
                if (q / kU * kU >= wn - w0) break;
                cfnma(a[t][q], l, sl[win].row[q]);
              }
            }
          }
        }
      }
      if (W > kU) {
#pragma unroll
        for (int t = 0; t < RPT; ++t) {
          C first[kU];
#pragma unroll
          for (int w = 0; w < kU; ++w) first[w] = a[t][w];
#pragma unroll
          for (int w = 0; w + kU < W; ++w) a[t][w] = a[t][w + kU];
#pragma unroll
          for (int w = 0; w < kU; ++w) a[t][W - kU + w] = first[w];
        }
      }
    }
#pragma unroll
    for (int t = 0; t < RPT; ++t)
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (fz[t] >= 0 && w < wn) st<R>(A, (g + t * stride) + (k0 + s0 + w) * lda, a[t][w]);
    // the stores before the other CTAs' reads of the pivot rows, and no CTA leaves while a
    // peer can still write to its shared memory
    cluster_sync_all();
  }
}

// ------------------------------------------------------------------ laswp
// Interchanges of rows k0 .. k0 + nbe - 1 (LAPACK's sequential order: row k0 + c with
// ipiv[k0 + c] for c = 0, 1, ...) applied to the columns j in [c_lo, min(c_hi, n)) that
// lie outside [s_lo, s_hi).  The sequence is first resolved, once per CTA, into the
// permutation of the rows it touches (destination row <- source row); then one warp per
// column loads every moved element (one per lane and slot, all loads in flight), meets at a
// warp barrier and stores them at their destinations.
constexpr int kSwpMaxNb = 128;   // interchanges per launch
constexpr int kSwpWarps = 8;
constexpr int kSwpHash = 512;    // open-addressing table of touched rows beyond the block

template <typename R>
__global__ void __launch_bounds__(kSwpWarps * 32) k_laswp(const MatInst* __restrict__ insts,
                                                         int64_t k0, int nb, int64_t c_lo,
                                                         int64_t c_hi, int64_t s_lo,
                                                         int64_t s_hi, int cols) {
  const MatInst& M = insts[blockIdx.y];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;
  const int nbe = (int)min((int64_t)nb, n - k0);
  const int64_t skip = s_hi - s_lo;
  auto column = [&](int64_t q) {  // compacted column index -> matrix column (or -1)
    int64_t j = c_lo + q;
    if (j >= s_lo) j += skip;
    return (j >= n || j >= c_hi) ? (int64_t)-1 : j;
  };
  const int64_t q0 = (int64_t)blockIdx.x * cols;
  if (column(q0) < 0) return;  // uniform per CTA
  __shared__ int32_t piv[kSwpMaxNb];
  __shared__ int32_t pos[2 * kSwpMaxNb], src[2 * kSwpMaxNb];  // slot: row, its source row
  __shared__ int32_t hkey[kSwpHash];
  __shared__ int16_t hslot[kSwpHash];
  __shared__ int32_t mpos[2 * kSwpMaxNb], msrc[2 * kSwpMaxNb];
  __shared__ int nmove;
  const int tid = threadIdx.x;
  for (int c = tid; c < nbe; c += blockDim.x) piv[c] = M.ipiv[k0 + c];
  for (int h = tid; h < kSwpHash; h += blockDim.x) hkey[h] = -1;
  __syncthreads();
  if (tid == 0) {
    int ns = nbe;
    for (int c = 0; c < nbe; ++c) pos[c] = src[c] = (int32_t)(k0 + c);
    for (int c = 0; c < nbe; ++c) {
      const int32_t p = piv[c];
      if (p == (int32_t)(k0 + c)) continue;
      int sp;
      if (p < (int32_t)(k0 + nbe)) {
        sp = p - (int32_t)k0;
      } else {
        int h = (int)(((uint32_t)p * 2654435761u) >> 23) & (kSwpHash - 1);
        while (hkey[h] != -1 && hkey[h] != p) h = (h + 1) & (kSwpHash - 1);
        if (hkey[h] == -1) {
          hkey[h] = p;
          hslot[h] = (int16_t)ns;
          pos[ns] = src[ns] = p;
          ++ns;
        }
        sp = hslot[h];
      }
      const int32_t t = src[c];
      src[c] = src[sp];
      src[sp] = t;
    }
    int nm = 0;
    for (int t = 0; t < ns; ++t)
      if (src[t] != pos[t]) {
        mpos[nm] = pos[t];
        msrc[nm] = src[t];
        ++nm;
      }
    nmove = nm;
  }
  __syncthreads();
  const int nm = nmove;
  if (nm == 0) return;
  const int lane = tid & 31, wid = tid >> 5;
  const int64_t lda = M.lda;
  constexpr int kPer = 2 * kSwpMaxNb / 32;
  for (int q = wid; q < cols; q += kSwpWarps) {
    const int64_t j = column(q0 + q);
    if (j < 0) break;
    cx<R> v[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int t = lane + 32 * u;
      if (t < nm) v[u] = ld<R>(M.a, msrc[t] + j * lda);
    }
    __syncwarp();  // every load of this column is performed before any store
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int t = lane + 32 * u;
      if (t < nm) st<R>(M.a, mpos[t] + j * lda, v[u]);
    }
  }
}

// ------------------------------------------------------------------ trsm (U12)
// U12 = L11^{-1} A12 for the columns [c_lo, min(c_hi, n)); L11 = unit lower nbe x nbe
// block at (k0, k0), staged once per CTA in shared memory; each warp solves per_warp columns
// (column = warp + kTrsmWarps * t), lane r holding row r.  The columns are the at most 96 to the
// right of a 32-column panel inside a 128-column block (all of them without the tensor cores).
// A warp takes per_warp of them, one after the other (32 dependent steps each): few for one
// system, where 16 made one CTA do all the work (8 us a launch, 2 us with two), 16 in a large
// batch, whose CTAs then stage the block once (see the launcher).
constexpr int kTrsmWarps = 8;
template <typename R>
__global__ void __launch_bounds__(kTrsmWarps * 32) k_trsm_panel(const MatInst* __restrict__ insts,
                                                               int64_t k0, int64_t c_lo,
                                                               int64_t c_hi, int per_warp) {
  const MatInst& M = insts[blockIdx.y];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;
  const int nbe = (int)min((int64_t)kPanelNB, n - k0);
  const int64_t lda = M.lda;
  const int64_t c_end = min(c_hi, n);
  const int64_t cta0 = c_lo + (int64_t)blockIdx.x * kTrsmWarps * per_warp;
  if (cta0 >= c_end) return;  // uniform per CTA
  static_assert(kPanelNB == 32, "a lane holds a row");
  __shared__ cx<R> sL[kPanelNB][kPanelNB + 1];
  for (int t = threadIdx.x; t < nbe * nbe; t += blockDim.x) {
    const int r = t % nbe, c = t / nbe;
    sL[r][c] = ld<R>(M.a, (k0 + r) + (k0 + c) * lda);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int tcol = 0; tcol < per_warp; ++tcol) {
    const int64_t j = cta0 + wid + (int64_t)kTrsmWarps * tcol;
    if (j >= c_end) break;
    cx<R> x = lane < nbe ? ld<R>(M.a, (k0 + lane) + j * lda) : cx<R>{0, 0};
    for (int c = 0; c < nbe; ++c) {
      cx<R> xc;
      xc.x = __shfl_sync(0xffffffffu, x.x, c);
      xc.y = __shfl_sync(0xffffffffu, x.y, c);
      if (lane > c && lane < nbe) x -= sL[lane][c] * xc;
    }
    if (lane < nbe) st<R>(M.a, (k0 + lane) + j * lda, x);
  }
}

// ------------------------------------------------------------------ SIMT gemm update
// C(m x m') -= A(m x kk) B(kk x m') with A = L21, B = U12, C = A22 of each instance.
constexpr int kGT = 64;   // tile edge
constexpr int kGK = 8;    // k chunk
constexpr int kGThreads = 256;

// Rows [k0 + nbe, n), columns [c_lo, min(c_hi, n)).
template <typename R>
__global__ void __launch_bounds__(kGThreads) k_gemm_update(const MatInst* __restrict__ insts,
                                                          int64_t k0, int nb, int64_t c_lo,
                                                          int64_t c_hi) {
  const MatInst& M = insts[blockIdx.y];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;
  const int nbe = (int)min((int64_t)nb, n - k0);
  const int64_t s = k0 + nbe;  // first trailing row
  const int64_t m = n - s;
  const int64_t c_end = min(c_hi, n);
  const int64_t w = c_end - c_lo;
  if (m <= 0 || w <= 0) return;
  const int64_t tiles_m = (m + kGT - 1) / kGT, tiles_n = (w + kGT - 1) / kGT;
  const int64_t t = blockIdx.x;
  if (t >= tiles_m * tiles_n) return;
  const int64_t ti = t % tiles_m, tj = t / tiles_m;
  const int64_t r0 = s + ti * kGT, c0 = c_lo + tj * kGT;
  const int64_t lda = M.lda;
  __shared__ cx<R> sA[kGK][kGT + 1];
  __shared__ cx<R> sB[kGK][kGT + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  cx<R> acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = cx<R>{0, 0};
  for (int kc = 0; kc < nbe; kc += kGK) {
    for (int e = threadIdx.x; e < kGK * kGT; e += kGThreads) {
      int rr = e % kGT, kk = e / kGT;
      int64_t gr = r0 + rr, gk = k0 + kc + kk;
      sA[kk][rr] = (gr < n && kc + kk < nbe) ? ld<R>(M.a, gr + gk * lda) : cx<R>{0, 0};
      int kb = e % kGK;
      int cc = e / kGK;
      int64_t gc = c0 + cc, gkb = k0 + kc + kb;
      sB[kb][cc] = (gc < c_end && kc + kb < nbe) ? ld<R>(M.a, gkb + gc * lda) : cx<R>{0, 0};
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kGK; ++kk) {
      cx<R> av[4], bv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) av[a] = sA[kk][tx + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) bv[b] = sB[kk][ty + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] += av[a] * bv[b];
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      int64_t gr = r0 + tx + 16 * a, gc = c0 + ty + 16 * b;
      if (gr < n && gc < c_end) {
        int64_t idx = gr + gc * lda;
        st<R>(M.a, idx, ld<R>(M.a, idx) - acc[a][b]);
      }
    }
}

// ------------------------------------------------------------------ -(L11^{-1} - I)
// For the tensor-core U12 solve: with L11^{-1} = I + N (N strictly lower),
// U12 = L11^{-1} A12 = A12 - (-N) A12.  Each CTA stages the unit lower block L11 (nbe x nbe at
// (k0, k0)) in shared memory and solves L11 x = e_j for its columns j (one warp per column); out (ld kLinvB, complex64) receives -N.
constexpr int kLinvB = 128;

// gridDim.x CTAs per instance take the columns j = blockIdx.x + gridDim.x i (spread over the
// triangle for balance), a warp one column after the other.  A launch for one instance took 68 us
// with 32 CTAs whose loads waited for one another and takes 23 with 16; each CTA stages the block,
// so a batch uses fewer (linv_ctas).
constexpr int kLinvWarps = 8;
static int linv_ctas(int ninst) {
  int n = 16;
  while (n > 1 && (int64_t)n * ninst > 2 * (int64_t)device_sm_count()) n /= 2;
  return n;
}
__global__ void __launch_bounds__(kLinvWarps * 32) k_linv_neg(
    const MatInst* __restrict__ insts, int64_t k0, float2* const* outs) {
  const MatInst& M = insts[blockIdx.y];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;
  const int nbe = (int)min((int64_t)kLinvB, n - k0);
  const int64_t lda = M.lda;
  extern __shared__ __align__(16) unsigned char linv_smem[];
  cx<float>* sL = reinterpret_cast<cx<float>*>(linv_smem);  // [kLinvB][kLinvB + 1]
  {  // a column per 128 threads, kFly of them in flight
    constexpr int kFly = 16;
    const int r = threadIdx.x % kLinvB, c0 = threadIdx.x / kLinvB, cols = blockDim.x / kLinvB;
    for (int cb = c0; cb < nbe; cb += cols * kFly) {
      cx<float> v[kFly];
#pragma unroll
      for (int e = 0; e < kFly; ++e) {
        const int c = cb + cols * e;
        v[e] = r < nbe && c < r ? ld<float>(M.a, (k0 + r) + (k0 + c) * lda) : cx<float>{0, 0};
      }
#pragma unroll
      for (int e = 0; e < kFly; ++e) {
        const int c = cb + cols * e;
        if (c < r) sL[r * (kLinvB + 1) + c] = v[e];
      }
    }
  }
  __syncthreads();
  float2* out = outs[blockIdx.y];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int kPer = kLinvB / 32;
  for (int j = blockIdx.x + gridDim.x * wid; j < kLinvB; j += gridDim.x * (blockDim.x >> 5)) {
    cx<float> x[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int r = lane + 32 * t;
      x[t] = cx<float>{(r == j && j < nbe) ? 1.f : 0.f, 0.f};
    }
    if (j < nbe) {
#pragma unroll
      for (int t = 0; t < kPer; ++t) {
        for (int cl = 0; cl < 32; ++cl) {
          const int c = 32 * t + cl;
          if (c >= nbe) break;
          if (c < j) continue;
          cx<float> xc;
          xc.x = __shfl_sync(0xffffffffu, x[t].x, cl);
          xc.y = __shfl_sync(0xffffffffu, x[t].y, cl);
#pragma unroll
          for (int u = t; u < kPer; ++u) {
            const int r = lane + 32 * u;
            if (r > c && r < nbe) x[u] -= sL[r * (kLinvB + 1) + c] * xc;
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int r = lane + 32 * t;
      const bool strict = r > j && r < nbe && j < nbe;
      out[r + (int64_t)j * kLinvB] = strict ? make_float2(-x[t].x, -x[t].y) : make_float2(0.f, 0.f);
    }
  }
}

void launch_linv_neg(const Launch& L, const MatInst* d, int ninst, int64_t k0, float2* const* outs) {
  const size_t smem = (size_t)kLinvB * (kLinvB + 1) * sizeof(cx<float>);
  static PerDeviceOnce attr;
  attr.call([&] {
    cudaFuncSetAttribute(k_linv_neg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  const int ctas = linv_ctas(ninst);
  k_linv_neg<<<dim3((unsigned)ctas, (unsigned)ninst), kLinvWarps * 32, smem,
               L.stream>>>(d, k0, outs);
  count_launch(1);
}

// The same for complex128 factors (out: complex128): the strict lower triangle of L11 packed
// by columns in shared memory (127 KB).  Bound by FP64 issue and the 128 dependent steps of a
// column: 95 us with 16 CTAs per instance, against 0.4 ms with one.
__global__ void __launch_bounds__(kLinvWarps * 32) k_linv_neg_c128(
    const MatInst* __restrict__ insts, int64_t k0, double2* const* outs) {
  const MatInst& M = insts[blockIdx.y];
  const int64_t n = M.n;
  if (!M.active || k0 >= n) return;
  const int nbe = (int)min((int64_t)kLinvB, n - k0);
  const int64_t lda = M.lda;
  extern __shared__ __align__(16) unsigned char linv_smem[];
  cx<double>* sL = reinterpret_cast<cx<double>*>(linv_smem);
  // column c: rows c + 1 .. kLinvB - 1 at c (2 kLinvB - c - 1) / 2
  auto at = [](int r, int c) { return c * (2 * kLinvB - c - 1) / 2 + r - c - 1; };
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  {  // a column per 128 threads, kFly of them in flight
    constexpr int kFly = 8;
    const int r = threadIdx.x % kLinvB, c0 = threadIdx.x / kLinvB, cols = blockDim.x / kLinvB;
    for (int cb = c0; cb < nbe; cb += cols * kFly) {
      cx<double> v[kFly];
#pragma unroll
      for (int e = 0; e < kFly; ++e) {
        const int c = cb + cols * e;
        v[e] = r < nbe && c < r ? ld<double>(M.a, (k0 + r) + (k0 + c) * lda) : cx<double>{0, 0};
      }
#pragma unroll
      for (int e = 0; e < kFly; ++e) {
        const int c = cb + cols * e;
        if (r < nbe && c < r) sL[at(r, c)] = v[e];
      }
    }
  }
  __syncthreads();
  constexpr int kPer = kLinvB / 32;
  double2* out = outs[blockIdx.y];
  for (int j = blockIdx.x + gridDim.x * wid; j < kLinvB; j += gridDim.x * warps) {
    cx<double> x[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) x[t] = cx<double>{lane + 32 * t == j ? 1.0 : 0.0, 0.0};
    if (j < nbe) {
#pragma unroll
      for (int t = 0; t < kPer; ++t) {
        for (int cl = 0; cl < 32; ++cl) {
          const int c = 32 * t + cl;
          if (c >= nbe) break;
          if (c < j) continue;
          cx<double> xc;
          xc.x = __shfl_sync(0xffffffffu, x[t].x, cl);
          xc.y = __shfl_sync(0xffffffffu, x[t].y, cl);
#pragma unroll
          for (int u = t; u < kPer; ++u) {
            const int r = lane + 32 * u;
            if (r > c && r < nbe) x[u] -= sL[at(r, c)] * xc;
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int r = lane + 32 * t;
      const bool strict = r > j && r < nbe && j < nbe;
      out[r + (int64_t)j * kLinvB] =
          strict ? make_double2(-x[t].x, -x[t].y) : make_double2(0.0, 0.0);
    }
  }
}

void launch_linv_neg_c128(const Launch& L, const MatInst* d, int ninst, int64_t k0,
                          double2* const* outs) {
  const size_t smem = (size_t)kLinvB * (kLinvB - 1) / 2 * sizeof(cx<double>);
  static PerDeviceOnce attr;
  attr.call([&] {
    cudaFuncSetAttribute(k_linv_neg_c128, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  const int ctas = linv_ctas(ninst);
  k_linv_neg_c128<<<dim3((unsigned)ctas, (unsigned)ninst), kLinvWarps * 32,
                    smem, L.stream>>>(d, k0, outs);
  count_launch(1);
}

// perm from LAPACK pivots (position i holds row perm[i] after the interchanges).  One thread
// carrying out n interchanges waits for shared memory twice in each (52 us for 1280 unknowns,
// 323 us for 8960), so every row follows its own position instead: interchange i concerns it
// only if it stands at i or at ipiv[i], which is tested for kPermGroup interchanges at once
// (25 and 156 us); a group that holds one is gone through in order.
constexpr int kPermGroup = 16, kPermTile = 2048;
__global__ void __launch_bounds__(256) k_make_perm(const MatInst* __restrict__ insts) {
  const MatInst& M = insts[blockIdx.y];
  if (!M.active || !M.perm) return;
  __shared__ alignas(16) int32_t piv[kPermTile];
  const int n = (int)M.n, e = blockIdx.x * 256 + threadIdx.x;
  if ((int)blockIdx.x * 256 >= n) return;
  int pos = e;  // threads past the last row stand where no interchange reaches
  for (int t0 = 0; t0 < n; t0 += kPermTile) {
    __syncthreads();
    for (int i = threadIdx.x; i < kPermTile; i += 256)
      piv[i] = t0 + i < n ? M.ipiv[t0 + i] : t0 + i;
    __syncthreads();
    const int end = min(kPermTile, n - t0);
    for (int g = 0; g < end; g += kPermGroup) {
      const int i0 = t0 + g;
      bool hit = (unsigned)(pos - i0) < (unsigned)kPermGroup;
#pragma unroll
      for (int q = 0; q < kPermGroup; ++q) hit = hit || piv[g + q] == pos;
      if (hit)
        for (int q = 0; q < kPermGroup; ++q) {
          const int p = piv[g + q];
          pos = pos == i0 + q ? p : pos == p ? i0 + q : pos;
        }
    }
  }
  if (e < n) M.perm[pos] = e;
}

// ------------------------------------------------------------------ launch wrappers
static int prec_is_single(int prec) { return prec == 1; }

// complex64: 1024 threads, 16 L values in flight per row; complex128: 512 threads and 8
// (the 64-register budget of 1024 threads would spill the FP64 values)
template <typename R>
struct LLCfg {
  static constexpr int kT = sizeof(R) == 4 ? kGetf2T : kGetf2T / 2;
  static constexpr int kBatch = sizeof(R) == 4 ? kLLBatch : kLLBatch / 2;
};

template <typename K, typename... Args>
static void cluster_launch(const Launch& L, K kernel, int ninst, int cs, int threads,
                           const MatInst* d, int64_t k0, int nb, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ninst * cs));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = L.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, d, k0, nb, args...);
  count_launch(1);
}

template <typename R>
static void getf2_ll_t(const Launch& L, const MatInst* d, int ninst, int64_t k0, int nb, int cs) {
  auto kernel = k_getf2_ll<R, LLCfg<R>::kT, LLCfg<R>::kBatch>;
  static PerDeviceOnce attr;
  attr.call([&] {  // clusters of 16 are beyond the portable size
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  cluster_launch(L, kernel, ninst, cs, LLCfg<R>::kT, d, k0, nb);
}

template <typename R, int W, int RPT, int T = 512>
static void getf2_reg_t(const Launch& L, const MatInst* d, int ninst, int64_t k0, int nb, int cs,
                        int threads, int share) {
  static PerDeviceOnce attr;
  attr.call([] {  // clusters of 16 are beyond the portable size
    cudaFuncSetAttribute(k_getf2_reg<R, W, RPT, T>,
                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  cluster_launch(L, k_getf2_reg<R, W, RPT, T>, ninst, cs, threads, d, k0, nb, share);
}

// The panel kernel's cluster size.  A column step costs about 1.5 us of barriers and exchanges
// plus the CTA's rows: 1.25 ns a row in complex64 (measured: 1.9, 2.2 and 3.2 us a column with
// 160, 560 and 1280 rows per CTA; half as much again when more than 5 rows per thread force
// sub-panels of 4 columns), 17 ns in complex128 (16 updates of 4 FMAs on average, two per
// clock).  A batch takes as many waves as its clusters need, one CTA per SM, and at most 8
// clusters of 16 or 18 of 8 fit the GPU's processing clusters.  64 systems of 10240 unknowns:
// 138 ms of panels with two CTAs each in one wave, 109 with four, see the launcher's choice.
static int panel_cluster(int nact, int64_t rows, bool single) {
  const int sms = device_sm_count();
  int best = 1;
  double best_cost = 1e300;
  for (int cs = 1; cs <= kRegMaxCS; cs *= 2) {
    const int resident = std::max(1, cs == 16 ? sms / 19 : cs == 8 ? sms / 19 * 9 / 4 : sms / cs);
    const double waves = (double)((nact + resident - 1) / resident);
    const double share = (double)((rows + cs - 1) / cs);
    const double row = single ? (share > 5 * 512 ? 1.9e-3 : 1.25e-3) : 17e-3;
    double cost = waves * (1.5 + 0.02 * cs + row * share);
    if (share > (single ? 10 : 5) * 512) cost *= 2.0;  // the streaming kernel
    if (cost < best_cost) {
      best_cost = cost;
      best = cs;
    }
  }
  return best;
}

// Columns in registers: as many as the rows per thread leave room for.  The streaming kernel takes
// one complex64 system beyond 81920 rows, one complex128 system beyond 40960.
bool launch_getf2(const Launch& L, const MatInst* d, int ninst, int nact, int64_t nmax, int64_t k0,
                  int nb, int prec, const PanelShape& shape) {
  const bool single = prec_is_single(prec);
  const int64_t rows = nmax - k0;
  const int cs = shape.cluster > 0 ? shape.cluster : panel_cluster(std::max(1, nact), rows, single);
  const int share = (int)(((rows + cs - 1) / cs + 31) / 32 * 32);  // rows per CTA
  // complex128: at least eight warps, which solve the U rows of a sub-panel's columns
  const int threads =
      std::min(512, std::max(single ? 64 : 256, share));
  const int q = shape.streaming ? INT_MAX : (share + threads - 1) / threads;  // rows per thread
  if (single) {
    if (q <= 1) return getf2_reg_t<float, 16, 1>(L, d, ninst, k0, nb, cs, threads, share), false;
    if (q <= 2) return getf2_reg_t<float, 16, 2>(L, d, ninst, k0, nb, cs, threads, share), false;
    if (q <= 5) return getf2_reg_t<float, 8, 5>(L, d, ninst, k0, nb, cs, threads, share), false;
    if (q <= 10) return getf2_reg_t<float, 4, 10>(L, d, ninst, k0, nb, cs, threads, share), false;
    getf2_ll_t<float>(L, d, ninst, k0, nb, cs);
  } else {
    if (threads <= 256 && q <= 1)
      return getf2_reg_t<double, 16, 1, 256>(L, d, ninst, k0, nb, cs, threads, share), false;
    if (q <= 1) return getf2_reg_t<double, 8, 1>(L, d, ninst, k0, nb, cs, threads, share), false;
    if (q <= 2) return getf2_reg_t<double, 8, 2>(L, d, ninst, k0, nb, cs, threads, share), false;
    if (q <= 5) return getf2_reg_t<double, 4, 5>(L, d, ninst, k0, nb, cs, threads, share), false;
    getf2_ll_t<double>(L, d, ninst, k0, nb, cs);
  }
  return true;
}

void launch_laswp(const Launch& L, const MatInst* d, int ninst, int64_t k0, int nb, int64_t c_lo,
                  int64_t c_hi, int64_t s_lo, int64_t s_hi, int prec) {
  // the excluded block may reach past the last column
  s_lo = std::min(s_lo, c_hi);
  s_hi = std::min(s_hi, c_hi);
  const int64_t cols = (c_hi - c_lo) - (s_hi - s_lo);
  if (cols <= 0) return;
  // columns per CTA: 128, halved down to 16 while the grid has less than two CTAs per SM (each
  // warp moves its columns one after the other, at memory latency: 24 us a launch for 8960
  // columns in 70 CTAs)
  int per = 128;
  while (per > 16 && (cols + per - 1) / per * ninst < 2 * (int64_t)device_sm_count()) per /= 2;
  dim3 grid((unsigned)((cols + per - 1) / per), (unsigned)ninst);
  for (int b0 = 0; b0 < nb; b0 += kSwpMaxNb) {  // sequential chunks of interchanges
    const int nbc = std::min(kSwpMaxNb, nb - b0);
    if (prec_is_single(prec))
      k_laswp<float><<<grid, kSwpWarps * 32, 0, L.stream>>>(d, k0 + b0, nbc, c_lo, c_hi, s_lo,
                                                              s_hi, per);
    else
      k_laswp<double><<<grid, kSwpWarps * 32, 0, L.stream>>>(d, k0 + b0, nbc, c_lo, c_hi, s_lo,
                                                               s_hi, per);
    count_launch(1);
  }
}

template <typename R>
static void trsm_t(const Launch& L, const MatInst* d, int ninst, int64_t k0, int64_t c_lo,
                   int64_t c_hi) {
  // complex128 columns are FP64-bound: one per warp in a small batch
  const int per_warp = ninst >= 32 ? 16 : sizeof(R) == 4 ? 2 : 1;
  const int64_t per = (int64_t)kTrsmWarps * per_warp;
  dim3 grid((unsigned)((c_hi - c_lo + per - 1) / per), (unsigned)ninst);
  k_trsm_panel<R><<<grid, kTrsmWarps * 32, 0, L.stream>>>(d, k0, c_lo, c_hi, per_warp);
  count_launch(1);
}

void launch_trsm_panel(const Launch& L, const MatInst* d, int ninst, int64_t k0, int64_t c_lo,
                       int64_t c_hi, int prec) {
  if (c_hi <= c_lo) return;
  if (prec_is_single(prec))
    trsm_t<float>(L, d, ninst, k0, c_lo, c_hi);
  else
    trsm_t<double>(L, d, ninst, k0, c_lo, c_hi);
}

void launch_gemm_update(const Launch& L, const MatInst* d, int ninst, int64_t k0, int nb,
                        int64_t nmax, int64_t c_lo, int64_t c_hi, int prec) {
  const int64_t m = nmax - k0 - nb;
  const int64_t w = c_hi - c_lo;
  if (m <= 0 || w <= 0) return;
  const int64_t tiles = ((m + kGT - 1) / kGT) * ((w + kGT - 1) / kGT);
  dim3 grid((unsigned)tiles, (unsigned)ninst);
  if (prec_is_single(prec))
    k_gemm_update<float><<<grid, kGThreads, 0, L.stream>>>(d, k0, nb, c_lo, c_hi);
  else
    k_gemm_update<double><<<grid, kGThreads, 0, L.stream>>>(d, k0, nb, c_lo, c_hi);
  count_launch(1);
}

void launch_make_perm(const Launch& L, const MatInst* d, int ninst, int64_t nmax) {
  k_make_perm<<<dim3((unsigned)((nmax + 255) / 256), (unsigned)ninst), 256, 0, L.stream>>>(d);
  count_launch(1);
}

}  // namespace bemgpu
