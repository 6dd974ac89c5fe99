// Triangular solves with a factored system, op(LU) x = b for op = A, A^H.
//
// Bound by latency for one system and by memory for a batch.  The factor's diagonal blocks
// (kTriNB rows) are inverted once per factorisation, so a solve is a chain of block rows
//   x_b = D_b^{-1} (b_b - sum_{j before b} op(T)_{bj} x_j)
// with no dependent steps inside a block.  One cooperative launch walks the chain: a CTA owns
// a block row, its warps stream the blocks in solve order with the next block's entries
// already in registers and wait for the x_j they need.  The vector is its own flag: the
// destination is filled with a bit pattern no arithmetic produces (an all-ones NaN), and a lane
// polls the entries it needs until they differ, so publishing is one store and needs neither a
// fence nor a flag.  Waits only point at blocks earlier in the order, every CTA takes its
// blocks in that order and all CTAs are resident, so the chain always advances; the waits are
// bounded all the same.  About 3 us a block row.  Measured per solve (both triangles) against
// one CTA per 512-row diagonal block and a product launch between the blocks: 1280 unknowns
// 0.61 -> 0.12 ms, 8960 unknowns 5.1 -> 0.85 ms (complex64), 5760 unknowns 15.2 -> 4.5 ms
// (complex128), 64 systems of 10240 unknowns 11.4 -> 9.0 ms (6 TB/s).
//
// Blocks: 64 rows in complex64, 32 in complex128 (the products with the inverse are on the
// critical path; 128 and 64 rows took 1.3 times as long), the inverse staged by one bulk copy.
// RG right-hand sides share every loaded entry.  Each row's sum has a fixed order
// (the blocks in solve order, inside a block a fixed split over threads) that depends on
// neither the batch nor RG.
//
// Accuracy: multiplying by an inverse is less accurate than substitution by up to the block's
// condition, so each block takes one correction with its own entries (x = y + D^{-1}(v - T y)),
// after which the backward errors are those of substitution (without it: two to four times
// those in complex128 at 128 to 300 unknowns, one refinement step more at 20480 unknowns in
// complex64).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "bemgpu_internal.h"
#include "linalg.cuh"
#include "tma.cuh"

namespace bemgpu {

namespace {
constexpr int kTriThreads = 512;
template <typename R>
constexpr int kTriNB = sizeof(R) == 4 ? 64 : 32;

template <int RG>
constexpr int kTriCtas = RG == 1 ? 2 : 1;  // per SM

template <typename R>
struct Vec;
template <>
struct Vec<float> {
  using T = float2;
};
template <>
struct Vec<double> {
  using T = double2;
};
template <typename R>
__device__ __forceinline__ cx<R> ldv(const void* p, int64_t i) {
  const typename Vec<R>::T v = static_cast<const typename Vec<R>::T*>(p)[i];
  return {v.x, v.y};
}
// an entry that has not been written yet (half of one counts)
__device__ __forceinline__ bool unset(cx<float> v) {
  return __float_as_uint(v.x) == 0xFFFFFFFFu || __float_as_uint(v.y) == 0xFFFFFFFFu;
}
__device__ __forceinline__ bool unset(cx<double> v) {
  return __double_as_longlong(v.x) == -1LL || __double_as_longlong(v.y) == -1LL;
}
template <typename R>
__device__ __forceinline__ cx<R> ldv_volatile(const void* p, int64_t i);
template <>
__device__ __forceinline__ cx<float> ldv_volatile<float>(const void* p, int64_t i) {
  cx<float> v;
  asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];"
               : "=f"(v.x), "=f"(v.y)
               : "l"(static_cast<const float2*>(p) + i)
               : "memory");
  return v;
}
template <>
__device__ __forceinline__ cx<double> ldv_volatile<double>(const void* p, int64_t i) {
  cx<double> v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "l"(static_cast<const double2*>(p) + i)
               : "memory");
  return v;
}
__device__ __forceinline__ void stv_relaxed(void* p, int64_t i, cx<float> v) {
  asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(static_cast<float2*>(p) + i),
               "f"(v.x), "f"(v.y)
               : "memory");
}
__device__ __forceinline__ void stv_relaxed(void* p, int64_t i, cx<double> v) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(static_cast<double2*>(p) + i),
               "d"(v.x), "d"(v.y)
               : "memory");
}
template <typename R>
__device__ __forceinline__ cx<R> recip(cx<R> a) {
  const R s = fmax(fabs(a.x), fabs(a.y));
  const R ar = a.x / s, ai = a.y / s;
  const R d = (ar * ar + ai * ai) * s;
  return {ar / d, -ai / d};
}
template <typename R>
__device__ __forceinline__ void fma_c(cx<R>& s, cx<R> a, cx<R> b) {
  s.x = fma(-a.y, b.y, fma(a.x, b.x, s.x));
  s.y = fma(a.y, b.x, fma(a.x, b.y, s.y));
}
}  // namespace

int tri_block(int prec) { return prec == 1 ? kTriNB<float> : kTriNB<double>; }
size_t tri_inv_bytes(int64_t n, int prec) {
  const int64_t nb = tri_block(prec), blocks = (n + nb - 1) / nb;
  return (size_t)(2 * blocks * nb * nb) * (prec == 1 ? 8 : 16);
}

// ------------------------------------------------------------------ block inverses
// grid (block, instance, triangle): inverses of the unit lower (z = 0) and the upper (z = 1)
// diagonal blocks, column-major kTriNB x kTriNB, zero outside the triangle and the matrix.  One
// warp per column of the inverse, the block in shared memory.
template <typename R>
__global__ void __launch_bounds__(kTriThreads) k_tri_inv(const MatInst* __restrict__ insts) {
  using C = cx<R>;
  constexpr int NB = kTriNB<R>, kPer = NB / 32, LD = NB + 1;
  const MatInst& M = insts[blockIdx.y];
  const int64_t n = M.n, r0 = (int64_t)blockIdx.x * NB;
  if (!M.active || r0 >= n) return;
  const int nbe = (int)min((int64_t)NB, n - r0);
  const bool upper = blockIdx.z == 1;
  extern __shared__ __align__(16) unsigned char tri_smem[];
  C* s = reinterpret_cast<C*>(tri_smem);  // [NB][LD], row-major
  C* di = s + NB * LD;                    // reciprocals of the upper block's diagonal
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int e = tid; e < nbe * nbe; e += kTriThreads) {
    const int r = e % nbe, c = e / nbe;
    s[r * LD + c] = ldv<R>(M.a, (r0 + r) + (r0 + c) * M.lda);
  }
  __syncthreads();
  if (upper && tid < nbe) di[tid] = recip(s[tid * LD + tid]);
  __syncthreads();
  const int64_t blocks = (n + NB - 1) / NB;
  C* out = static_cast<C*>(M.dinv) + ((upper ? blocks : 0) + blockIdx.x) * NB * NB;
  for (int j = wid; j < NB; j += kTriThreads / 32) {
    C x[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) x[t] = C{lane + 32 * t == j && j < nbe ? (R)1 : (R)0, (R)0};
    if (j < nbe) {
      if (!upper) {
#pragma unroll
        for (int t = 0; t < kPer; ++t)
          for (int cl = 0; cl < 32; ++cl) {
            const int c = 32 * t + cl;
            if (c >= nbe) break;
            if (c < j) continue;
            const C xc = {__shfl_sync(0xffffffffu, x[t].x, cl),
                          __shfl_sync(0xffffffffu, x[t].y, cl)};
#pragma unroll
            for (int u = t; u < kPer; ++u) {
              const int r = lane + 32 * u;
              if (r > c && r < nbe) x[u] -= s[r * LD + c] * xc;
            }
          }
      } else {
#pragma unroll
        for (int t = kPer - 1; t >= 0; --t)
          for (int cl = 31; cl >= 0; --cl) {
            const int c = 32 * t + cl;
            if (c > j) continue;
            if (lane == cl) x[t] = x[t] * di[c];
            const C xc = {__shfl_sync(0xffffffffu, x[t].x, cl),
                          __shfl_sync(0xffffffffu, x[t].y, cl)};
#pragma unroll
            for (int u = 0; u <= t; ++u) {
              const int r = lane + 32 * u;
              if (r < c) x[u] -= s[r * LD + c] * xc;
            }
          }
      }
    }
#pragma unroll
    for (int t = 0; t < kPer; ++t) out[lane + 32 * t + (int64_t)j * NB] = x[t];
  }
}

template <typename R>
static void tri_inv_t(const Launch& L, const MatInst* d, int ninst, int64_t nmax) {
  constexpr int NB = kTriNB<R>;
  const size_t smem = sizeof(cx<R>) * (size_t)(NB * (NB + 1) + NB);
  static PerDeviceOnce attr;
  attr.call([&] {
    cudaFuncSetAttribute(k_tri_inv<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  k_tri_inv<R><<<dim3((unsigned)((nmax + NB - 1) / NB), (unsigned)ninst, 2), kTriThreads, smem,
                 L.stream>>>(d);
  count_launch(1);
}

void launch_tri_inv(const Launch& L, const MatInst* d, int ninst, int64_t nmax, int prec) {
  if (ninst <= 0 || nmax <= 0) return;
  if (prec == 1)
    tri_inv_t<float>(L, d, ninst, nmax);
  else
    tri_inv_t<double>(L, d, ninst, nmax);
}

// ------------------------------------------------------------------ the chain
// Partial sums of the block's rows to shared memory (op(A) = A: one per row and thread of the
// row; A^H: the warp's sum), and the sum of a row; all threads take part in row_sums.
template <class C, bool TRANS, int RG, int RW, int KQ, int NB>
__device__ __forceinline__ void row_sums(const C (&s)[TRANS ? RW : 1][RG], C* sred, int nr,
                                         int tid) {
  if (!TRANS) {
#pragma unroll
    for (int g = 0; g < RG; ++g)
      if (g < nr) sred[(g * KQ + tid / NB) * NB + tid % NB] = s[0][g];
  } else {
#pragma unroll
    for (int u = 0; u < (TRANS ? RW : 1); ++u)
#pragma unroll
      for (int g = 0; g < RG; ++g)
        if (g < nr) {
          C t = s[u][g];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
            t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
          }
          if ((tid & 31) == 0) sred[g * KQ * NB + (tid >> 5) * RW + u] = t;
        }
  }
  __syncthreads();
}
template <class C, bool TRANS, int KQ, int NB>
__device__ __forceinline__ C row_sum(const C* sred, int g, int r) {
  C t = sred[g * KQ * NB + r];
  if (!TRANS) {
#pragma unroll
    for (int u = 1; u < KQ; ++u) t += sred[(g * KQ + u) * NB + r];
  }
  return t;
}

// LOWER: op(T) is lower triangular (blocks in ascending order).  T is L when LOWER != TRANS.
// Block rows q0 <= q < q1 of the chain; the source is x or y (src_y), through perm when swaps is
// set, the destination the other one, filled with the unset pattern.
struct ChainArgs {
  int ninst, groups;
  int64_t q0, q1;
  int swaps, src_y;
};
template <typename R, bool LOWER, bool TRANS, int RG>
__global__ void __launch_bounds__(kTriThreads, kTriCtas<RG>)
    k_trsv_chain(const MatInst* __restrict__ insts, const ChainArgs args, int* err) {
  using C = cx<R>;
  constexpr int NB = kTriNB<R>;
  constexpr int P = NB * NB / kTriThreads;      // entries of a block per thread
  constexpr int KQ = kTriThreads / NB;          // op(A) = A: threads per row
  constexpr int RW = NB / (kTriThreads / 32);   // op(A) = A^H: rows per warp
  constexpr int KL = NB / 32;                   //              entries per lane and row
  constexpr bool kUpperTri = LOWER == TRANS;
  constexpr int kOwn = (RG * NB + kTriThreads - 1) / kTriThreads;  // rows per thread
  extern __shared__ __align__(128) unsigned char chain_smem[];
  C* sD = reinterpret_cast<C*>(chain_smem);       // [NB * NB] inverse of the diagonal block
  C* sx = sD + NB * NB;                         // [RG][NB]
  C* sred = sx + RG * NB;                       // [RG][KQ][NB]
  C* sw = sred;                                 // [warp][RG][32], before the sums
  static_assert(P <= 32 && KQ * NB == kTriThreads, "a warp's columns, shared sums");
  __shared__ alignas(8) uint64_t bar;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int row = tid % NB, kq = tid / NB;
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  uint32_t phase = 0;
  const int groups = args.groups;
  const int64_t per = (int64_t)args.ninst * groups, items = (args.q1 - args.q0) * per;
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const int64_t q = args.q0 + item / per;     // position of the block in the chain
    const int inst = (int)(item % per) / groups, grp = (int)(item % per) % groups;
    const MatInst& M = insts[inst];
    const int64_t n = M.n, nblk = (n + NB - 1) / NB;
    const int r0g = grp * RG;
    if (!M.active || q >= nblk || r0g >= M.nrhs) continue;  // uniform over the CTA
    const int nr = min(RG, M.nrhs - r0g);
    const int64_t lda = M.lda, ldx = M.ldx;
    const void* src = args.src_y ? M.y : M.x;
    void* dst = args.src_y ? M.x : M.y;
    const int64_t b = LOWER ? q : nblk - 1 - q, row0 = b * NB;
    __syncthreads();  // the previous item is done with shared memory
    if (tid == 0) {
      constexpr uint32_t bytes = NB * NB * sizeof(C);
      mbar_arrive_expect_tx(&bar, bytes);
      bulk_g2s(sD, static_cast<const C*>(M.dinv) + ((kUpperTri ? nblk : 0) + b) * NB * NB, bytes,
               &bar);
    }
    C bv[kOwn];  // the right-hand sides of this thread's rows
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const int e = tid + o * kTriThreads;
      const int64_t r = row0 + e % NB;
      bv[o] = C{0, 0};
      if (e < nr * NB && r < n)
        bv[o] = ldv<R>(src, (int64_t)(r0g + e / NB) * ldx + (args.swaps ? M.perm[r] : r));
    }
    C pre[P];  // as stored: conjugated where used, as a use at the load would wait for it
    auto fetch = [&](int64_t qj) {  // this thread's entries of block (b, j)
      const int64_t c0 = (LOWER ? qj : nblk - 1 - qj) * NB;
      if (!TRANS) {
        const bool ok = row0 + row < n;
#pragma unroll
        for (int e = 0; e < P; ++e) {
          const int64_t c = c0 + kq * P + e;
          pre[e] = ok && c < n ? ldv<R>(M.a, (row0 + row) + c * lda) : C{0, 0};
        }
      } else {
#pragma unroll
        for (int e = 0; e < P; ++e) {
          const int64_t r = row0 + wid * RW + e / KL, c = c0 + lane + 32 * (e % KL);
          pre[e] = r < n && c < n ? ldv<R>(M.a, c + r * lda) : C{0, 0};
        }
      }
    };
    C acc[TRANS ? RW : 1][RG];
#pragma unroll
    for (int u = 0; u < (TRANS ? RW : 1); ++u)
#pragma unroll
      for (int g = 0; g < RG; ++g) acc[u][g] = C{0, 0};
    // Warps advance on their own: each polls the flag, takes the x values of its columns and
    // adds its products while the next block's entries are in flight.
    if (q > args.q0) fetch(args.q0);
    bool ok = true;
    C* wx = sw + wid * RG * 32;  // op(A) = A: x at the P columns of the warp's row segment
    for (int64_t qj = args.q0; qj < q; ++qj) {
      const int64_t c0 = (LOWER ? qj : nblk - 1 - qj) * NB;
      // entry c of right-hand side g, once it has been written
      auto await = [&](int g, int64_t c, bool want, C& v) {
        const int64_t i = (int64_t)(r0g + g) * ldx + c;
        want = want && c < n;
        v = C{0, 0};
        for (uint32_t it = 0; it < kSpinLimit; ++it) {
          if (want) v = ldv_volatile<R>(dst, i);
          if (!__any_sync(0xffffffffu, want && unset(v))) return true;
          if ((it & 1023) == 1023 && *(volatile int*)err) return false;  // another CTA gave up
        }
        if (lane == 0) atomicExch(err, kErrTimeout);
        return false;
      };
      auto await_row = [&](int g, int64_t c, C(&v)[KL]) {  // the entries c + 32 i
        const int64_t i0 = (int64_t)(r0g + g) * ldx + c;
#pragma unroll
        for (int i = 0; i < KL; ++i) v[i] = C{0, 0};
        for (uint32_t it = 0; it < kSpinLimit; ++it) {
          bool missing = false;
#pragma unroll
          for (int i = 0; i < KL; ++i)
            if (c + 32 * i < n) v[i] = ldv_volatile<R>(dst, i0 + 32 * i);
#pragma unroll
          for (int i = 0; i < KL; ++i) missing = missing || (c + 32 * i < n && unset(v[i]));
          if (!__any_sync(0xffffffffu, missing)) return true;
          if ((it & 1023) == 1023 && *(volatile int*)err) return false;  // another CTA gave up
        }
        if (lane == 0) atomicExch(err, kErrTimeout);
        return false;
      };
      if (!TRANS) {
#pragma unroll
        for (int g = 0; g < RG; ++g) {
          if (g >= nr) break;
          C v;
          ok = ok && await(g, c0 + kq * P + lane, lane < P, v);
          if (lane < P) wx[g * 32 + lane] = v;
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < P; ++e)
#pragma unroll
          for (int g = 0; g < RG; ++g)
            if (g < nr) fma_c(acc[0][g], pre[e], wx[g * 32 + e]);
        __syncwarp();
      } else {
#pragma unroll
        for (int g = 0; g < RG; ++g) {
          if (g >= nr) break;
          C xv[KL];
          // all of a lane's entries in one round: the next round trip starts at the last's end
          ok = ok && await_row(g, c0 + lane, xv);
#pragma unroll
          for (int e = 0; e < P; ++e)
            fma_c(acc[TRANS ? e / KL : 0][g], C{pre[e].x, -pre[e].y}, xv[e % KL]);
        }
      }
      if (!ok) break;
      if (qj + 1 < q) fetch(qj + 1);
    }
    ok = !__syncthreads_or(!ok);
    if (ok) fetch(q);  // the diagonal block itself
    if (!ok) {  // the copy in flight lands before the CTA leaves (bounded)
      if (tid == 0) mbar_wait(&bar, phase, err);
      __syncthreads();
      return;
    }
    // the rows' sums; v = b - sum, then y = D^{-1} v the same way
    row_sums<C, TRANS, RG, RW, KQ, NB>(acc, sred, nr, tid);
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const int e = tid + o * kTriThreads;
      if (e < nr * NB) {
        bv[o] = bv[o] - row_sum<C, TRANS, KQ, NB>(sred, e / NB, e % NB);
        if (row0 + e % NB >= n) bv[o] = C{0, 0};
        sx[e] = bv[o];
      }
    }
    __syncthreads();
    const bool here = mbar_wait(&bar, phase, err);
    phase ^= 1;
    if (__syncthreads_or(!here)) return;
    // sred's rows = D^{-1} times the vectors in sx
    auto times_inverse = [&]() {
      C y[TRANS ? RW : 1][RG];
#pragma unroll
      for (int u = 0; u < (TRANS ? RW : 1); ++u)
#pragma unroll
        for (int g = 0; g < RG; ++g) y[u][g] = C{0, 0};
#pragma unroll
      for (int e = 0; e < P; ++e) {
        const int c = TRANS ? lane + 32 * (e % KL) : kq * P + e;
        C d;
        if (TRANS) {
          d = sD[c + (wid * RW + e / KL) * NB];
          d.y = -d.y;
        } else {
          d = sD[row + c * NB];
        }
#pragma unroll
        for (int g = 0; g < RG; ++g)
          if (g < nr) fma_c(y[TRANS ? e / KL : 0][g], d, sx[g * NB + c]);
      }
      row_sums<C, TRANS, RG, RW, KQ, NB>(y, sred, nr, tid);
    };
    times_inverse();
    {
      // r = v - op(T)_bb y with the block's own entries, x = y + D^{-1} r
      constexpr bool kUnit = !kUpperTri;
      C yv[kOwn];
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int e = tid + o * kTriThreads;
        if (e < nr * NB) yv[o] = row_sum<C, TRANS, KQ, NB>(sred, e / NB, e % NB);
      }
      __syncthreads();
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int e = tid + o * kTriThreads;
        if (e < nr * NB) sx[e] = yv[o];
      }
      __syncthreads();
      C t[TRANS ? RW : 1][RG];
#pragma unroll
      for (int u = 0; u < (TRANS ? RW : 1); ++u)
#pragma unroll
        for (int g = 0; g < RG; ++g) t[u][g] = C{0, 0};
#pragma unroll
      for (int e = 0; e < P; ++e) {
        const int c = TRANS ? lane + 32 * (e % KL) : kq * P + e;
        const int r = TRANS ? wid * RW + e / KL : row;
        const int i = TRANS ? c : r, j = TRANS ? r : c;  // entry of T
        if (kUnit ? i > j : i <= j) {
#pragma unroll
          for (int g = 0; g < RG; ++g)
            if (g < nr)
              fma_c(t[TRANS ? e / KL : 0][g], TRANS ? C{pre[e].x, -pre[e].y} : pre[e],
                    sx[g * NB + c]);
        }
      }
      row_sums<C, TRANS, RG, RW, KQ, NB>(t, sred, nr, tid);
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int e = tid + o * kTriThreads, g = e / NB, r = e % NB;
        if (e < nr * NB) {
          C v = bv[o] - row_sum<C, TRANS, KQ, NB>(sred, g, r);
          if (kUnit) v -= yv[o];
          sx[e] = row0 + r < n ? v : C{0, 0};
        }
      }
      __syncthreads();
      times_inverse();
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int e = tid + o * kTriThreads, g = e / NB, r = e % NB;
        if (e < nr * NB && row0 + r < n)
          stv_relaxed(dst, (int64_t)(r0g + g) * ldx + row0 + r,
                      yv[o] + row_sum<C, TRANS, KQ, NB>(sred, g, r));
      }
    }
  }
}

// every entry of x or y: not written yet
template <typename R>
__global__ void k_tri_unset(const MatInst* __restrict__ insts, int of_y) {
  const MatInst& M = insts[blockIdx.z];
  const int rhs = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!M.active || rhs >= M.nrhs || i >= M.n) return;
  cx<R> v;
  if constexpr (sizeof(R) == 4)
    v.x = v.y = __uint_as_float(0xFFFFFFFFu);
  else
    v.x = v.y = __longlong_as_double(-1LL);
  stv_relaxed(of_y ? M.y : M.x, (int64_t)rhs * M.ldx + i, v);
}

// ------------------------------------------------------------------ many right-hand sides
// With many right-hand sides the work, not the chain, is the bound: the chain solves outer
// blocks of kOuter block rows for all of them, and a tiled product takes each solved block out
// of the rows that follow.  128 x N tiles, 4 x N / 8 entries per thread, K-chunks of 16 with the
// next chunk in registers; every entry adds its columns in order with the same four FMAs.
// Complex64 is bound by FP32 issue: the four FMAs of two right-hand sides go through the paired
// instructions, and with more than 32 right-hand sides a thread takes eight of them, which halves
// its loads of A.  One solve of 20480 unknowns with 181 right-hand sides: 33 ms with a product
// kernel of eight right-hand sides per CTA, 23 with 128 x 32 tiles and six single operations an
// entry, 18 so (8 ms at the FP32 peak).
constexpr int kManyRhs = 8;   // right-hand sides of a system from which this path is taken
constexpr int kOuter = 8;
constexpr int kUpM = 128, kUpK = 16;

// The tile's products in shared memory: A and the vectors' chunk, whose complex64 parts lie in
// planes (real, imaginary, -imaginary) so that neighbouring right-hand sides make a pair.
template <typename R, int N>
struct UpTile {
  using C = cx<R>;
  C a[kUpK][kUpM];
  C x[kUpK][N + 1];
  __device__ void put(int k, int g, C v) { x[k][g] = v; }
};
template <int N>
struct UpTile<float, N> {
  using C = cx<float>;
  C a[kUpK][kUpM];
  alignas(16) float re[kUpK][N + 4], im[kUpK][N + 4], ni[kUpK][N + 4];
  __device__ void put(int k, int g, C v) {
    re[k][g] = v.x;
    im[k][g] = v.y;
    ni[k][g] = -v.y;
  }
};
template <typename R, int TN>
struct UpSum {
  using C = cx<R>;
  C acc[4][TN];
  __device__ void zero() {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < TN; ++b) acc[a][b] = C{0, 0};
  }
  __device__ void add(const UpTile<R, 8 * TN>& t, int kk, int tx, int ty) {
    C av[4], xv[TN];
#pragma unroll
    for (int a = 0; a < 4; ++a) av[a] = t.a[kk][tx + 32 * a];
#pragma unroll
    for (int b = 0; b < TN; ++b) xv[b] = t.x[kk][ty * TN + b];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < TN; ++b) fma_c(acc[a][b], av[a], xv[b]);
  }
  __device__ C get(int a, int b) const { return acc[a][b]; }
};
template <int TN>
struct UpSum<float, TN> {
  using C = cx<float>;
  float2 re[4][TN / 2], im[4][TN / 2];
  __device__ void zero() {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < TN / 2; ++b) re[a][b] = im[a][b] = make_float2(0.f, 0.f);
  }
  __device__ void add(const UpTile<float, 8 * TN>& t, int kk, int tx, int ty) {
    C av[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) av[a] = t.a[kk][tx + 32 * a];
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {  // four right-hand sides at a time
      const float4 r = *reinterpret_cast<const float4*>(&t.re[kk][ty * TN + 4 * h]);
      const float4 i = *reinterpret_cast<const float4*>(&t.im[kk][ty * TN + 4 * h]);
      const float4 m = *reinterpret_cast<const float4*>(&t.ni[kk][ty * TN + 4 * h]);
      const float2 br[2] = {make_float2(r.x, r.y), make_float2(r.z, r.w)};
      const float2 bi[2] = {make_float2(i.x, i.y), make_float2(i.z, i.w)};
      const float2 bm[2] = {make_float2(m.x, m.y), make_float2(m.z, m.w)};
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float2 ax = make_float2(av[a].x, av[a].x), ay = make_float2(av[a].y, av[a].y);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          float2& sr = re[a][2 * h + b];
          float2& si = im[a][2 * h + b];
          sr = __ffma2_rn(ay, bm[b], __ffma2_rn(ax, br[b], sr));
          si = __ffma2_rn(ay, br[b], __ffma2_rn(ax, bi[b], si));
        }
      }
    }
  }
  __device__ C get(int a, int b) const {
    const float2 r = re[a][b / 2], i = im[a][b / 2];
    return b & 1 ? C{r.y, i.y} : C{r.x, i.x};
  }
};

template <typename R, bool LOWER, int TN>
__global__ void __launch_bounds__(256, TN == 8 ? 2 : 1)
    k_many_update(const MatInst* __restrict__ insts, int64_t q0, int64_t q1, int src_y) {
  using C = cx<R>;
  constexpr int NB = kTriNB<R>, kUpN = 8 * TN;
  const MatInst& M = insts[blockIdx.z];
  const int64_t n = M.n, nblk = (n + NB - 1) / NB;
  if (!M.active || q0 >= nblk) return;
  // solved columns [c0, c1), rows [lo, hi) to update
  const int64_t e1 = min(q1, nblk);
  const int64_t c0 = LOWER ? q0 * NB : (nblk - e1) * NB;
  const int64_t c1 = LOWER ? min(e1 * NB, n) : min((nblk - q0) * NB, n);
  const int64_t lo = LOWER ? c1 : 0, hi = LOWER ? n : c0;
  const int64_t r0 = lo + (int64_t)blockIdx.x * kUpM;
  const int g0 = blockIdx.y * kUpN;
  if (r0 >= hi || g0 >= M.nrhs) return;  // uniform over the CTA
  const int64_t lda = M.lda, ldx = M.ldx;
  const void* sol = src_y ? M.x : M.y;   // the chain's destination
  void* rest = src_y ? M.y : M.x;
  __shared__ UpTile<R, kUpN> tile;
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  UpSum<R, TN> sum;
  sum.zero();
  constexpr int kA = kUpM * kUpK / 256, kX = kUpN * kUpK / 256;
  C na[kA], nx[kX];
  auto load = [&](int64_t k) {
#pragma unroll
    for (int e = 0; e < kA; ++e) {
      const int t = tid + 256 * e;
      const int64_t r = r0 + t % kUpM, c = k + t / kUpM;
      na[e] = r < hi && c < c1 ? ldv<R>(M.a, r + c * lda) : C{0, 0};
    }
#pragma unroll
    for (int e = 0; e < kX; ++e) {
      const int t = tid + 256 * e;
      const int64_t c = k + t % kUpK;
      const int g = g0 + t / kUpK;
      nx[e] = g < M.nrhs && c < c1 ? ldv<R>(sol, (int64_t)g * ldx + c) : C{0, 0};
    }
  };
  load(c0);
  for (int64_t k = c0; k < c1; k += kUpK) {
#pragma unroll
    for (int e = 0; e < kA; ++e) {
      const int t = tid + 256 * e;
      tile.a[t / kUpM][t % kUpM] = na[e];
    }
#pragma unroll
    for (int e = 0; e < kX; ++e) {
      const int t = tid + 256 * e;
      tile.put(t % kUpK, t / kUpK, nx[e]);
    }
    __syncthreads();
    if (k + kUpK < c1) load(k + kUpK);
#pragma unroll
    for (int kk = 0; kk < kUpK; ++kk) sum.add(tile, kk, tx, ty);
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < TN; ++b) {
      const int64_t r = r0 + tx + 32 * a;
      const int g = g0 + ty * TN + b;
      if (r < hi && g < M.nrhs) {
        const int64_t i = (int64_t)g * ldx + r;
        C v = ldv<R>(rest, i);
        v -= sum.get(a, b);
        stv_relaxed(rest, i, v);
      }
    }
}

// to_y: y = P x; else x = y
template <typename R>
__global__ void k_tri_move(const MatInst* __restrict__ insts, int to_y, int swaps) {
  const MatInst& M = insts[blockIdx.z];
  const int rhs = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!M.active || rhs >= M.nrhs || i >= M.n) return;
  const int64_t off = (int64_t)rhs * M.ldx;
  stv_relaxed(to_y ? M.y : M.x, off + i, ldv<R>(to_y ? M.x : M.y, off + (swaps ? M.perm[i] : i)));
}

namespace {
struct ChainOrder {
  std::mutex mu;
  cudaEvent_t last = nullptr;  // end of the device's most recent chain
};
ChainOrder& chain_order() {
  static ChainOrder per_device[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  return per_device[dev];
}
}  // namespace

template <typename R, bool LOWER, bool TRANS, int RG>
static void chain_t(const Launch& L, const MatInst* d, ChainArgs args, int32_t max_rhs) {
  constexpr int NB = kTriNB<R>;
  constexpr size_t smem = sizeof(cx<R>) * (size_t)(NB * NB + RG * NB + RG * kTriThreads);
  auto kernel = k_trsv_chain<R, LOWER, TRANS, RG>;
  static PerDeviceOnce attr;
  attr.call([&] {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  args.groups = (max_rhs + RG - 1) / RG;
  const int64_t items = (args.q1 - args.q0) * args.ninst * args.groups;
  const int64_t resident = (int64_t)kTriCtas<RG> * device_sm_count();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(items, resident));
  cfg.blockDim = dim3(kTriThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = L.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  // two chains on different streams, each holding part of the SMs, would wait for CTAs of
  // their own that cannot start: the chains of a device run one after the other
  ChainOrder& order = chain_order();
  std::lock_guard<std::mutex> lk(order.mu);
  if (!order.last) cudaEventCreateWithFlags(&order.last, cudaEventDisableTiming);
  cudaStreamWaitEvent(L.stream, order.last, 0);
  cudaLaunchKernelEx(&cfg, kernel, d, args, L.err_flag);
  cudaEventRecord(order.last, L.stream);
  count_launch(1);
}

// One triangle.  many: outer blocks with products between them.
template <typename R, bool LOWER, bool TRANS>
static void triangle(const Launch& L, const MatInst* d, int ninst, int64_t nmax, int32_t max_rhs,
                     int src_y, int swaps, bool many) {
  constexpr int NB = kTriNB<R>;
  const int64_t nblk = (nmax + NB - 1) / NB;
  k_tri_unset<R><<<dim3((unsigned)((nmax + 255) / 256), (unsigned)max_rhs, (unsigned)ninst), 256, 0,
                   L.stream>>>(d, !src_y);
  count_launch(1);
  ChainArgs args{ninst, 1, 0, nblk, swaps, src_y};
  if constexpr (!TRANS) {
    if (many) {
      for (int64_t q = 0; q < nblk; q += kOuter) {
        args.q0 = q;
        args.q1 = std::min<int64_t>(q + kOuter, nblk);
        chain_t<R, LOWER, false, 4>(L, d, args, max_rhs);
        // rows after the outer block (short instances have fewer and skip the tiles)
        const int64_t rows = nmax - q * NB;
        if (args.q1 < nblk) {
          const int tn = sizeof(R) == 4 && max_rhs > 32 ? 8 : 4;  // right-hand sides a thread
          const dim3 grid((unsigned)((rows + kUpM - 1) / kUpM),
                          (unsigned)((max_rhs + 8 * tn - 1) / (8 * tn)), (unsigned)ninst);
          if (tn == 4) {
            k_many_update<R, LOWER, 4><<<grid, 256, 0, L.stream>>>(d, q, args.q1, src_y);
          } else {
            if constexpr (sizeof(R) == 4)
              k_many_update<R, LOWER, 8><<<grid, 256, 0, L.stream>>>(d, q, args.q1, src_y);
          }
          count_launch(1);
        }
      }
      return;
    }
    if (max_rhs >= 4) return chain_t<R, LOWER, false, 4>(L, d, args, max_rhs);
  }
  chain_t<R, LOWER, TRANS, 1>(L, d, args, max_rhs);
}

template <typename R>
static void getrs_t(const Launch& L, const MatInst* d, int ninst, int64_t nmax, int32_t max_rhs,
                    int trans, int swaps, bool many) {
  const dim3 g((unsigned)((nmax + 255) / 256), (unsigned)max_rhs, (unsigned)ninst);
  if (trans) {  // (LU)^H = U^H L^H
    triangle<R, true, true>(L, d, ninst, nmax, max_rhs, 0, 0, false);
    triangle<R, false, true>(L, d, ninst, nmax, max_rhs, 1, 0, false);
  } else if (many) {  // the products change the source, so the permutation comes first
    k_tri_move<R><<<g, 256, 0, L.stream>>>(d, 1, swaps);
    triangle<R, true, false>(L, d, ninst, nmax, max_rhs, 1, 0, true);
    triangle<R, false, false>(L, d, ninst, nmax, max_rhs, 0, 0, true);
    k_tri_move<R><<<g, 256, 0, L.stream>>>(d, 0, 0);
    count_launch(2);
  } else {
    triangle<R, true, false>(L, d, ninst, nmax, max_rhs, 0, swaps, false);
    triangle<R, false, false>(L, d, ninst, nmax, max_rhs, 1, 0, false);
  }
}

bool many_rhs(int32_t nrhs) { return nrhs >= kManyRhs; }

void launch_getrs(const Launch& L, const MatInst* d, int ninst, int64_t nmax, int32_t max_rhs,
                  int trans, int prec, int swaps, bool many) {
  if (nmax <= 0 || ninst <= 0 || max_rhs <= 0) return;
  if (prec == 1)
    getrs_t<float>(L, d, ninst, nmax, max_rhs, trans, swaps, many);
  else
    getrs_t<double>(L, d, ninst, nmax, max_rhs, trans, swaps, many);
}

}  // namespace bemgpu
