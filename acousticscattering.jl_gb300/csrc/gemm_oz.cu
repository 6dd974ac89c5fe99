// Complex128 products on the bfloat16 tensor cores: C -= A B, in K-blocks of at most 128.
//
// The FP64 pipe of this part issues two FMAs per clock and SM (about 1.2 TFLOP/s over the
// GPU), the bfloat16 tensor cores 1.9 PFLOP/s.  The update is therefore computed from
// integer digits (the slicing of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59 (2012)):
// with one exponent per operand row, |x| <= 2^(e-1),
//   x = 2^e sum_{p=1..7} d_p 2^(-8p) + O(2^(e-57)),   d_p integers in [-128, 128],
// exact in bfloat16.  A product of two digits is at most 2^14, so the sum over K = 128
// complex terms is at most 2^22 per digit pair and exact in the FP32 accumulators; the
// pairs with p + q = d share one accumulator ("level" d = 2..9, at most seven pairs: exact
// up to d = 5 for any operands, and a few units of 2^(-8d) in the worst case beyond, below
// 2^-53 of the largest possible result).  The levels are added in 64-bit integers and
// rounded to FP64 once.  What is dropped (digits beyond the seventh, levels above 9) is about
// 2^-55 of sqrt(K) (largest |a| of the row) x (largest |b| of the column) of the K-block, below
// the accumulated rounding errors of 4 K FP64 operations when no index k stands out: backward
// errors of LUs of 128 to 2049 unknowns are those of the FP64 pipe's (stopping at level 8 made
// them up to twice as large).  It is not relative to sum_k |a||b|: where the sizes differ along
// k, the caller gives a power of two per k that moves between the operands (kexp).
//
// Tile and layout: 128 x 32 complex entries of C per CTA, all eight levels of the real and
// imaginary part in tensor memory (2 x 8 x 32 = 512 columns).  The levels of a part form two
// accumulators of N = 128, levels 2..5 and 6..9.  tcgen05.mma instructions are only ordered
// among themselves when they share accumulator and shape, so every instruction takes a whole
// accumulator: the B slices of a K-chunk are stacked along N (slice 1 first) between blocks of
// zeros, and slice p of A meets the four blocks that belong to the accumulator's levels, some
// of them zeros.  34 digit pairs take 11 instructions per real product, 1.3 times the tensor
// work of instructions cut to the slices that exist, whose accumulators overlap.  K-chunks of
// 16: rows of 64 bytes, 16 real then 16 imaginary digits, in the 64-byte swizzle.  A stage is 7
// slices of both operands and the zeros (78 KB), two stages.
//
// Roles as in gemm_tc.cu: a producer thread (bulk copies), a tcgen05.mma issuer, eight
// epilogue warps that move the levels of a tile to 64-bit integers in registers, release
// the tensor memory, then convert, scale and update C while the next tile's products run.
// Every wait is bounded.
//
// Bound by the tensor pipe and the shared-memory operand reads: 44 instructions of 64 cycles in
// each of the 8 chunks of a tile and K-block take at least 22.5k cycles, the FP64 conversion
// and update of the epilogue about 8k beside them, moving the levels out of tensor memory about
// 2k in between.  The trailing updates of an LU of 5760 unknowns: 718 ms on the FP64 pipe (0.7
// TFLOP/s), 13 ms here (12 with instructions cut to the slices that exist).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bemgpu_internal.h"
#include "gemm_oz.cuh"
#include "tc_common.cuh"

namespace bemgpu {

constexpr int kOzM = 128, kOzN = 32;        // tile of C
constexpr int kOzKC = 16;                   // K per chunk
constexpr int kOzBlockChunks = kOzK / kOzKC;
constexpr int kOzSlices = 7;
constexpr int kOzLevels = 8;                // digit products p + q = 2..9
constexpr int kOzABlock = kOzM * 64;        // one slice of a chunk, 64-byte rows
constexpr int kOzBBlock = kOzN * 64;
constexpr int kOzAChunk = kOzSlices * kOzABlock;  // 56 KB
constexpr int kOzBChunk = kOzSlices * kOzBBlock;  // 14 KB
constexpr int kOzLow = 3, kOzHigh = 1;      // blocks of zeros before and after the B slices
constexpr int kOzAccN = 4 * kOzN;           // columns of an accumulator: four levels
constexpr int kOzStage = kOzAChunk + (kOzLow + kOzHigh) * kOzBBlock + kOzBChunk;
constexpr int kOzStages = 2;
constexpr int kOzThreads = 320;             // producer, MMA, 8 epilogue warps
constexpr int kOzEpiThreads = 256;
constexpr uint32_t kOzTmem = 512;
constexpr uint32_t kOzIm = kOzLevels * kOzN;  // first tensor-memory column of the imaginary part
constexpr int kOzMark = 1 << 20;            // exponent field of such a row while it is packed
constexpr int kOzDrop = -200000;            // shift of a column that is taken as zeros
static_assert(kOzStage % 1024 == 0 && kOzABlock % 1024 == 0 && kOzBBlock % 1024 == 0, "swizzle");
static_assert(kOzLevels * kOzN == 2 * kOzAccN, "two accumulators");

// ------------------------------------------------------------------ slicing
// Fixed-point value of x 2^sh in units of 2^(e - 56), e = row exponent field - 1021.
__device__ __forceinline__ long long oz_fixed(double x, int sh, int erow) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF);
  long long m = (b & 0xFFFFFFFFFFFFFLL) | 0x10000000000000LL;
  const int s = ex + sh - erow + 2;  // <= 2
  if (ex == 0 || s < -53) return 0;
  m = s >= 0 ? m << s : (m + (1LL << (-s - 1))) >> -s;
  return b < 0 ? -m : m;
}
__device__ __forceinline__ long long oz_fixed(float x, int sh, int erow) {  // zero when subnormal
  const uint32_t b = __float_as_uint(x);
  const int ex = (int)((b >> 23) & 0xFF);
  long long m = (long long)((b & 0x7FFFFFu) | 0x800000u) << 29;
  const int s = ex + 896 + sh - erow + 2;  // exponent field of the same value in FP64
  if (ex == 0 || s < -53) return 0;
  m = s >= 0 ? m << s : (m + (1LL << (-s - 1))) >> -s;
  return (int32_t)b < 0 ? -m : m;
}
// FP64 exponent field of the larger of two magnitudes (0: none)
__device__ __forceinline__ int oz_expo(double2 v) {
  return (int)(max((uint32_t)__double2hiint(v.x) & 0x7FFFFFFFu,
                   (uint32_t)__double2hiint(v.y) & 0x7FFFFFFFu) >> 20);
}
__device__ __forceinline__ int oz_expo(float2 v) {
  const int e = (int)(max(__float_as_uint(v.x) & 0x7FFFFFFFu,
                          __float_as_uint(v.y) & 0x7FFFFFFFu) >> 23);
  return e == 0 ? 0 : e == 0xFF ? 0x7FF : e + 896;
}
// bfloat16 bits of two digits (biased by 128, 0..256)
__device__ __forceinline__ uint32_t oz_bf16x2(uint32_t d0, uint32_t d1) {
  const float f0 = __uint_as_float(0x4B000000u | d0) - 8388736.0f;
  const float f1 = __uint_as_float(0x4B000000u | d1) - 8388736.0f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// The field of an entry shifted by its column's scale, kOzMark for a NaN or an infinity, far
// below every field for a zero or a column taken as zeros.
__device__ __forceinline__ int oz_shifted(int field, int sh) {
  return field == 0x7FF ? kOzMark : field == 0 ? kOzDrop : field + sh;
}

// One CTA per R rows of an operand tile of T rows and K-block: the rows' exponents, then the
// slices, eight K values of one row per work item (14 vector stores of eight digits).  Integer
// work on small pieces: R is a quarter of the tile so that an operand of a few thousand rows
// fills the GPU.
template <class V2, int T, int R, bool TRANS>
__global__ void __launch_bounds__(256) k_oz_pack(const OzPackInst* __restrict__ insts) {
  const OzPackInst& P = insts[blockIdx.y];
  if ((P.single != 0) != (sizeof(V2) == sizeof(float2))) return;
  const int64_t row0 = (int64_t)blockIdx.x * R;
  // rows beyond the operand up to the end of its last tile are packed as zeros
  const int kb = (int)blockIdx.z * kOzK, kk = min(kOzK, P.kk - kb);
  if (row0 >= (P.rows + T - 1) / T * T || kk <= 0) return;
  const int64_t k0 = P.k0 + kb;
  constexpr int kBlock = T * 64, kChunk = kOzSlices * kBlock;
  constexpr int kPer = 256 / R;  // threads per row in the exponent pass
  __shared__ int s_exp[R], s_sh[kOzK];  // row exponents, column scales
  const V2* A = static_cast<const V2*>(P.a);
  const int tid = threadIdx.x;
  for (int r = tid; r < R; r += 256) s_exp[r] = kOzNone + 1021;
  if (tid < kOzK) {
    int sh = 0;
    if (P.kexp && tid < kk) {
      const int f = P.kexp[kb + tid];
      sh = f == 0 ? (TRANS ? 0 : kOzDrop) : TRANS ? 1023 - f : f - 1023;
    }
    s_sh[tid] = sh;
  }
  __syncthreads();
  {
    const int r = TRANS ? tid / kPer : tid % R, g = TRANS ? tid % kPer : tid / R;
    const int64_t gr = row0 + r;
    int mx = kOzNone + 1021;
    if (gr < P.rows)
      for (int k = g; k < kk; k += kPer)
        mx = max(mx, oz_shifted(oz_expo(A[TRANS ? (k0 + k) + (P.r0 + gr) * P.lda
                                                : (P.r0 + gr) + (k0 + k) * P.lda]),
                                s_sh[k]));
    atomicMax(&s_exp[r], mx);
  }
  __syncthreads();
  int32_t* exps = P.exps + (int64_t)blockIdx.z * ((P.rows + T - 1) / T * T);
  for (int r = tid; r < R; r += 256) {
    const int e = s_exp[r];
    exps[row0 + r] = e == kOzMark ? kOzNaN : e - 1021;
  }
  const int all = (P.kk + kOzKC - 1) / kOzKC, chunks = (kk + kOzKC - 1) / kOzKC;
  uint8_t* out = static_cast<uint8_t*>(P.out) + ((size_t)(row0 / T) * all + kb / kOzKC) * kChunk;
  const int rt = (int)(row0 % T);  // first row inside the tile
  const int groups = chunks * 2;  // eight K values each
  for (int item = tid; item < R * groups; item += 256) {
    const int r = TRANS ? item / groups : item % R, g = TRANS ? item % groups : item / R;
    const int64_t gr = row0 + r;
    const int erow = s_exp[r];
    unsigned long long zr[8], zi[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int k = g * 8 + e;
      V2 v = V2{0, 0};
      if (gr < P.rows && k < kk)
        v = A[TRANS ? (k0 + k) + (P.r0 + gr) * P.lda : (P.r0 + gr) + (k0 + k) * P.lda];
      // digits + 128 in the bytes (byte 6 keeps a carry into bit 8)
      const int sh = s_sh[k];
      zr[e] = (unsigned long long)(oz_fixed(v.x, sh, erow) + 0x0080808080808080LL);
      zi[e] = (unsigned long long)(oz_fixed(v.y, sh, erow) + 0x0080808080808080LL);
    }
    const int sw = ((rt + r) >> 1) & 3, half = g & 1;
    uint8_t* base = out + (size_t)(g >> 1) * kChunk + (rt + r) * 64;
#pragma unroll
    for (int p = 0; p < kOzSlices; ++p) {
      uint32_t wr[4], wi[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        auto dig = [&](unsigned long long z) {
          const uint32_t d = (uint32_t)(z >> (8 * (6 - p)));
          return p == 0 ? d : d & 0xFFu;
        };
        wr[e] = oz_bf16x2(dig(zr[2 * e]), dig(zr[2 * e + 1]));
        wi[e] = oz_bf16x2(dig(zi[2 * e]), dig(zi[2 * e + 1]));
      }
      uint8_t* o = base + p * kBlock;
      *reinterpret_cast<uint4*>(o + ((half ^ sw) << 4)) = make_uint4(wr[0], wr[1], wr[2], wr[3]);
      *reinterpret_cast<uint4*>(o + (((2 + half) ^ sw) << 4)) =
          make_uint4(wi[0], wi[1], wi[2], wi[3]);
    }
  }
}

// The scales of the K index from side B (complex128, at most kOzK of them): lanes along k,
// kKexpRows operand rows per CTA.  The largest of integers, whatever the order.  Bound by latency:
// a CTA's loads are one round.
constexpr int kKexpRows = 16;
__global__ void __launch_bounds__(256) k_oz_kexp(const OzPackInst* __restrict__ insts) {
  const OzPackInst& P = insts[blockIdx.y];
  const int64_t row0 = (int64_t)blockIdx.x * kKexpRows;
  if (row0 >= P.rows || P.kk <= 0) return;  // uniform over the CTA
  const int width = P.kk <= 32 ? 32 : kOzK, step = 256 / width;
  const int k = threadIdx.x % width;
  const int64_t end = min(row0 + kKexpRows, P.rows);
  const double2* A = static_cast<const double2*>(P.a) + P.k0 + k + P.r0 * P.lda;
  int mx = 0;
  if (k < P.kk) {
    constexpr int kFly = 8;
    for (int64_t r0 = row0 + threadIdx.x / width; r0 < end; r0 += kFly * step) {
      double2 v[kFly];
#pragma unroll
      for (int u = 0; u < kFly; ++u) {
        const int64_t r = r0 + u * step;
        v[u] = r < end ? A[r * P.lda] : double2{0.0, 0.0};
      }
#pragma unroll
      for (int u = 0; u < kFly; ++u) {
        const int x = (__double2hiint(v[u].x) >> 20) & 0x7FF;
        const int y = (__double2hiint(v[u].y) >> 20) & 0x7FF;
        mx = max(mx, max(x == 0x7FF ? 0 : x, y == 0x7FF ? 0 : y));
      }
    }
  }
  __shared__ int sh[256];
  sh[threadIdx.x] = mx;
  __syncthreads();
  if (threadIdx.x < width && k < P.kk) {
    for (int u = 1; u < step; ++u) mx = max(mx, sh[threadIdx.x + u * width]);
    atomicMax(P.kexp + k, mx);
  }
}

// ------------------------------------------------------------------ the GEMM
// Shared-memory descriptor: K-major operand, 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;  // SWIZZLE_64B
  return d;
}
// kind::f16, FP32 accumulate, BF16 operands, M = 128, N = n
__device__ __forceinline__ uint32_t oz_idesc(uint32_t n, bool negate_a) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((negate_a ? 1u : 0u) << 13) | ((n >> 3) << 17) |
         ((uint32_t)(kOzM >> 4) << 24);
}

struct OzShared {
  uint64_t full[kOzStages];
  uint64_t empty[kOzStages];
  uint64_t tfull, tempty;
  uint32_t tmem_base;
  int abort_flag;
  int32_t prefix[kOzMaxInst + 1];
};

__device__ __forceinline__ void oz_coords(const OzShared& S, const OzGemmInst* insts, int ninst,
                                          int64_t t, int* inst, int64_t* mt, int64_t* nt) {
  int lo = 0, hi = ninst - 1;  // largest instance with prefix <= t
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (S.prefix[mid] <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  const int64_t local = t - (int64_t)S.prefix[lo];
  *inst = lo;
  if (insts[lo].n_first) {
    const int64_t ntiles = (insts[lo].n + kOzN - 1) / kOzN;
    *nt = local % ntiles;
    *mt = local / ntiles;
  } else {
    const int64_t mtiles = (insts[lo].m + kOzM - 1) / kOzM;
    *mt = local % mtiles;
    *nt = local / mtiles;
  }
}

// v 2^t where 2^t is no normal number
__device__ __noinline__ double oz_scaled_far(double v, int t) { return scalbn(v, t); }
__device__ __forceinline__ double oz_scaled(long long v, int t) {
  if (t < -1022 || t > 1023) return oz_scaled_far((double)v, t);
  return (double)v * __longlong_as_double((long long)(t + 1023) << 52);
}

__global__ void __launch_bounds__(kOzThreads, 1)
    k_oz_gemm(const OzGemmInst* __restrict__ insts, int ninst, int* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  OzShared& S = *reinterpret_cast<OzShared*>(base + kOzStages * kOzStage);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (insts[0].gate && *insts[0].gate > insts[0].gate_cap) return;  // uniform over the grid
  if (threadIdx.x == 0) {
    for (int s = 0; s < kOzStages; ++s) {
      mbar_init(&S.full[s], 1);
      mbar_init(&S.empty[s], 1);
    }
    mbar_init(&S.tfull, 1);
    mbar_init(&S.tempty, kOzEpiThreads);
    S.abort_flag = 0;
    int32_t acc = 0;
    S.prefix[0] = 0;
    for (int i = 0; i < ninst; ++i) {
      const OzGemmInst& G = insts[i];
      if (G.m > 0 && G.n > 0 && G.kk > 0)
        acc += (int32_t)(((G.m + kOzM - 1) / kOzM) * ((G.n + kOzN - 1) / kOzN));
      S.prefix[i + 1] = acc;
    }
    mbar_fence_init();
  }
  // the zeros around the B slices of every stage, for the tensor core's reads
  for (int e = threadIdx.x; e < kOzStages * (kOzLow + kOzHigh) * kOzBBlock / 16; e += kOzThreads) {
    constexpr int kPer = kOzBBlock / 16;
    const int stage = e / ((kOzLow + kOzHigh) * kPer), r = e % ((kOzLow + kOzHigh) * kPer);
    const int block = r / kPer < kOzLow ? r / kPer : r / kPer + kOzSlices;
    *reinterpret_cast<uint4*>(base + stage * kOzStage + kOzAChunk + block * kOzBBlock +
                              r % kPer * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
            smem_addr(&S.tmem_base)),
        "r"(kOzTmem)
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  const int64_t total = S.prefix[ninst];
  volatile int* abort_flag = &S.abort_flag;

  if (warp == 0) {
    // ------------------------------------------------ producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int armed[kOzStages];
      uint32_t armed_par[kOzStages];
      for (int s = 0; s < kOzStages; ++s) armed[s] = 0, armed_par[s] = 0;
      for (int64_t t = blockIdx.x; t < total && !*abort_flag; t += gridDim.x) {
        int inst;
        int64_t mt, nt;
        oz_coords(S, insts, ninst, t, &inst, &mt, &nt);
        const OzGemmInst& G = insts[inst];
        const int chunks = (G.kk + kOzKC - 1) / kOzKC;
        const uint8_t* pa = static_cast<const uint8_t*>(G.apack) + (size_t)mt * chunks * kOzAChunk;
        const uint8_t* pb = static_cast<const uint8_t*>(G.bpack) + (size_t)nt * chunks * kOzBChunk;
        for (int c = 0; c < chunks; ++c) {
          if (!tc_wait(&S.empty[stage], phase ^ 1, err, abort_flag)) break;
          uint8_t* dst = base + stage * kOzStage;
          armed[stage] = 1;
          armed_par[stage] = phase;
          mbar_arrive_expect_tx(&S.full[stage], kOzAChunk + kOzBChunk);
          bulk_g2s(dst, pa + (size_t)c * kOzAChunk, kOzAChunk, &S.full[stage]);
          bulk_g2s(dst + kOzAChunk + kOzLow * kOzBBlock, pb + (size_t)c * kOzBChunk, kOzBChunk,
                   &S.full[stage]);
          if (++stage == kOzStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // every copy this thread issued has landed before the CTA exits (bounded)
      for (int q = 0; q < kOzStages; ++q) {
        if (!armed[q]) continue;
        for (uint32_t it = 0; it < kSpinLimit; ++it)
          if (mbar_try_wait(&S.full[q], armed_par[q])) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, tphase = 0;
      const uint32_t sbase = smem_addr(base);
      for (int64_t t = blockIdx.x; t < total && !*abort_flag; t += gridDim.x) {
        int inst;
        int64_t mt, nt;
        oz_coords(S, insts, ninst, t, &inst, &mt, &nt);
        const int chunks = (insts[inst].kk + kOzKC - 1) / kOzKC;
        bool ok = true;
        for (int c = 0; c < chunks; ++c) {
          if (c % kOzBlockChunks == 0) {  // a K-block begins with empty accumulators
            if (!tc_wait(&S.tempty, tphase ^ 1, err, abort_flag)) {
              ok = false;
              break;
            }
            tc_fence_after();
          }
          if (!tc_wait(&S.full[stage], phase, err, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = sbase + stage * kOzStage;
          const uint32_t b0 = a0 + kOzAChunk + kOzLow * kOzBBlock;  // B slice 1
          const uint32_t pos = oz_idesc(kOzAccN, false), neg = oz_idesc(kOzAccN, true);
          // slice p + 1 of A into levels 2 + 4 h .. 5 + 4 h: B slices 4 h - p + 1 .. 4 h - p + 4,
          // those outside 1..7 zeros
          auto products = [&](int p, int h, uint32_t acc) {
            const uint32_t dr = tmem + h * kOzAccN, di = dr + kOzIm;
            const uint64_t a_re = oz_desc(a0 + p * kOzABlock);
            const uint64_t a_im = oz_desc(a0 + p * kOzABlock + 32);
            const uint64_t b_re = oz_desc(b0 + (4 * h - p) * kOzBBlock);
            const uint64_t b_im = oz_desc(b0 + (4 * h - p) * kOzBBlock + 32);
            mma_bf16(dr, a_re, b_re, pos, acc);
            mma_bf16(di, a_re, b_im, pos, acc);
            mma_bf16(dr, a_im, b_im, neg, 1u);
            mma_bf16(di, a_im, b_re, pos, 1u);
          };
          static_assert(kOzLow >= 3 && 4 + kOzLow >= kOzSlices && 8 - kOzSlices <= kOzHigh,
                        "every block of an accumulator lies in the stage");
          const uint32_t more = c % kOzBlockChunks == 0 ? 0u : 1u;
#pragma unroll
          for (int p = 0; p < 4; ++p) products(p, 0, p == 0 ? more : 1u);
#pragma unroll
          for (int p = 0; p < kOzSlices; ++p) products(p, 1, p == 0 ? more : 1u);
          mma_commit(&S.empty[stage]);
          if (++stage == kOzStages) {
            stage = 0;
            phase ^= 1;
          }
          if (c % kOzBlockChunks == kOzBlockChunks - 1 || c + 1 == chunks) {
            mma_commit(&S.tfull);
            tphase ^= 1;
          }
        }
        if (!ok) break;
      }
    }
  } else {
    // ------------------------------------------------ epilogue (warps 2..9)
    // warp w reads TMEM lanes of quadrant w % 4; warps 2..5 take columns 0..15 of the tile,
    // warps 6..9 columns 16..31
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 16);
    uint32_t tphase = 0;
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
      int inst;
      int64_t mt, nt;
      oz_coords(S, insts, ninst, t, &inst, &mt, &nt);
      const OzGemmInst& G = insts[inst];
      const int64_t gr = mt * kOzM + row;
      const int64_t gc = nt * kOzN + half * 16;
      const int ncol = gr < G.m ? (int)max((int64_t)0, min((int64_t)16, G.n - gc)) : 0;
      double2* C = static_cast<double2*>(G.c) + (G.c_r0 + gr) + (G.c_c0 + gc) * G.ldc;
      const int64_t as = (G.m + kOzM - 1) / kOzM * kOzM, bs = (G.n + kOzN - 1) / kOzN * kOzN;
      const int blocks = (G.kk + kOzK - 1) / kOzK;
      bool gone = false;
      for (int kb = 0; kb < blocks; ++kb) {
        const int32_t er = gr < G.m ? G.aexp[kb * as + gr] : kOzNone;
        const int32_t* be = G.bexp + kb * bs;
        const bool ok = tc_wait(&S.tfull, tphase, err, abort_flag);
        if (!__all_sync(0xffffffffu, ok)) {
          gone = true;
          break;
        }
        tc_fence_after();
        tphase ^= 1;
        long long v[2][16];
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            float f[kOzLevels][8];
#pragma unroll
            for (int d = 0; d < kOzLevels; ++d)
              tmem_ld8(tl + part * kOzIm + (uint32_t)(d * kOzN + g * 8), f[d]);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              // levels 2..4 in units of 2^-32, levels 5..9 in units of 2^-64, sum in 2^-56
              const long long h = (long long)__float2int_rn(f[0][j]) * 65536 +
                                  (long long)__float2int_rn(f[1][j]) * 256 +
                                  (long long)__float2int_rn(f[2][j]);
              const long long l = (long long)__float2int_rn(f[3][j]) * 16777216 +
                                  (long long)__float2int_rn(f[4][j]) * 65536 +
                                  (long long)__float2int_rn(f[5][j]) * 256 +
                                  (long long)(__float2int_rn(f[6][j]) +
                                              ((__float2int_rn(f[7][j]) + 128) >> 8));
              v[part][g * 8 + j] = (h << 24) + ((l + 128) >> 8);
            }
          }
        tc_fence_before();
        mbar_arrive(&S.tempty);
        double2 x[16];  // every load in flight before the first store
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < ncol) x[j] = C[(int64_t)j * G.ldc];
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < ncol) {
            const int32_t ec = be[gc + j];
            if (er == kOzNaN || ec == kOzNaN) {
              x[j].x = x[j].y = __longlong_as_double(0x7FF8000000000000LL);
            } else {
              x[j].x -= oz_scaled(v[0][j], er + ec - 56);
              x[j].y -= oz_scaled(v[1][j], er + ec - 56);
            }
            C[(int64_t)j * G.ldc] = x[j];
          }
      }
      if (gone) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kOzTmem)
                 : "memory");
  }
}

// ------------------------------------------------------------------ host side
size_t oz_pack_bytes(int64_t rows, int kk, OzSide side) {
  const int64_t t = side == kOzA ? kOzM : kOzN;
  const int64_t chunk = side == kOzA ? kOzAChunk : kOzBChunk;
  return (size_t)((rows + t - 1) / t) * ((kk + kOzKC - 1) / kOzKC) * chunk;
}
size_t oz_exps(int64_t rows, OzSide side) {
  const int64_t t = side == kOzA ? kOzM : kOzN;
  return (size_t)((rows + t - 1) / t) * t;
}
int64_t oz_tiles(int64_t m, int64_t n) {
  return m > 0 && n > 0 ? ((m + kOzM - 1) / kOzM) * ((n + kOzN - 1) / kOzN) : 0;
}

void launch_oz_kexp(const Launch& L, const OzPackInst* d, int ninst, int64_t max_rows, int max_kk) {
  if (ninst <= 0 || max_rows <= 0 || max_kk <= 0) return;
  k_oz_kexp<<<dim3((unsigned)((max_rows + kKexpRows - 1) / kKexpRows), (unsigned)ninst), 256, 0,
              L.stream>>>(d);
  count_launch(1);
}

void launch_oz_pack(const Launch& L, const OzPackInst* d, int ninst, int64_t max_rows, int max_kk,
                    OzSide side, bool single) {
  if (ninst <= 0 || max_rows <= 0 || max_kk <= 0) return;
  const int64_t t = side == kOzA ? kOzM : kOzN;
  const dim3 grid((unsigned)((max_rows + t - 1) / t * 4), (unsigned)ninst,
                  (unsigned)((max_kk + kOzK - 1) / kOzK));
  if (side == kOzA) {
    if (single)
      k_oz_pack<float2, kOzM, kOzM / 4, false><<<grid, 256, 0, L.stream>>>(d);
    else
      k_oz_pack<double2, kOzM, kOzM / 4, false><<<grid, 256, 0, L.stream>>>(d);
  } else {
    k_oz_pack<double2, kOzN, kOzN / 4, true><<<grid, 256, 0, L.stream>>>(d);
  }
  count_launch(1);
}

void launch_oz_gemm(const Launch& L, const OzGemmInst* d, int ninst, const int64_t* tiles) {
  const size_t smem = 1024 + kOzStages * kOzStage + sizeof(OzShared);
  static PerDeviceOnce attr;
  attr.call([&] {
    cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  });
  for (int i0 = 0; i0 < ninst; i0 += kOzMaxInst) {
    const int n = std::min(kOzMaxInst, ninst - i0);
    int64_t total = 0;
    for (int i = 0; i < n; ++i) total += tiles[i0 + i];
    if (total <= 0) continue;
    const int64_t sms = device_sm_count();
    k_oz_gemm<<<(unsigned)std::min(total, sms), kOzThreads, smem, L.stream>>>(d + i0, n, L.err_flag);
    count_launch(1);
  }
}

}  // namespace bemgpu
