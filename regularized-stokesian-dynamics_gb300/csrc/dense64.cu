// FP64 dense factorisations on the tensor cores: Cholesky (DPOTRF 'U'),
// inverse from the factor (DPOTRI 'U') and triangular solves for the grand
// resistance (MATREV, src/matrices.f90:4-34).
//
// GB300's FP64 pipe makes 2 multiply-adds per SM and cycle (1.2 TFLOP/s in
// all), so products of FP64 matrices are formed from integers on the bf16
// tensor cores instead (the error-free splitting of K. Ozaki, T. Ogita, S.
// Oishi and S. M. Rump, Numer. Algorithms 59, 2012):
//   - an operand column is scaled by a power of two to |x| < 1, rounded to
//     56 bits and cut into 7 signed base-256 digits (-128..128), each exact
//     in bf16 (oz_split); where the terms of a sum pair a small factor with a
//     large one (U^-1 against U), k is scaled by a power of two too;
//   - digit products are integers of at most 2^14; those of one weight s = i
//     + j are summed in one FP32 accumulator of tensor memory, exactly: K =
//     128 of them in up to 7 pairs stay below 2^24 (oz_gemm);
//   - every 128 of K the 8 accumulators (s = 0..7) are added into two 64-bit
//     integers per output, which become one FP64 value at the end.
// Of a term x y, |x|, |y| < 1, the weights left out (s = 8..12) come to less
// than 2^-61, and the entries' roundings to at most 2^-56 (|x| + |y|), none
// for entries within a factor of 4 of the largest; there is no rounding in the
// sum.  (With s = 7 left out too it was up to 2^-53.4 a term, 2^-56.3 in the
// mean, and residuals of well-conditioned inverses three times those of FP64
// multiply-adds.)  So a product is off by at most about 2^-54 of its columns'
// largest entries per term: normwise what a chain of FP64 multiply-adds may be off, not
// entry by entry, which is why the ill-conditioned solves and inverses below do
// not multiply by inverses.
//
// Layout: both operands are K-major (K contiguous), split beforehand into
// slices [digit][batch][column][K] of bf16; C(r, c) = sum_k R(k, r) S(k, c).
//
//   potrf   right-looking, 64 columns a step: the diagonal block and its
//           inverse in one CTA (potf2_inv_f64), the row panel by substitution
//           (subst64) and the updates P^T P as oz_gemm, of the outer panel's
//           256 rows after each step and of the rest once per outer panel (a
//           tile's last step, its FP64 additions, costs as much as 128 of K)
//   trsm64  solves for many right-hand sides, 128 unknowns a step by
//           substitution, the updates as oz_gemm
//   potri   U^-1 by recursive doubling of the diagonal inverses (all pairs of
//           a level in one batched launch) or by trsm64 on the identity, then
//           U^-1 U^-T as one product
//   trsv    block substitution for a few right-hand sides, one launch a step
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>

#include "pdl.cuh"
#include "rsd_internal.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int OZ_S = 7, OZ_W = 8;           // digits, and weights kept of their products
constexpr int OZ_TC = 128, OZ_TR = 64;      // columns and rows of a C tile (MMA M and N)
constexpr int OZ_KC = 32;                   // K of a stage: 64-byte rows, 64-byte swizzle
constexpr int OZ_GROUP = 4;                 // stages between two drains: K = 128
constexpr int OZ_A = OZ_TC * OZ_KC * 2, OZ_B = OZ_TR * OZ_KC * 2;
constexpr int OZ_STAGES = 2, OZ_STAGE = OZ_S * (OZ_A + OZ_B);
constexpr int OZ_SMEM = OZ_STAGES * OZ_STAGE + 1024 + 128;
constexpr int OZ_THREADS = 320;             // TMA, MMA, 8 drain warps
constexpr int OZ_TMEM = OZ_W * OZ_TR;
constexpr int OZ_NONFINITE = 1 << 20;       // exponent of a column that holds an infinity or a NaN
constexpr int OZ_ZERO = -(1 << 20);
constexpr unsigned long long OZ_WAIT_NS = 500ull * 1000 * 1000;
constexpr int NB64 = 64;                    // panel width of the factorisation
constexpr int NBO64 = 256;                  // rows between two updates of the whole trailing matrix
constexpr int NBS64 = 128;                  // unknowns a step of the solves with many right-hand sides
constexpr int GROWTH64 = 3;                 // largest exponent of a scaled inverse factor for the fast inverse

// ------------------------------------------------------------------ split
// Batch z: X + z sX, columns beyond cn - z cstep and K beyond kn - z kstep
// are zero (the ragged last pair of a level).  trans: entry (k, c) at X[c + k
// ld] instead of X[k + c ld].  tri: only k <= c (trans: c <= k) is stored.
// ks: entry (k, c) of batch z is taken times 2^(ksgn ks[k + z kstride]).
struct oz_split_job {
  const int* ks;
  int ksgn, kstride;
  const double* X;
  int64_t ld, sX;
  int K, cols, nb, trans, tri;
  int kn, kstep, cn, cstep;
  __nv_bfloat16* D;
  int* E;
  int Kld;
};

__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// exponent field of x times 2^sh; OZ_ZERO for zero, OZ_NONFINITE
__device__ __forceinline__ int oz_field(double x, int sh) {
  const unsigned long long b = abs_bits(x);
  const int E = (int)(b >> 52);
  return b == 0 ? OZ_ZERO : (E == 0x7ff ? OZ_NONFINITE : (E ? E : 1) + sh);
}

// x 2^sh scaled to |x| < 2^55 by the column's largest exponent field, rounded
__device__ __forceinline__ long long oz_fixed(double x, int sh, int emax) {
  const unsigned long long b = abs_bits(x);
  if (b == 0) return 0;
  const int E = (int)(b >> 52);
  unsigned long long m = (b & 0xfffffffffffffull) | (E ? 0x10000000000000ull : 0ull);
  const int k = (E ? E : 1) + sh - emax + 2;
  if (k >= 0)
    m <<= min(k, 2);
  else
    m = k > -56 ? (m + (1ull << (-k - 1))) >> -k : 0ull;
  return __double_as_longlong(x) < 0 ? -(long long)m : (long long)m;
}

__device__ __forceinline__ void oz_digits(long long q, int (&d)[OZ_S]) {
#pragma unroll
  for (int i = OZ_S - 1; i > 0; i--) {
    const int t = (int)((q + 128) & 255) - 128;
    d[i] = t;
    q = (q - t) >> 8;
  }
  d[0] = (int)q;
}

__device__ __forceinline__ int oz_shift(const oz_split_job& J, int z, int k) {
  return J.ks && k < min(J.K, J.kn - z * J.kstep) ? J.ksgn * J.ks[k + z * J.kstride] : 0;
}

__device__ __forceinline__ void oz_store2(const oz_split_job& J, int z, int c, int k, double x0, double x1, int emax) {
  int d0[OZ_S], d1[OZ_S];
  oz_digits(oz_fixed(x0, oz_shift(J, z, k), emax), d0);
  oz_digits(oz_fixed(x1, oz_shift(J, z, k + 1), emax), d1);
#pragma unroll
  for (int i = 0; i < OZ_S; i++) {
    __nv_bfloat162 v;
    v.x = __float2bfloat16_rn((float)d0[i]);
    v.y = __float2bfloat16_rn((float)d1[i]);
    *reinterpret_cast<__nv_bfloat162*>(J.D + ((int64_t)(i * J.nb + z) * J.cols + c) * J.Kld + k) = v;
  }
}

// |x| < 2^exponent for a column whose largest field is f
__device__ __forceinline__ int oz_exponent(int f) {
  return f == OZ_NONFINITE ? f : (f == OZ_ZERO ? 0 : f - 1022);
}

constexpr int SPLIT_THREADS = 256, SPLIT_COLS = 8, SPLIT_TCOLS = 32;

// Both operands of a product in one launch (blockIdx.y).  K-contiguous input:
// a warp per column, two passes; otherwise 32 columns per CTA through shared
// memory, so that reads and writes stay coalesced.  Integer arithmetic on the
// bits throughout: the FP64 pipe would bound it.
__global__ void __launch_bounds__(SPLIT_THREADS) oz_split(oz_split_job J0, oz_split_job J1) {
  pdl_enter();
  const oz_split_job& J = blockIdx.y ? J1 : J0;
  const int z = blockIdx.z, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (z >= J.nb) return;
  const double* X = J.X + z * J.sX;
  const int Kv = min(J.K, J.kn - z * J.kstep), Cv = min(J.cols, J.cn - z * J.cstep);
  if (!J.trans) {
    const int c = blockIdx.x * SPLIT_COLS + warp;
    if (c >= J.cols) return;
    const int kv = c < Cv ? (J.tri ? min(Kv, c + 1) : Kv) : 0;
    const double* x = X + (int64_t)c * J.ld;
    int m = OZ_ZERO;
    for (int k = lane; k < kv; k += 32) m = max(m, oz_field(x[k], oz_shift(J, z, k)));
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) J.E[z * J.cols + c] = oz_exponent(m);
    for (int k = 2 * lane; k < J.Kld; k += 64)
      oz_store2(J, z, c, k, k < kv ? x[k] : 0.0, k + 1 < kv ? x[k + 1] : 0.0, m);
  } else {
    __shared__ int red[8][SPLIT_TCOLS];
    __shared__ double tile[64][SPLIT_TCOLS + 1];
    const int c0 = blockIdx.x * SPLIT_TCOLS, c = c0 + lane;
    if (c0 >= J.cols) return;
    auto at = [&](int k) { return c < Cv && k < Kv && (!J.tri || c <= k) ? X[c + (int64_t)k * J.ld] : 0.0; };
    int m = OZ_ZERO;
#pragma unroll 4
    for (int k = warp; k < Kv; k += 8) m = max(m, oz_field(at(k), oz_shift(J, z, k)));
    red[warp][lane] = m;
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int w = 1; w < 8; w++) m = max(m, red[w][lane]);
      red[0][lane] = m;
      if (c < J.cols) J.E[z * J.cols + c] = oz_exponent(m);
    }
    __syncthreads();
    for (int k0 = 0; k0 < J.Kld; k0 += 64) {
#pragma unroll
      for (int q = 0; q < 8; q++) tile[warp + 8 * q][lane] = at(k0 + warp + 8 * q);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int cc = 4 * warp + q;
        if (c0 + cc < J.cols && k0 + 2 * lane < J.Kld)
          oz_store2(J, z, c0 + cc, k0 + 2 * lane, tile[2 * lane][cc], tile[2 * lane + 1][cc],
                    red[0][cc]);
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------- product
struct oz_args {
  int K;            // K extent
  int m, n;         // rows and columns of C
  int ncap, nstep;  // batch z has min(n, ncap - z nstep) columns
  int tri;          // skip the tiles strictly below the diagonal
  int klo_row, klo_col, khi_col;  // K starts at the tile's first row / column, ends with its last column
  int add;          // 1: C += the product, 0: C = the product
  int neg;          // the product is taken times -1
  const int* gate;  // no product above GROWTH64
  double* C;
  int64_t ld, sC;
  const int *ER, *ES;  // exponents of R's and S's columns
  int rcols, scols;    // columns per batch in the slices
  int nb;
  int* err;
  unsigned long long wait_ns;
};

__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
  // K-major, 64-byte swizzle: rows of 64 B, 8-row groups 512 B apart
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

// kind::f16 with bf16 operands and FP32 accumulation, M = 128, both K-major
__device__ __forceinline__ void mma_bf16(uint32_t d, uint32_t a, uint32_t b, int N, uint32_t acc) {
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(OZ_TC >> 4) << 24);
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(desc_sw64(a)), "l"(desc_sw64(b)), "r"(idesc), "r"(acc));
}

// sgn (hi + lo 2^-32) 2^e, rounded to nearest, with integer operations (two
// 64-bit conversions and a scaling would take the FP64 pipe ~27 cycles per
// output and SM lane pair; 2 per cycle and SM is all it does)
__device__ __forceinline__ double oz_value(long long hi, long long lo, int e, unsigned long long sgn) {
  unsigned long long L = (unsigned long long)hi << 32;
  long long H = (hi >> 32) + (lo >> 63);
  L += (unsigned long long)lo;
  H += L < (unsigned long long)lo;
  if (H < 0) {  // magnitude; the sign goes into the result's bits
    sgn ^= 0x8000000000000000ull;
    L = ~L + 1ull;
    H = ~H + (L == 0);
  }
  unsigned long long m;
  int p;
  if (H) {
    const int lz = __clzll(H);  // 0 < H < 2^32: 31 < lz < 64
    m = (unsigned long long)H << lz | L >> (64 - lz);
    p = 127 - lz;
  } else {
    const int lz = L ? __clzll((long long)L) : 0;
    m = L << lz;
    p = 63 - lz;
  }
  const int E = p + e - 32 + 1023;
  unsigned long long r = (m >> 11) + ((m >> 10) & 1);  // 53 bits, the leading one counts into the exponent
  if (m == 0) return __longlong_as_double((long long)sgn);
  if (E < 1 || E > 2046) {  // out of FP64's normal range
    const double v = ldexp((double)r, p - 52 + e - 32);
    return sgn >> 63 ? -v : v;
  }
  return __longlong_as_double((long long)(((unsigned long long)(E - 1) << 52) + r) ^ (long long)sgn);
}

#define OZ_LD16(v, addr)                                                                                              \
  asm volatile(                                                                                                       \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "     \
      "%15}, [%16];"                                                                                                  \
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),   \
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])                      \
      : "r"(addr))

// One 64 x 128 tile of C per CTA (the MMA's M is C's columns, so that a
// thread of the epilogue owns 32 consecutive rows of one column).  The digit
// slices of R lie one after another in shared memory, so one MMA multiplies
// digit i of S with several digits of R at once: its N columns land in the
// accumulators s = i, i + 1, ... which are neighbours in tensor memory.
// Bound: 8 x 1088 cycles of MMA per K = 128, then the drain (8 x 8192 values
// into integers) and, once per tile, the conversion (~40 integer
// instructions) and an FP64 addition per output.  Measured in the FP64 step
// at N = 512 (factor of order 5632, inverse and factor of 3072): 9.5 ms of
// products where the FP64 pipe took 348 ms for the reference's full inverse;
// with 64-bit conversions and a scaling on the FP64 pipe instead of oz_value
// 26.4 ms, and with an update of the whole trailing matrix every 64 columns
// 65 ms.
__global__ void __launch_bounds__(OZ_THREADS, 1) oz_gemm(const __grid_constant__ CUtensorMap tmS,
                                                         const __grid_constant__ CUtensorMap tmR, const oz_args a) {
  pdl_enter();
  const int row0 = blockIdx.x * OZ_TR, col0 = blockIdx.y * OZ_TC, z = blockIdx.z;
  const int nz = min(a.n, a.ncap - z * a.nstep);
  if (col0 >= nz || (a.tri && row0 > col0 + OZ_TC - 1) || (a.gate && *a.gate > GROWTH64)) return;
  int klo = 0, khi = a.K;
  if (a.klo_row) klo = max(klo, row0);
  if (a.klo_col) klo = max(klo, col0);
  klo &= ~(OZ_KC - 1);
  if (a.khi_col) khi = min(khi, col0 + OZ_TC);
  const int nch = khi > klo ? (khi - klo + OZ_KC - 1) / OZ_KC : 0;

  extern __shared__ unsigned char smraw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t bars[2 * OZ_STAGES + 2];
  __shared__ uint32_t tslot;
  __shared__ volatile int abort_flag;
  __shared__ int rexp[OZ_TR];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const uint32_t sbase = smem_u32(base), bar0 = smem_u32(bars);
#define OZ_FULL(s) (bar0 + 8u * (uint32_t)(s))
#define OZ_EMPTY(s) (bar0 + 8u * (uint32_t)(OZ_STAGES + (s)))
  const uint32_t accfull = bar0 + 8u * (2 * OZ_STAGES), accempty = accfull + 8u;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tslot)),
                 "r"(OZ_TMEM));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 32) {
    for (int s = 0; s < OZ_STAGES; s++) {
      mbar_init(OZ_FULL(s), 1);
      mbar_init(OZ_EMPTY(s), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, 256);
    asm volatile("fence.mbarrier_init.release.cluster;");
    abort_flag = 0;
  }
  if (t >= 64 && t < 64 + OZ_TR) {
    const int r = row0 + t - 64;
    rexp[t - 64] = r < a.m ? a.ER[z * a.rcols + r] : 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t taddr = tslot;

  if (warp == 0) {
    if (lane == 0) {  // TMA producer
      int last[OZ_STAGES];
      for (int s = 0; s < OZ_STAGES; s++) last[s] = -1;
      for (int c = 0; c < nch; c++) {
        const int s = c % OZ_STAGES;
        if (c >= OZ_STAGES && !mbar_wait(OZ_EMPTY(s), ((c / OZ_STAGES) - 1) & 1, &abort_flag, a.err, 21, a.wait_ns))
          break;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(OZ_FULL(s)), "r"(OZ_STAGE)
                     : "memory");
        const uint32_t st = sbase + s * OZ_STAGE;
        const int k = klo + c * OZ_KC;
        for (int i = 0; i < OZ_S; i++) tma_load(st + i * OZ_A, &tmS, k, (i * a.nb + z) * a.scols + col0, OZ_FULL(s));
        for (int i = 0; i < OZ_S; i++)
          tma_load(st + OZ_S * OZ_A + i * OZ_B, &tmR, k, (i * a.nb + z) * a.rcols + row0, OZ_FULL(s));
        last[s] = c;
      }
      if (abort_flag) {  // let the copies already issued land before the CTA exits
        for (int s = 0; s < OZ_STAGES; s++)
          if (last[s] >= 0) {
            const uint64_t t0 = global_ns();
            while (!mbar_try_wait(OZ_FULL(s), (last[s] / OZ_STAGES) & 1) && global_ns() - t0 < OZ_WAIT_NS) {
            }
          }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      int issued = 0;
      for (int c = 0; c < nch; c++) {
        const int s = c % OZ_STAGES, g = c / OZ_GROUP;
        if (c % OZ_GROUP == 0 && g > 0) {
          if (!mbar_wait(accempty, (g - 1) & 1, &abort_flag, a.err, 22, a.wait_ns)) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
        }
        if (!mbar_wait(OZ_FULL(s), (c / OZ_STAGES) & 1, &abort_flag, a.err, 23, a.wait_ns)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t st = sbase + s * OZ_STAGE, sr = st + OZ_S * OZ_A;
#pragma unroll
        for (int kk = 0; kk < OZ_KC / 16; kk++) {
          const uint32_t first = (c % OZ_GROUP == 0 && kk == 0) ? 0u : 1u;
#pragma unroll
          for (int i = 0; i < OZ_S; i++) {
            const int w = min(OZ_S, OZ_W - i);  // digits 0..w-1 of R
            const uint32_t sa = st + i * OZ_A + kk * 32, sb = sr + kk * 32, acc = i == 0 ? first : 1u;
            mma_bf16(taddr + i * OZ_TR, sa, sb, OZ_TR * min(w, 4), acc);
            if (i == 1) {  // the first of weight 7
              mma_bf16(taddr + 5 * OZ_TR, sa, sb + 4 * OZ_B, OZ_TR * 2, 1u);
              mma_bf16(taddr + 7 * OZ_TR, sa, sb + 6 * OZ_B, OZ_TR, first);
            } else if (w > 4) {
              mma_bf16(taddr + (i + 4) * OZ_TR, sa, sb + 4 * OZ_B, OZ_TR * (w - 4), acc);
            }
          }
        }
        mma_commit(OZ_EMPTY(s));
        issued = 1;
        if (c % OZ_GROUP == OZ_GROUP - 1 || c == nch - 1) mma_commit(accfull);
      }
      if (abort_flag && issued) {  // the tensor memory is not freed under MMAs still running
        mma_commit(accfull);
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) {
        }
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;  // TMEM lanes 32q.., rows 32 half.. of the tile
    const int ngrp = (nch + OZ_GROUP - 1) / OZ_GROUP;
    long long hi[32], lo[32];
#pragma unroll
    for (int j = 0; j < 32; j++) hi[j] = lo[j] = 0;
    const uint32_t lane_addr = taddr + ((uint32_t)(32 * q) << 16) + 32 * half;
    bool ok = true;
    for (int g = 0; g < ngrp && ok; g++) {
      ok = __all_sync(0xffffffffu, mbar_wait(accfull, g & 1, &abort_flag, a.err, 24, a.wait_ns) ? 1 : 0) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int s = 0; s < OZ_W; s++) {
#pragma unroll
        for (int jh = 0; jh < 32; jh += 16) {
          uint32_t v[16];
          OZ_LD16(v, lane_addr + s * OZ_TR + jh);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const int d = __float2int_rn(__uint_as_float(v[j]));
            if (s < 4)
              hi[jh + j] += (long long)d * (1 << (8 * (3 - s)));
            else
              lo[jh + j] += (long long)d * (1 << (8 * (7 - s)));
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(accempty) : "memory");
    }
    const int c = col0 + 32 * q + lane;
    if (ok && !abort_flag && c < nz) {
      const int e = a.ES[z * a.scols + c];
      double* C = a.C + z * a.sC + (int64_t)c * a.ld + row0 + 32 * half;
      const int nr = min(32, a.m - row0 - 32 * half);
      const unsigned long long sgn = a.neg ? 0x8000000000000000ull : 0ull;
      auto value = [&](int j) {
        const int er = rexp[32 * half + j];
        return max(e, er) == OZ_NONFINITE ? __longlong_as_double(0x7ff8000000000000ll)
                                          : oz_value(hi[j], lo[j], e + er - 38, sgn);
      };
      if (a.add) {
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 8) {  // eight loads in flight
          double old[8];
#pragma unroll
          for (int j = 0; j < 8; j++) old[j] = j0 + j < nr ? C[j0 + j] : 0.0;
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (j0 + j < nr) C[j0 + j] = old[j] + value(j0 + j);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; j++)
          if (j < nr) C[j] = value(j);
      }
    }
  }
#undef OZ_FULL
#undef OZ_EMPTY
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(OZ_TMEM));
  }
}

// -------------------------------------------------------- diagonal block
// A jb x jb diagonal block (jb <= 64; padded with the identity): the upper
// Cholesky factor U in place and W = U^-1 (64 x 64, column-major, zero below
// the diagonal), in one CTA.  Gauss-Jordan on [S | I]: step k subtracts l_ik =
// S_ki / d_k times row k from every row i > k, of S (columns j >= i) and of
// the inverse of the unit lower factor that grows in the place of the
// eliminated part (columns j <= k), so one 64 x 64 array holds both and a
// step is two FP64 warp instructions per row.  Warp 0 takes row k + 1 first,
// then the next pivot's reciprocal and multipliers beside the other rows, so
// a step has one barrier.  Bound by the FP64 pipe (64 cycles per warp
// instruction and SM quarter): 62 us a block, 67 with the roots taken where
// they are stored and the pivot tested in FP64, 96 with one row in flight per
// warp; a column-by-column factor and inverse of 128 took 263 + 466 us.
// info: first failing global index + 1.
constexpr int PF_LD = NB64 + 1;
__device__ __forceinline__ int half_exponent(double d) {
  const int E = (int)(abs_bits(d) >> 52);
  return E == 0 || E == 0x7ff ? 0 : (E - 1023) >> 1;
}
__global__ void diag_exponents(int n, const double* __restrict__ A, int64_t lda, int* __restrict__ e) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) e[i] = half_exponent(A[i + (int64_t)i * lda]);
}
__global__ void __launch_bounds__(256) potf2_inv_f64(double* __restrict__ A, int64_t lda, int jb,
                                                     int* __restrict__ info, int j0, double* __restrict__ Wout) {
  pdl_enter();
  __shared__ double S[NB64 * PF_LD];  // S(i, j) at [i * PF_LD + j]
  __shared__ double l[2][NB64], sq[NB64], rd[NB64];
  __shared__ int failed[2];  // pivot k's verdict in [k & 1]: read in step k, while the next one is made
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int e = t; e < NB64 * NB64; e += 256) {
    const int i = e % NB64, j = e / NB64;
    S[i * PF_LD + j] = i <= j && j < jb ? A[i + (int64_t)j * lda] : (i == j ? 1.0 : 0.0);
  }
  if (t < 2) failed[t] = 0;
  __syncthreads();
  // multipliers l_ik of pivot k (d its value) into l[k & 1]
  auto pivot = [&](int k, double d) {
    const long long bits = __double_as_longlong(d);  // positive and finite, off the FP64 pipe
    if (bits <= 0 || bits >= 0x7ff0000000000000LL) {
      if (lane == 0) {
        failed[k & 1] = 1;
        atomicCAS(info, 0, j0 + k + 1);
      }
      return;
    }
    const double r = __drcp_rn(d);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = lane + 32 * h;
      if (i > k) l[k & 1][i] = S[k * PF_LD + i] * r;
    }
  };
  if (warp == 0) pivot(0, S[0]);
  __syncthreads();
  for (int k = 0; k < NB64 - 1; k++) {
    if (failed[k & 1]) return;
    const double* lk = l[k & 1];
    // row k; in column k the identity enters: 0 - l_ik 1
    const double s0 = lane == k ? 1.0 : S[k * PF_LD + lane], s1 = lane + 32 == k ? 1.0 : S[k * PF_LD + lane + 32];
    // Q rows i, i + step, ... in flight
    auto rows = [&](auto q, int i0, int step) {
      constexpr int Q = decltype(q)::value;
      double x0[Q], x1[Q], li[Q];
#pragma unroll
      for (int u = 0; u < Q; u++) {
        const int i = i0 + u * step;
        if (i < NB64) {
          li[u] = -lk[i];
          x0[u] = lane == k ? 0.0 : S[i * PF_LD + lane];
          x1[u] = lane + 32 == k ? 0.0 : S[i * PF_LD + lane + 32];
        }
      }
#pragma unroll
      for (int u = 0; u < Q; u++) {
        const int i = i0 + u * step;
        if (i < NB64) {
          if (lane <= k || lane >= i) S[i * PF_LD + lane] = fma(li[u], s0, x0[u]);
          if (lane + 32 <= k || lane + 32 >= i) S[i * PF_LD + lane + 32] = fma(li[u], s1, x1[u]);
        }
      }
    };
    if (warp == 0) {
      const double d = fma(-lk[k + 1], S[k * PF_LD + k + 1], S[(k + 1) * PF_LD + k + 1]);
      rows(std::integral_constant<int, 1>{}, k + 1, 1);
      pivot(k + 1, d);
    } else {
      for (int i = k + 1 + warp; i < NB64; i += 28) rows(std::integral_constant<int, 4>{}, i, 7);
    }
    __syncthreads();
  }
  if (failed[(NB64 - 1) & 1]) return;
  if (t < NB64) {
    sq[t] = sqrt(S[t * PF_LD + t]);
    rd[t] = 1.0 / sq[t];
  }
  __syncthreads();
  // U_kj = S_kj / sqrt(d_k); W_ij = (L^-1)_ji / sqrt(d_j) with unit diagonal
  for (int e = t; e < NB64 * NB64; e += 256) {
    const int i = e % NB64, j = e / NB64;
    if (i <= j && j < jb) A[i + (int64_t)j * lda] = i == j ? sq[i] : S[i * PF_LD + j] * rd[i];
    Wout[e] = i < j ? S[j * PF_LD + i] * rd[j] : (i == j ? rd[j] : 0.0);
  }
}

// ------------------------------------------------ substitution, many systems
// Solves against a w-wide diagonal block U (w <= W) on the FP64 pipe, in place:
// U^T x = b, or U x = b (BACK), the entries of system q at B[i + q ldb].  Through
// the block's explicit inverse the residual would grow by the condition number
// of the block (factor of stiff pairs at 1e8: 4600 eps of the scaled matrix, 8
// so).  16 lanes per system; with U's entries divided by the pivot of their step
// a step is a broadcast and at most W / 16 multiply-adds, and the unknowns are
// scaled at the end.  Bound by the chain of steps and the FP64 pipe (64 cycles per
// warp instruction and SM quarter): 22.5 us for 64 to 640 systems of 64, 27 for
// 2100 (from cold; 34 for 2600 with one load of U in flight per thread).
// The reciprocals of the diagonal come from the 64-wide inverses in Wd.
constexpr int SUB_SYS = 8, SUB_THREADS = 16 * SUB_SYS;
template <int W>
constexpr int SUB_SMEM = (W * (W + 1) + W) * (int)sizeof(double);
template <int W, bool BACK>
__global__ void __launch_bounds__(SUB_THREADS) subst64(int w, const double* __restrict__ U, int64_t ldu,
                                                       const double* __restrict__ Wd, int nsys, double* __restrict__ B,
                                                       int64_t ldb) {
  pdl_enter();
  constexpr int R = W / 16, LD = W + 1;
  extern __shared__ __align__(16) double sub_smem[];
  // step k takes unknown at(k); S(k, i): U's entry of step k and unknown at(i) by the pivot of step k, k < i
  double *S = sub_smem, *rd = S + W * LD;
  const int t = threadIdx.x, l = t & 15, q = blockIdx.x * SUB_SYS + (t >> 4);
  auto at = [](int i) { return BACK ? W - 1 - i : i; };
  double* Bq = B + (int64_t)q * ldb;
  if (t < W) rd[t] = at(t) < w ? Wd[(at(t) / NB64) * NB64 * NB64 + (at(t) % NB64) * (NB64 + 1)] : 1.0;
  double b[R];
#pragma unroll
  for (int j = 0; j < R; j++) b[j] = q < nsys && at(l + 16 * j) < w ? Bq[at(l + 16 * j)] : 0.0;
  __syncthreads();
  for (int e0 = t; e0 < W * W; e0 += 16 * SUB_THREADS) {  // U(r, c), r < c, by columns, 16 loads in flight
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const int e = e0 + u * SUB_THREADS, r = e % W, c = e / W;
      v[u] = r < c && c < w ? U[r + (int64_t)c * ldu] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const int e = e0 + u * SUB_THREADS, r = e % W, c = e / W, k = BACK ? at(c) : r, i = BACK ? at(r) : c;
      if (r < c) S[k * LD + i] = v[u] * rd[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int kb = 0; kb < R; kb++)
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      const double x = __shfl_sync(0xffffffffu, b[kb], kk, 16);
      const double* s = S + (16 * kb + kk) * LD + l;
      if (kk < 15 && l > kk) b[kb] = fma(-s[16 * kb], x, b[kb]);
#pragma unroll
      for (int j = kb + 1; j < R; j++) b[j] = fma(-s[16 * j], x, b[j]);
    }
#pragma unroll
  for (int j = 0; j < R; j++)
    if (q < nsys && at(l + 16 * j) < w) Bq[at(l + 16 * j)] = b[j] * rd[l + 16 * j];
}

// ------------------------------------------------------- substitution steps
// Forward step b of U^T y = x: every CTA forms y_b = W_b^T x_b, the first one
// stores it, and each updates its columns, x_c -= U(b, c)^T y_b.
template <int NR>
__global__ void __launch_bounds__(256) trsv64_fwd(int n, int b, const double* __restrict__ U, int64_t ldu,
                                                  const double* __restrict__ W, double* __restrict__ X,
                                                  double* __restrict__ Y, int64_t ldx) {
  pdl_enter();
  __shared__ double x[NR][NB64], y[NR][NB64];
  const int j0 = b * NB64, jb = min(NB64, n - j0), t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int e = t; e < NB64 * NR; e += 256) x[e / NB64][e % NB64] = e % NB64 < jb ? X[j0 + e % NB64 + (e / NB64) * ldx] : 0.0;
  __syncthreads();
  const double* Wb = W + (size_t)b * NB64 * NB64;
  for (int i = warp; i < jb; i += 8) {  // column i of W_b
    const double w0 = Wb[lane + (size_t)i * NB64], w1 = Wb[lane + 32 + (size_t)i * NB64];
#pragma unroll
    for (int r = 0; r < NR; r++) {
      double v = w0 * x[r][lane] + w1 * x[r][lane + 32];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) y[r][i] = v;
    }
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int e = t; e < jb * NR; e += 256) Y[j0 + e % jb + (e / jb) * ldx] = y[e / jb][e % jb];
  for (int c = j0 + jb + blockIdx.x * 8 + warp; c < n; c += gridDim.x * 8) {
    const double* u = U + j0 + (int64_t)c * ldu;  // a full block: jb = 64
    const double u0 = u[lane], u1 = u[lane + 32];
#pragma unroll
    for (int r = 0; r < NR; r++) {
      double v = u0 * y[r][lane] + u1 * y[r][lane + 32];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) X[c + r * ldx] -= v;
    }
  }
}

// Backward step b of U x = y: x_b = W_b y_b (stored by the first CTA), then
// y_i -= U(i, b) x_b for the rows above, a thread per row.
template <int NR>
__global__ void __launch_bounds__(128) trsv64_bwd(int n, int b, const double* __restrict__ U, int64_t ldu,
                                                  const double* __restrict__ W, double* __restrict__ Y,
                                                  double* __restrict__ X, int64_t ldx) {
  pdl_enter();
  __shared__ double x[NR][NB64], y[NR][NB64];
  const int j0 = b * NB64, jb = min(NB64, n - j0), t = threadIdx.x;
  for (int e = t; e < NB64 * NR; e += 128) y[e / NB64][e % NB64] = e % NB64 < jb ? Y[j0 + e % NB64 + (e / NB64) * ldx] : 0.0;
  __syncthreads();
  const double* Wb = W + (size_t)b * NB64 * NB64;
  {  // two threads per row, the columns halved
    const int i = t >> 1, h = t & 1;
    double acc[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) acc[r] = 0.0;
#pragma unroll 8
    for (int k = 32 * h; k < 32 * h + 32; k++) {
      const double w = Wb[i + (size_t)k * NB64];
#pragma unroll
      for (int r = 0; r < NR; r++) acc[r] = fma(w, y[r][k], acc[r]);
    }
#pragma unroll
    for (int r = 0; r < NR; r++) {
      const double v = acc[r] + __shfl_xor_sync(0xffffffffu, acc[r], 1);
      if (h == 0) x[r][i] = v;
    }
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int e = t; e < jb * NR; e += 128) X[j0 + e % jb + (e / jb) * ldx] = x[e / jb][e % jb];
  // 4 threads per row, 16 columns each: rows are few, and each FP64
  // instruction of a warp takes the pipe 64 cycles
  const int part = t & 3;
  for (int i = blockIdx.x * 32 + (t >> 2); i - (t >> 2) < j0; i += gridDim.x * 32) {
    double acc[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) acc[r] = 0.0;
    if (i < j0)
#pragma unroll 8
      for (int k = part; k < jb; k += 4) {
        const double u = U[i + (int64_t)(j0 + k) * ldu];
#pragma unroll
        for (int r = 0; r < NR; r++) acc[r] = fma(u, x[r][k], acc[r]);
      }
#pragma unroll
    for (int r = 0; r < NR; r++) {
      double v = acc[r];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (part == 0 && i < j0) Y[i + r * ldx] -= v;
    }
  }
}

// the NB64 diagonal inverses into the diagonal of V (ld)
__global__ void put_diag64(int n, const double* __restrict__ W, double* __restrict__ V, int64_t ld) {
  pdl_enter();
  const int b = blockIdx.x, j0 = b * NB64, jb = min(NB64, n - j0);
  for (int e = threadIdx.x; e < NB64 * NB64; e += blockDim.x) {
    const int i = e % NB64, j = e / NB64;
    if (i < jb && j < jb) V[j0 + i + (int64_t)(j0 + j) * ld] = W[(size_t)b * NB64 * NB64 + e];
  }
}

__global__ void put_ones64(int n, double* __restrict__ V, int64_t ld) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) V[i + (int64_t)i * ld] = 1.0;
}

// largest exponent of the rows of V (e) scaled by the diagonal (dexp)
__global__ void growth64(int n, const int* __restrict__ e, const int* __restrict__ dexp, int* __restrict__ out) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int g = i < n ? e[i] + dexp[i] : 0;
  g = __reduce_max_sync(0xffffffffu, g);
  if ((threadIdx.x & 31) == 0) atomicMax(out, g);
}

// ------------------------------------------------------------------- host
int oz_init(rsd_ctx* ctx) {
  RSD_TRY(rsd_smem(ctx, oz_gemm, OZ_SMEM));
  RSD_TRY(rsd_smem(ctx, subst64<NBS64, false>, SUB_SMEM<NBS64>));
  return rsd_smem(ctx, subst64<NBS64, true>, SUB_SMEM<NBS64>);
}

// A split operand: nb batches of `cols` columns of K entries each.
struct oz_op {
  __nv_bfloat16* D = nullptr;
  int* E = nullptr;
  int K = 0, Kld = 0, cols = 0, nb = 1;
};

size_t oz_slices(int K, int cols, int nb) {
  return (sizeof(__nv_bfloat16) * (size_t)OZ_S * nb * cols * ((K + 63) / 64 * 64) + 255) & ~(size_t)255;
}
size_t oz_bytes(int K, int cols, int nb) { return oz_slices(K, cols, nb) + sizeof(int) * (size_t)nb * cols; }

int oz_alloc(rsd_ctx* ctx, const char* name, int K, int cols, int nb, oz_op* o) {
  o->K = K;
  o->Kld = (K + 63) / 64 * 64;
  o->cols = cols;
  o->nb = nb;
  const size_t slices = oz_slices(K, cols, nb);
  char* p = (char*)rsd_scratch(ctx, name, oz_bytes(K, cols, nb));
  if (!p) return RSD_ENOMEM;
  o->D = (__nv_bfloat16*)p;
  o->E = (int*)(p + slices);
  return RSD_OK;
}

oz_split_job oz_job(const oz_op& o, const double* X, int64_t ld, int trans, int tri) {
  return oz_split_job{nullptr, 1, 0, X, ld, 0, o.K, o.cols, o.nb, trans, tri, o.K, 0, o.cols, 0, o.D, o.E, o.Kld};
}

int oz_split_blocks(const oz_split_job& J) {
  const int w = J.trans ? SPLIT_TCOLS : SPLIT_COLS;
  return (J.cols + w - 1) / w;
}

void oz_split_launch(cudaStream_t s, const oz_split_job& J0, const oz_split_job* J1 = nullptr) {
  const int nx = std::max(oz_split_blocks(J0), J1 ? oz_split_blocks(*J1) : 0);
  const int nz = std::max(J0.nb, J1 ? J1->nb : 0);
  pdl_launch(oz_split, dim3(nx, J1 ? 2 : 1, nz), SPLIT_THREADS, 0, s, J0, J1 ? *J1 : J0);
}

int oz_map(rsd_ctx* ctx, CUtensorMap* tm, const oz_op& o, int box_rows) {
  memset(tm, 0, sizeof *tm);
  const cuuint64_t dims[2] = {(cuuint64_t)o.Kld, (cuuint64_t)OZ_S * o.nb * o.cols};
  const cuuint64_t strides[1] = {(cuuint64_t)o.Kld * 2};
  const cuuint32_t box[2] = {OZ_KC, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  PFN_cuTensorMapEncodeTiled_v12000 encode = rsd_tensor_map_encoder();
  if (!encode) return rsd_fail(ctx, RSD_EUNSUP, "cuTensorMapEncodeTiled is not available");
  CUresult r = encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, o.D, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return rsd_fail(ctx, RSD_EUNSUP, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return RSD_OK;
}

// C(r, c) = or += +- sum_k R(k, r) S(k, c); `a` carries the options
int oz_gemm_launch(rsd_ctx* ctx, const oz_op& R, const oz_op& S, int m, int n, double* C, int64_t ld, oz_args a) {
  CUtensorMap tmR, tmS;
  RSD_TRY(oz_map(ctx, &tmR, R, OZ_TR));
  RSD_TRY(oz_map(ctx, &tmS, S, OZ_TC));
  a.K = R.K;
  a.m = m;
  a.n = n;
  if (!a.nstep) a.ncap = n;
  a.C = C;
  a.ld = ld;
  a.ER = R.E;
  a.ES = S.E;
  a.rcols = R.cols;
  a.scols = S.cols;
  a.nb = S.nb;
  a.err = ctx->d_info + 1;
  a.wait_ns = ctx->tc_wait_ns > 0 ? (unsigned long long)ctx->tc_wait_ns : OZ_WAIT_NS;
  const dim3 grid((m + OZ_TR - 1) / OZ_TR, (n + OZ_TC - 1) / OZ_TC, S.nb);
  pdl_launch(oz_gemm, grid, OZ_THREADS, OZ_SMEM, ctx->stream, tmS, tmR, a);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

template <int W, bool BACK>
void subst_launch(cudaStream_t s, int w, const double* U, int64_t ldu, const double* Wd, int nsys, double* B, int64_t ldb) {
  pdl_launch(subst64<W, BACK>, (nsys + SUB_SYS - 1) / SUB_SYS, SUB_THREADS, SUB_SMEM<W>, s, w, U, ldu, Wd, nsys, B, ldb);
}

// What a factorisation leaves for the inverse and the solves: the inverses of
// the diagonal blocks and half the exponents of the matrix's diagonal.
int factor64(rsd_ctx* ctx, int n, const char* tag, rsd_factor64* f) {
  const size_t w = (size_t)((n + NB64 - 1) / NB64) * NB64 * NB64;
  const std::string name = std::string("potrf64_") + tag;
  double* p = (double*)rsd_scratch(ctx, name.c_str(), sizeof(double) * w + sizeof(int) * (size_t)n);
  if (!p) return RSD_ENOMEM;
  f->W = p;
  f->dexp = reinterpret_cast<int*>(p + w);
  return RSD_OK;
}

int read_status(rsd_ctx* ctx, const char* what) {
  RSD_CUDA(ctx, cudaMemcpyAsync(ctx->h_info, ctx->d_info, 3 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  RSD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (ctx->h_info[1]) return rsd_fail(ctx, RSD_ETIMEOUT, "%s: tensor-core product timed out (code %d)", what, ctx->h_info[1]);
  return RSD_OK;
}

}  // namespace

// Upper Cholesky factor in place; the inverses of its 64-wide diagonal blocks
// stay in the tag's buffer for potri and the solves.
int rsd_potrf_upper_tag(rsd_ctx* ctx, int n, double* d_A, int64_t lda, int* info, const char* tag) {
  if (n < 1 || lda < n) return rsd_fail(ctx, RSD_EARG, "potrf: n=%d lda=%lld", n, (long long)lda);
  RSD_TRY(oz_init(ctx));
  cudaStream_t s = ctx->stream;
  rsd_factor64 f;
  RSD_TRY(factor64(ctx, n, tag, &f));
  oz_op b, o;
  RSD_TRY(oz_alloc(ctx, "oz_a", NB64, n, 1, &b));
  RSD_TRY(oz_alloc(ctx, "oz_b", NBO64, n, 1, &o));
  RSD_CUDA(ctx, cudaMemsetAsync(ctx->d_info, 0, 2 * sizeof(int), s));
  pdl_launch(diag_exponents, (n + 255) / 256, 256, 0, s, n, d_A, lda, f.dexp);
  for (int J0 = 0; J0 < n; J0 += NBO64) {
    const int JB = n - J0 < NBO64 ? n - J0 : NBO64;
    for (int j0 = J0; j0 < J0 + JB; j0 += NB64) {
      const int jb = n - j0 < NB64 ? n - j0 : NB64, rest = n - j0 - jb;
      double* Wb = f.W + (size_t)(j0 / NB64) * NB64 * NB64;
      pdl_launch(potf2_inv_f64, 1, 256, 0, s, d_A + j0 + (int64_t)j0 * lda, lda, jb, ctx->d_info, j0, Wb);
      if (rest <= 0) break;
      double* P = d_A + j0 + (int64_t)(j0 + jb) * lda;  // the row panel, U^-T P
      subst_launch<NB64, false>(s, NB64, d_A + j0 + (int64_t)j0 * lda, lda, Wb, rest, P, lda);
      const int m_in = J0 + JB - (j0 + jb);  // rows of this outer panel still to update
      if (m_in <= 0) continue;
      b.cols = rest;
      oz_split_launch(s, oz_job(b, P, lda, 0, 0));
      oz_args up{};
      up.tri = up.add = up.neg = 1;
      RSD_TRY(oz_gemm_launch(ctx, b, b, m_in, rest, P + jb, lda, up));
    }
    const int rest = n - J0 - JB;
    if (rest <= 0) break;
    const double* P = d_A + J0 + (int64_t)(J0 + JB) * lda;
    o.cols = rest;
    oz_split_launch(s, oz_job(o, P, lda, 0, 0));
    oz_args up{};
    up.tri = up.add = up.neg = 1;
    RSD_TRY(oz_gemm_launch(ctx, o, o, rest, rest, d_A + (J0 + JB) * (lda + 1), lda, up));
  }
  RSD_CUDA(ctx, cudaGetLastError());
  RSD_TRY(read_status(ctx, "potrf"));
  *info = ctx->h_info[0];
  return RSD_OK;
}

namespace {

// X <- U^-T X (trans) or U^-1 X for many right-hand sides, 128 unknowns a step:
// the block by substitution, then the product that takes it out of the rows
// left.  Rows of X, of U^-1 and columns of U carry the scale of the factored
// matrix's diagonal (dexp).  With explicit inverses of blocks in the
// substitution's place, or of U, the residual would grow by their condition
// numbers (condition 1e10, right-hand sides A X0: 8e-8 of arrangement's result
// through A^-1, 1e-15 so).  eye: X starts as the identity, so block
// b has columns from its own on.
int trsm64(rsd_ctx* ctx, int n, const double* U, int64_t ldu, const rsd_factor64& f, double* X, int64_t ldx, int nrhs,
           bool trans, bool eye) {
  RSD_TRY(oz_init(ctx));
  cudaStream_t s = ctx->stream;
  const int last = (n - 1) / NBS64 * NBS64;
  for (int p = 0; p <= last; p += NBS64) {
    const int j0 = trans ? p : last - p, j1 = std::min(n, j0 + NBS64), c0 = eye ? j0 : 0, nc = nrhs - c0;
    const double *Ub = U + j0 + (int64_t)j0 * ldu, *Wb = f.W + (size_t)(j0 / NB64) * NB64 * NB64;
    double* Xc = X + (int64_t)c0 * ldx;
    if (trans)
      subst_launch<NBS64, false>(s, j1 - j0, Ub, ldu, Wb, nc, Xc + j0, ldx);
    else
      subst_launch<NBS64, true>(s, j1 - j0, Ub, ldu, Wb, nc, Xc + j0, ldx);
    const int r0 = trans ? j1 : 0, m = trans ? n - j1 : j0;  // rows left
    if (m <= 0) continue;
    oz_op R, S;
    RSD_TRY(oz_alloc(ctx, "oz_a", NBS64, m, 1, &R));
    RSD_TRY(oz_alloc(ctx, "oz_b", NBS64, nc, 1, &S));
    oz_split_job r = oz_job(R, trans ? U + j0 + (int64_t)r0 * ldu : U + r0 + (int64_t)j0 * ldu, ldu, !trans, 0);
    oz_split_job x = oz_job(S, Xc + j0, ldx, 0, 0);
    r.kn = x.kn = j1 - j0;
    if (!trans) {
      r.ks = x.ks = f.dexp + j0;
      r.ksgn = -1;
    }
    oz_split_launch(s, r, &x);
    oz_args a{};
    a.add = a.neg = 1;
    RSD_TRY(oz_gemm_launch(ctx, R, S, m, nc, Xc + r0, ldx, a));
  }
  return RSD_OK;
}

}  // namespace

// V = U^-1 by pairs of blocks, [V11, -V11 U12 V22; 0, V22], from the 64-wide
// inverses on, all pairs of a size at once: few and large products, whose
// residual grows with the condition number of the blocks.
static int inverse_by_pairs(rsd_ctx* ctx, int n, const double* d_A, int64_t lda, const rsd_factor64& f, double* V) {
  cudaStream_t s = ctx->stream;
  pdl_launch(put_diag64, (n + NB64 - 1) / NB64, 256, 0, s, n, f.W, V, n);
  for (int h = NB64; h < n; h *= 2) {
    // pair z: blocks [2 z h, 2 z h + h) and [2 z h + h, min(2 z h + 2 h, n))
    const int np = (n - h + 2 * h - 1) / (2 * h);
    const int64_t dA = 2LL * h * (lda + 1), dV = 2LL * h * (n + 1);
    const int c2 = std::min(h, n - h);  // columns of the first pair
    oz_op R, S;
    RSD_TRY(oz_alloc(ctx, "oz_a", h, h, np, &R));
    RSD_TRY(oz_alloc(ctx, "oz_b", h, c2, np, &S));
    double* T = V + (int64_t)h * n;  // block (1, 2) of the first pair
    // T = U12 V22
    oz_split_job r = oz_job(R, d_A + (int64_t)h * lda, lda, 1, 0);
    r.sX = dA;
    r.kn = n - h;
    r.kstep = 2 * h;
    oz_split_job q = oz_job(S, V + h + (int64_t)h * n, n, 0, 1);
    q.sX = dV;
    q.kn = q.cn = n - h;
    q.kstep = q.cstep = 2 * h;
    r.ks = q.ks = f.dexp + h;  // column k of U against row k of U^-1
    r.kstride = q.kstride = 2 * h;
    r.ksgn = -1;
    oz_split_launch(s, r, &q);
    oz_args a{};
    a.khi_col = 1;
    a.sC = dV;
    a.ncap = n - h;  // the last pair's second block may be narrower
    a.nstep = 2 * h;
    RSD_TRY(oz_gemm_launch(ctx, R, S, h, c2, T, n, a));
    // V12 = -V11 T
    r = oz_job(R, V, n, 1, 1);
    r.sX = dV;
    q = oz_job(S, T, n, 0, 0);
    q.sX = dV;
    q.cn = n - h;
    q.cstep = 2 * h;
    oz_split_launch(s, r, &q);
    oz_args b{};
    b.klo_row = b.neg = 1;
    b.sC = dV;
    b.ncap = n - h;
    b.nstep = 2 * h;
    RSD_TRY(oz_gemm_launch(ctx, R, S, h, c2, T, n, b));
  }
  return RSD_OK;
}

// The workspaces of the inverse: 2 for V = U^-1 and its digits (25.5 n^2 bytes),
// 1 where only those of the form in place can be had (36 IP64 n), 0 for neither.
constexpr int IP64 = 512;
int rsd_potri64_space(rsd_ctx* ctx, int n) {
  size_t pairs = 0;  // the right operands of inverse_by_pairs
  for (int h = NB64; h < n; h *= 2) pairs = std::max(pairs, oz_bytes(h, std::min(h, n - h), (n + h - 1) / (2 * h)));
  if (rsd_scratch_try(ctx, "potri64_V", sizeof(double) * (size_t)n * n) &&
      rsd_scratch_try(ctx, "oz_a", oz_bytes(n, n, 1)) && rsd_scratch_try(ctx, "oz_b", std::max(pairs, oz_bytes(NBO64, 2 * n, 1))))
    return 2;
  for (const char* name : {"potri64_V", "oz_a", "oz_b"}) rsd_scratch_free(ctx, name);
  return rsd_scratch_try(ctx, "potri64_T", sizeof(double) * (size_t)n * IP64) &&
         rsd_scratch_try(ctx, "oz_a", oz_bytes(IP64, n, 1)) &&
         rsd_scratch_try(ctx, "oz_b", std::max(oz_bytes(IP64, IP64, 1), oz_bytes(NBO64, 2 * n, 1)));
}

// A^-1 in place of its factor, IP64 columns at a time.  V = U^-1 from the last
// columns on: a block's columns are U^-1 of the identity's by substitution, which
// needs the columns of U before them only.  Then V V^T from the first columns on:
// the entries above and in block J take the columns of V from J on only.  The
// digits of V are made anew for each block they meet.  Factor and inverse of order
// 1536 take 5.3 ms so and 3.5 through V in its own memory, of order 3072 15.0 and
// 7.7, with the same residual.
static int inverse_in_place(rsd_ctx* ctx, int n, double* d_A, int64_t lda, const rsd_factor64& f) {
  cudaStream_t s = ctx->stream;
  double* T = (double*)rsd_scratch(ctx, "potri64_T", sizeof(double) * (size_t)n * IP64);
  if (!T) return RSD_ENOMEM;
  const int last = (n - 1) / IP64 * IP64;
  for (int j0 = last; j0 >= 0; j0 -= IP64) {
    const int j1 = std::min(n, j0 + IP64), w = j1 - j0;
    RSD_CUDA(ctx, cudaMemsetAsync(T, 0, sizeof(double) * (size_t)j1 * w, s));
    pdl_launch(put_ones64, (w + 255) / 256, 256, 0, s, w, T + j0, (int64_t)j1);
    RSD_TRY(trsm64(ctx, j1, d_A, lda, f, T, j1, w, false, false));
    RSD_CUDA(ctx, cudaMemcpy2DAsync(d_A + (int64_t)j0 * lda, sizeof(double) * lda, T, sizeof(double) * j1,
                                    sizeof(double) * j1, w, cudaMemcpyDeviceToDevice, s));
  }
  for (int j0 = 0; j0 < n; j0 += IP64) {
    const int j1 = std::min(n, j0 + IP64);
    for (int k0 = j0; k0 < n; k0 += IP64) {
      const int wk = std::min(n, k0 + IP64) - k0;
      oz_op R, S;
      RSD_TRY(oz_alloc(ctx, "oz_a", wk, j1, 1, &R));
      RSD_TRY(oz_alloc(ctx, "oz_b", wk, j1 - j0, 1, &S));
      oz_split_job r = oz_job(R, d_A + (int64_t)k0 * lda, lda, 1, 0);
      oz_split_job x = oz_job(S, d_A + j0 + (int64_t)k0 * lda, lda, 1, 0);
      oz_split_launch(s, r, &x);
      oz_args a{};
      a.add = k0 > j0;
      RSD_TRY(oz_gemm_launch(ctx, R, S, j1, j1 - j0, d_A + (int64_t)j0 * lda, lda, a));
    }
  }
  return RSD_OK;
}

// A^-1 (upper triangle) from the factor in A and what potrf left with it, as V
// V^T with V = U^-1.  V comes by pairs of blocks first; with the rows of V scaled
// by the diagonal of the factored matrix its largest entry bounds what the pairs
// add to the residual.  Up to 2^GROWTH64 (mobilities: below 4) A^-1 is formed from
// it, beyond (near contacts: 1e2 at a gap of 1e-4) the product stands aside for
// trsm64 on the identity.  ||A X - I|| / (||A|| ||X||) of stiff pairs at 1e4 and
// 1e8: 12 and 900 eps by pairs, 0.8 and 0.8 by substitution.  N = 512, order 3072:
// the FP64 step takes 3.6 ms longer that way.
int rsd_potri64(rsd_ctx* ctx, int n, double* d_A, int64_t lda, const rsd_factor64& f) {
  RSD_TRY(oz_init(ctx));
  cudaStream_t s = ctx->stream;
  RSD_CUDA(ctx, cudaMemsetAsync(ctx->d_info, 0, 3 * sizeof(int), s));
  const int space = rsd_potri64_space(ctx, n);
  if (!space) return rsd_fail(ctx, RSD_ENOMEM, "cannot allocate the workspaces of an inverse of order %d", n);
  if (space == 1) {
    RSD_TRY(inverse_in_place(ctx, n, d_A, lda, f));
    return read_status(ctx, "potri");
  }
  double* V = (double*)rsd_scratch(ctx, "potri64_V", sizeof(double) * (size_t)n * n);
  if (!V) return RSD_ENOMEM;
  oz_op R;
  for (int exact = 0; exact < 2; exact++) {
    if (exact) {
      RSD_CUDA(ctx, cudaMemsetAsync(V, 0, sizeof(double) * (size_t)n * n, s));
      pdl_launch(put_ones64, (n + 255) / 256, 256, 0, s, n, V, (int64_t)n);
      RSD_TRY(trsm64(ctx, n, d_A, lda, f, V, n, n, false, true));
    } else {
      RSD_TRY(inverse_by_pairs(ctx, n, d_A, lda, f, V));
    }
    RSD_TRY(oz_alloc(ctx, "oz_a", n, n, 1, &R));
    oz_split_launch(s, oz_job(R, V, n, 1, 1));
    oz_args a{};
    a.tri = a.klo_row = a.klo_col = 1;
    if (!exact) {
      pdl_launch(growth64, (n + 255) / 256, 256, 0, s, n, R.E, f.dexp, ctx->d_info + 2);
      a.gate = ctx->d_info + 2;
    }
    RSD_TRY(oz_gemm_launch(ctx, R, R, n, n, d_A, lda, a));
    RSD_TRY(read_status(ctx, "potri"));
    if (ctx->h_info[2] <= GROWTH64) break;
  }
  return RSD_OK;
}

int rsd_potri_upper_tag(rsd_ctx* ctx, int n, double* d_A, int64_t lda, const char* tag) {
  rsd_factor64 f;
  RSD_TRY(factor64(ctx, n, tag, &f));
  return rsd_potri64(ctx, n, d_A, lda, f);
}

int rsd_potrf64_factor(rsd_ctx* ctx, int n, const char* tag, rsd_factor64* f) { return factor64(ctx, n, tag, f); }

// U^T Y = X (X is overwritten) for 1 to 4 right-hand sides of length n
int rsd_trsv64_fwd(rsd_ctx* ctx, int n, const double* U, int64_t ldu, const double* W, double* X, double* Y,
                   int64_t ldx, int nrhs) {
  if (nrhs < 1 || nrhs > 4) return rsd_fail(ctx, RSD_EARG, "trsv: nrhs %d", nrhs);
  cudaStream_t s = ctx->stream;
  for (int b = 0; b * NB64 < n; b++) {
    const int rest = std::max(0, n - (b + 1) * NB64);
    const int grid = std::max(1, std::min(2 * ctx->sm_count, (rest + 7) / 8));
    switch (nrhs) {
      case 1: pdl_launch(trsv64_fwd<1>, grid, 256, 0, s, n, b, U, ldu, W, X, Y, ldx); break;
      case 2: pdl_launch(trsv64_fwd<2>, grid, 256, 0, s, n, b, U, ldu, W, X, Y, ldx); break;
      case 3: pdl_launch(trsv64_fwd<3>, grid, 256, 0, s, n, b, U, ldu, W, X, Y, ldx); break;
      default: pdl_launch(trsv64_fwd<4>, grid, 256, 0, s, n, b, U, ldu, W, X, Y, ldx); break;
    }
  }
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// U X = Y (Y is overwritten)
int rsd_trsv64_bwd(rsd_ctx* ctx, int n, const double* U, int64_t ldu, const double* W, double* Y, double* X,
                   int64_t ldx, int nrhs) {
  if (nrhs < 1 || nrhs > 4) return rsd_fail(ctx, RSD_EARG, "trsv: nrhs %d", nrhs);
  cudaStream_t s = ctx->stream;
  for (int b = (n + NB64 - 1) / NB64 - 1; b >= 0; b--) {
    const int grid = std::max(1, std::min(2 * ctx->sm_count, (b * NB64 + 31) / 32));
    switch (nrhs) {
      case 1: pdl_launch(trsv64_bwd<1>, grid, 128, 0, s, n, b, U, ldu, W, Y, X, ldx); break;
      case 2: pdl_launch(trsv64_bwd<2>, grid, 128, 0, s, n, b, U, ldu, W, Y, X, ldx); break;
      case 3: pdl_launch(trsv64_bwd<3>, grid, 128, 0, s, n, b, U, ldu, W, Y, X, ldx); break;
      default: pdl_launch(trsv64_bwd<4>, grid, 128, 0, s, n, b, U, ldu, W, Y, X, ldx); break;
    }
  }
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// Solve (U^T U) X = B in place with the factor of `tag`: substitution, a
// launch per 64 unknowns for up to 4 right-hand sides, on the tensor cores for
// more (arrangement, matrices.f90:432-445).
int rsd_potrs_upper_tag(rsd_ctx* ctx, int n, const double* d_U, int64_t ldu, double* d_X, int64_t ldx, int nrhs,
                        const char* tag) {
  cudaStream_t s = ctx->stream;
  rsd_factor64 f;
  RSD_TRY(factor64(ctx, n, tag, &f));
  if (nrhs <= 4) {
    double* Y = (double*)rsd_scratch(ctx, "potrs64_Y", sizeof(double) * (size_t)n * nrhs);
    double* X = (double*)rsd_scratch(ctx, "potrs64_X", sizeof(double) * (size_t)n * nrhs);
    if (!Y || !X) return RSD_ENOMEM;
    const size_t col = sizeof(double) * n;
    RSD_CUDA(ctx, cudaMemcpy2DAsync(X, col, d_X, sizeof(double) * ldx, col, nrhs, cudaMemcpyDeviceToDevice, s));
    RSD_TRY(rsd_trsv64_fwd(ctx, n, d_U, ldu, f.W, X, Y, n, nrhs));
    RSD_TRY(rsd_trsv64_bwd(ctx, n, d_U, ldu, f.W, Y, X, n, nrhs));
    RSD_CUDA(ctx, cudaMemcpy2DAsync(d_X, sizeof(double) * ldx, X, col, col, nrhs, cudaMemcpyDeviceToDevice, s));
    return RSD_OK;
  }
  oz_op big;  // the largest operands first: the buffers grow once
  RSD_TRY(oz_alloc(ctx, "oz_a", NBS64, n, 1, &big));
  RSD_TRY(oz_alloc(ctx, "oz_b", NBS64, nrhs, 1, &big));
  RSD_CUDA(ctx, cudaMemsetAsync(ctx->d_info, 0, 2 * sizeof(int), s));
  RSD_TRY(trsm64(ctx, n, d_U, ldu, f, d_X, ldx, nrhs, true, false));
  RSD_TRY(trsm64(ctx, n, d_U, ldu, f, d_X, ldx, nrhs, false, false));
  return read_status(ctx, "potrs");
}
