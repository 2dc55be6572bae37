// Mixed-precision grand-resistance solve: FP32 factorisations, FP64
// refinement.  Same outputs as STEPPER_NOGmres (src/stepper.f90:348-410):
// U_par = RPP^-1 (Fe + RPQ EIN) and SijN_hyd = (RPQ^T RPP^-1 RPQ - RQQ) EIN
// with R = M^-1 + L, but without forming M^-1.
//
// Augmented system in (f, U), with w = [U; -EIN]:
//     M f = w                    (f = R_inf w, the far-field forces)
//     f_P + (L w)_P = Fe          (force balance with lubrication)
// and then SijN_hyd = f_Q + (L w)_Q.  Its residual needs only the products
// M f (an HBM-bound dense GEMV in double-single arithmetic over M's two
// FP32 planes, ~FP64 accuracy for the sums) and L w (an FP64 block-sparse
// product over the near pairs, L is never formed densely here).  The correction is
// solved with FP32 factors:
//   M' = [M_QQ M_QP; M_PQ M_PP] = U'^T U'  (stresslets ordered first), so the
//   trailing block U'_PP is the Cholesky factor of the Schur complement
//   A = M_PP - M_PQ M_QQ^-1 M_QP and (M^-1)_PP = A^-1 = U'_PP^-1 U'_PP^-T;
//   RPP32 = A^-1 + rfu = V^T V.
//   correction: y = M^-1 r1; dU = RPP^-1 (r2 - y_P); df = y + M^-1 [dU; 0].
// Iterates until ||r|| <= tol ||b|| per right-hand side.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "dsf.cuh"
#include "pdl.cuh"
#include "rsd_internal.cuh"

template <typename T>
int rsd_gemv(rsd_ctx* ctx, int trans, int m, int k, T alpha, const T* A, int64_t lda, const T* X, int64_t ldx,
             int nrhs, T beta, T* y, int64_t ldy);
template <typename T>
int rsd_potrf_upper_t(rsd_ctx* ctx, int n, T* d_A, int64_t lda, int* info, const char* tag, int tc,
                      int* d_status = nullptr, rsd_factor_use use = RSD_FACTOR_STEP);
template <typename T>
int rsd_potri_upper_t(rsd_ctx* ctx, int n, T* d_A, int64_t lda, const char* tag, int tc, const T* W = nullptr,
                      int* d_err = nullptr);
template <typename T>
int rsd_mirror_upper_t(rsd_ctx* ctx, int n, T* d_A, int64_t lda);
int rsd_wide_inverses_s(rsd_ctx* ctx, int n, const float* U, int64_t ldu, const char* tag, const float* W128,
                        float** W2out);
const float* rsd_potrf_inverses_s(rsd_ctx* ctx, int n, const char* tag);
int rsd_potrs_wide_s(rsd_ctx* ctx, int n, const float* U, int64_t ldu, const float* W2, float* X, int64_t ldx,
                     int nrhs, float* Y);

namespace {

// particle of grand-matrix index x
__device__ __forceinline__ int grand_pid(int N, int x) {
  return x < 3 * N ? x / 3 : (x < 6 * N ? (x - 3 * N) / 3 : (x - 6 * N) / 5);
}

// The FP32 matrix M32 is M in [Q, P] order, Q padded to Qp (a multiple of the
// factorisation's block, so that the diagonal blocks of U_PP are blocks of
// the factor) and P to Pp (a multiple of 4, for 16-byte columns) with the
// identity; np = Qp + Pp.
struct mixed_dims {
  int64_t P, Q, n, Qp, Pp, np;
};

// M32 from the hi plane holding only the stored half (entries whose row's
// particle is at most the column's; the rest is read at the transposed
// position): 32 x 32 output tiles, the direct and the transposed source tiles
// staged in shared memory so that reads and writes stay coalesced; a tile
// loads only the kinds it needs.
__device__ __forceinline__ int64_t perm_src(const mixed_dims& d, int64_t i) {  // -1: padding
  if (i < d.Qp) return i < d.Q ? d.P + i : -1;
  return i < d.Qp + d.P ? i - d.Qp : -1;
}

__global__ void convert_perm_half(int N, mixed_dims d, const float* __restrict__ Mh, int64_t ld,
                                  float* __restrict__ M32) {
  pdl_enter();
  __shared__ float D[32][33], T[32][33];
  __shared__ int64_t si[32], sj[32];
  __shared__ int pi[32], pj[32], need;
  const int64_t I0 = (int64_t)blockIdx.x * 32, J0 = (int64_t)blockIdx.y * 32, n = d.np;
  const int tx = threadIdx.x, ty = threadIdx.y;
  if (ty == 0) {
    const int64_t i = perm_src(d, I0 + tx), j = perm_src(d, J0 + tx);
    si[tx] = i;
    sj[tx] = j;
    pi[tx] = i >= 0 ? grand_pid(N, (int)i) : -1;
    pj[tx] = j >= 0 ? grand_pid(N, (int)j) : -1;
    // need: bit 0 = some entry stored directly, bit 1 = some entry transposed
    const int big = 1 << 30;
    const int imin = __reduce_min_sync(0xffffffffu, i >= 0 ? pi[tx] : big), imax = __reduce_max_sync(0xffffffffu, pi[tx]);
    const int jmin = __reduce_min_sync(0xffffffffu, j >= 0 ? pj[tx] : big), jmax = __reduce_max_sync(0xffffffffu, pj[tx]);
    if (tx == 0) need = (imin <= jmax ? 1 : 0) | (imax > jmin ? 2 : 0);
  }
  __syncthreads();
  const int t = ty * 32 + tx;
  // rows contiguous in the source and no padding in the tile
  const bool full = si[0] >= 0 && si[31] - si[0] == 31 && sj[0] >= 0 && sj[31] - sj[0] == 31;
  if (need == 1 && full && (n & 3) == 0 && (si[0] & 3) == 0) {
    // all in place: one 16-byte move per thread (4 rows of one column)
    const int r4 = 4 * (t & 7), k = t >> 3;
    *reinterpret_cast<float4*>(M32 + I0 + r4 + (J0 + k) * n) =
        *reinterpret_cast<const float4*>(Mh + si[0] + r4 + sj[k] * ld);
    return;
  }
  for (int k = ty; k < 32; k += blockDim.y) {
    // (I0 + tx, J0 + k) in place; (I0 + k, J0 + tx) at the mirrored position
    if ((need & 1) && si[tx] >= 0 && sj[k] >= 0) D[k][tx] = Mh[si[tx] + sj[k] * ld];
    if ((need & 2) && sj[tx] >= 0 && si[k] >= 0) T[k][tx] = Mh[sj[tx] + si[k] * ld];
  }
  __syncthreads();
  for (int k = ty; k < 32; k += blockDim.y) {
    const int64_t i = I0 + tx, j = J0 + k;
    if (i >= n || j >= n) continue;
    float v;
    if (si[tx] < 0 || sj[k] < 0)
      v = i == j ? 1.f : 0.f;
    else
      v = pi[tx] <= pj[k] ? D[k][tx] : T[tx][k];
    M32[i + j * n] = v;
  }
}

// x (FP64) as float pairs
__global__ void to_dsf_vec(int64_t n, const double* __restrict__ x, float2* __restrict__ xs) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const dsf d = dsf_from(x[t]);
  xs[t] = make_float2(d.hi, d.lo);
}

// Symmetric M f over the stored half of M's planes: the entries whose row's
// particle is at most the column's (pair blocks in the rows of their first
// particle, and the whole diagonal particle blocks).  A CTA takes a 128 x 128
// tile: row products of its stored entries (-> prow[R][C]) and column
// products of its entries strictly above the particle diagonal
// (-> pcol[C][R]), in double-single; tiles with no stored entry write zero
// partials, in double-single arithmetic on the FP32 pipe (the FP64 pipe of
// GB300 would bound an FP64 product at ~1/60 of the FP32 rate; this one is
// bound by HBM).  About half of M is read.  Needs ld % 4 == 0.
constexpr int SYMV_T = 128;
constexpr int symv_smem(int nr) { return (int)(sizeof(dsf) * 8 * nr * SYMV_T + sizeof(float2) * nr * SYMV_T * 33); }
template <int NR>
__global__ void __launch_bounds__(256) symv_planes_part(int N, int n, const float* __restrict__ Mh,
                                                        const float* __restrict__ Ml, int64_t ld,
                                                        const float2* __restrict__ xs, int nbt,
                                                        double* __restrict__ prow, double* __restrict__ pcol) {
  pdl_enter();
  // dynamic shared memory (symv_smem(NR) bytes): the row partials of the 8
  // warps, then the per-lane column partials, reduced after the tile
  extern __shared__ __align__(16) unsigned char symv_raw[];
  auto red = reinterpret_cast<dsf(*)[NR][SYMV_T]>(symv_raw);
  auto colp = reinterpret_cast<float2(*)[SYMV_T][33]>(symv_raw + sizeof(dsf) * 8 * NR * SYMV_T);
  __shared__ int skip;
  const int R = blockIdx.x, C = blockIdx.y, r0 = R * SYMV_T, c0 = C * SYMV_T;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  double* pr = prow + ((size_t)R * nbt + C) * NR * SYMV_T;
  double* pc = pcol + ((size_t)C * nbt + R) * NR * SYMV_T;
  if (warp == 0) {  // stored entries exist iff min over rows of pid <= max over columns
    int rmin = 1 << 30, cmax = -1;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = r0 + 4 * lane + k, c = c0 + 4 * lane + k;
      if (r < n) rmin = min(rmin, grand_pid(N, r));
      if (c < n) cmax = max(cmax, grand_pid(N, c));
    }
    rmin = __reduce_min_sync(0xffffffffu, rmin);
    cmax = __reduce_max_sync(0xffffffffu, cmax);
    if (lane == 0) skip = rmin > cmax;
  }
  __syncthreads();
  if (skip) {
    for (int e = t; e < NR * SYMV_T; e += 256) pr[e] = pc[e] = 0.0;
    return;
  }
  const int rb = r0 + 4 * lane;  // this lane's four rows (past n: the padding of the column)
  int prr[4];
  dsf xr[NR][4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool ok = rb + k < n;
    prr[k] = ok ? grand_pid(N, rb + k) : (1 << 30);
#pragma unroll
    for (int r = 0; r < NR; r++) {
      const float2 v = ok ? xs[rb + k + (int64_t)r * n] : make_float2(0.f, 0.f);
      xr[r][k] = dsf(v.x, v.y);
    }
  }
  const int pmin = min(min(prr[0], prr[1]), min(prr[2], prr[3]));  // a section may end among them
  dsacc racc[NR][4];
#pragma unroll
  for (int r = 0; r < NR; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) racc[r][k] = dsacc(0);
#pragma unroll 8
  for (int cc = 0; cc < SYMV_T / 8; cc++) {
    const int cl = warp * (SYMV_T / 8) + cc, c = c0 + cl;
    dsacc cacc[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) cacc[r] = dsacc(0);
    if (c < n) {
      const int pcn = grand_pid(N, c);
      if (rb < n && pmin <= pcn) {  // the lane's rows hold stored entries of this column
        const int64_t o = rb + (int64_t)c * ld;
        const float4 h = *reinterpret_cast<const float4*>(Mh + o), l = *reinterpret_cast<const float4*>(Ml + o);
        const dsf m[4] = {dsf(h.x, l.x), dsf(h.y, l.y), dsf(h.z, l.z), dsf(h.w, l.w)};
#pragma unroll
        for (int r = 0; r < NR; r++) {
          const float2 xv = xs[c + (int64_t)r * n];
          const dsf xc(xv.x, xv.y);
#pragma unroll
          for (int k = 0; k < 4; k++) {
            if (prr[k] <= pcn) racc[r][k] = fma(m[k], xc, racc[r][k]);
            if (prr[k] < pcn) cacc[r] = fma(m[k], xr[r][k], cacc[r]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < NR; r++) {
      dsacc_norm(cacc[r]);
      colp[r][cl][lane] = make_float2(cacc[r].hi, cacc[r].lo);
    }
  }
#pragma unroll
  for (int r = 0; r < NR; r++)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      dsacc_norm(racc[r][k]);
      red[warp][r][4 * lane + k] = dsf(racc[r][k].hi, racc[r][k].lo);
    }
  __syncthreads();
  for (int e = t; e < NR * SYMV_T; e += 256) {
    const int r = e / SYMV_T, il = e % SYMV_T;
    dsf v = red[0][r][il];
#pragma unroll
    for (int w = 1; w < 8; w++) v = v + red[w][r][il];
    pr[e] = dsf_to(v);
    dsf u(colp[r][il][0].x, colp[r][il][0].y);
#pragma unroll 8
    for (int q = 1; q < 32; q++) u = u + dsf(colp[r][il][q].x, colp[r][il][q].y);
    pc[e] = dsf_to(u);
  }
}

// y(:, r) += alpha * (sum_C prow[K][C] + sum_R pcol[K][R]) for row block K, fixed order
__global__ void symv_planes_reduce(int n, int nr, int nbt, const double* __restrict__ prow,
                                   const double* __restrict__ pcol, double alpha, double* __restrict__ y,
                                   int64_t ldy) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int K = i / SYMV_T, e = i % SYMV_T;
  for (int r = 0; r < nr; r++) {
    double s0 = 0.0, s1 = 0.0;
    for (int J = 0; J < nbt; J++) {
      s0 += prow[(((size_t)K * nbt + J) * nr + r) * SYMV_T + e];
      s1 += pcol[(((size_t)K * nbt + J) * nr + r) * SYMV_T + e];
    }
    y[i + (int64_t)r * ldy] += alpha * (s0 + s1);
  }
}

__global__ void copy_block_f(int64_t rows, int64_t cols, const float* __restrict__ S, int64_t lds,
                             float* __restrict__ D, int64_t ldd) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= rows * cols) return;
  const int64_t i = t % rows, j = t / rows;
  D[i + j * ldd] = S[i + j * lds];
}

// w = [U; -EIN] per column
__global__ void build_w(int64_t P, int64_t Q, int nr, const double* __restrict__ U, const double* __restrict__ ein,
                        double* __restrict__ w) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = P + Q;
  if (t >= n * nr) return;
  const int64_t i = t % n, c = t / n;
  w[t] = i < P ? U[i + c * P] : -ein[i - P];
}

// r2 = Fe_c - f_P - (Lw)_P  (Fe only in column 0 when have_fe)
__global__ void build_r2(int64_t P, int64_t n, int nr, const double* __restrict__ Fe, int have_fe,
                         const double* __restrict__ f, const double* __restrict__ Lw, double* __restrict__ r2) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P * nr) return;
  const int64_t i = t % P, c = t / P;
  const double fe = (have_fe && c == 0) ? Fe[i] : 0.0;
  r2[t] = fe - f[i + c * n] - Lw[i + c * n];
}

// ---- the stationary iteration's elementwise work, fused into the four
// kernels between its products and solves (an iteration of a small system is
// launches and little else)

// w = [U; -EIN], r1 = w, fs = f as float pairs
__global__ void it_begin(int64_t P, int64_t Q, int nr, const double* __restrict__ U, const double* __restrict__ ein,
                         const double* __restrict__ f, double* __restrict__ w, double* __restrict__ r1,
                         float2* __restrict__ fs) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n = P + Q;
  if (t >= n * nr) return;
  const int64_t i = t % n, c = t / n;
  w[t] = r1[t] = i < P ? U[i + c * P] : -ein[i - P];
  const dsf d = dsf_from(f[t]);
  fs[t] = make_float2(d.hi, d.lo);
}

// r2 = Fe_c - f_P - (Lw)_P (Fe only in column 0 when have_fe); t32 = r1 in the
// padded [Q, P] order; per block of the grid the sums of squares of (r1, r2)
// and of b = ([0; -EIN], Fe), added up by the host.  blockIdx.y = column.
constexpr int IT_BLOCKS = 32;
__global__ void __launch_bounds__(256) it_residual(mixed_dims d, const double* __restrict__ r1,
                                                   const double* __restrict__ ein, const double* __restrict__ Fe,
                                                   int have_fe, const double* __restrict__ f,
                                                   const double* __restrict__ Lw, double* __restrict__ r2,
                                                   float* __restrict__ t32, double* __restrict__ part) {
  pdl_enter();
  __shared__ double sr[256], sb[256];
  const int c = blockIdx.y;
  const double *r1c = r1 + c * d.n, *fc = f + c * d.n, *lc = Lw + c * d.n;
  const bool fe = have_fe && c == 0;
  double a = 0.0, b = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < d.np; i += (int64_t)gridDim.x * 256) {
    const int64_t q = perm_src(d, i);
    float o = 0.f;
    if (q >= 0) {
      const double v = r1c[q];
      a += v * v;
      o = (float)v;
      if (q >= d.P) {
        const double e = ein[q - d.P];
        b += e * e;
      } else {
        const double g = fe ? Fe[q] : 0.0, x = g - fc[q] - lc[q];
        r2[q + c * d.P] = x;
        a += x * x;
        b += g * g;
      }
    }
    t32[i + c * d.np] = o;
  }
  sr[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      sr[threadIdx.x] += sr[threadIdx.x + h];
      sb[threadIdx.x] += sb[threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * (c * gridDim.x + blockIdx.x)] = sr[0];
    part[2 * (c * gridDim.x + blockIdx.x) + 1] = sb[0];
  }
}

// Per block of the grid the sums of squares of the sizes of r2's terms, |Fe| + |f_P|
// + (|L||w|)_P, in La the last.
__global__ void __launch_bounds__(256) it_scale(int64_t P, const double* __restrict__ Fe, const double* __restrict__ f,
                                                const double* __restrict__ La, double* __restrict__ part) {
  pdl_enter();
  __shared__ double red[256];
  double a = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < P; i += (int64_t)gridDim.x * 256) {
    const double v = (Fe ? fabs(Fe[i]) : 0.0) + fabs(f[i]) + La[i];
    a += v * v;
  }
  red[threadIdx.x] = a;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// y = unperm(x32) (y = M^-1 r1); u32 = r2 - y_P, zero past P
__global__ void it_velocity(mixed_dims d, int nr, const float* __restrict__ x32, const double* __restrict__ r2,
                            double* __restrict__ y, float* __restrict__ u32) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.np * nr) return;
  const int64_t i = t % d.np, c = t / d.np, q = perm_src(d, i);
  double v = 0.0;
  if (q >= 0) {
    v = (double)x32[t];
    y[q + c * d.n] = v;
  }
  if (i >= d.Qp) u32[i - d.Qp + c * d.Pp] = q >= 0 ? (float)(r2[q + c * d.P] - v) : 0.f;
}

// t32 = [0; dU]
__global__ void it_force(mixed_dims d, int nr, const float* __restrict__ du, float* __restrict__ t32) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.np * nr) return;
  const int64_t i = t % d.np, c = t / d.np;
  t32[t] = i < d.Qp ? 0.f : du[i - d.Qp + c * d.Pp];
}

// f += y + unperm(x32), U += dU
__global__ void it_update(mixed_dims d, int nr, const float* __restrict__ x32, const double* __restrict__ y,
                          const float* __restrict__ du, double* __restrict__ f, double* __restrict__ U) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.np * nr) return;
  const int64_t i = t % d.np, c = t / d.np, q = perm_src(d, i);
  if (q < 0) return;
  f[q + c * d.n] += y[q + c * d.n] + (double)x32[t];
  if (q < d.P) U[q + c * d.P] += (double)du[q + c * d.Pp];
}

// ---- the same pieces one by one, for the GMRES below (one right-hand side)

// y32 = x in the padded [Q, P] order
__global__ void to32_perm(mixed_dims d, const double* __restrict__ x, float* __restrict__ y) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.np) return;
  const int64_t q = perm_src(d, t);
  y[t] = q >= 0 ? (float)x[q] : 0.f;
}

// y (FP64, [P, Q] order) += unperm(x32)
__global__ void from32_add(mixed_dims d, const float* __restrict__ x, double* __restrict__ y) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.np) return;
  const int64_t q = perm_src(d, t);
  if (q >= 0) y[q] += (double)x[t];
}

// S = f_Q + (Lw)_Q of column c; U_par = U column 0
__global__ void outputs(int64_t P, int64_t Q, int c, const double* __restrict__ f, const double* __restrict__ Lw,
                        const double* __restrict__ U, double* __restrict__ Upar, double* __restrict__ S) {
  pdl_enter();
  const int64_t n = P + Q;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < Q) S[t] = f[P + t + c * n] + Lw[P + t + c * n];
  if (t < P) Upar[t] = U[t];
}

inline unsigned nblk(int64_t n) { return (unsigned)((n + 255) / 256); }

// ---- flexible GMRES on the augmented system (one right-hand side at a time)
// x = (f [n], U [P]); A x = (M f - [U; 0], f_P + (L [U; 0])_P); the
// preconditioner is the correction of the stationary iteration above.
// Krylov vectors are FP64 of length n + P.

// out[k] = V_k . w for k < nk (one block per k)
__global__ void gm_dots(int64_t len, int nk, const double* __restrict__ V, int64_t ldv, const double* __restrict__ w,
                        double* __restrict__ out) {
  pdl_enter();
  __shared__ double red[256];
  const int k = blockIdx.x;
  double a = 0.0;
  for (int64_t i = threadIdx.x; i < len; i += 256) a += V[i + k * ldv] * w[i];
  red[threadIdx.x] = a;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[k] = red[0];
}

// w -= sum_k h[k] V_k; hacc[k] += h[k] (thread 0 of block 0)
__global__ void gm_orth(int64_t len, int nk, const double* __restrict__ V, int64_t ldv, const double* __restrict__ h,
                        double* __restrict__ w, double* __restrict__ hacc) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0)
    for (int k = 0; k < nk; k++) hacc[k] += h[k];
  if (i >= len) return;
  double s = w[i];
  for (int k = 0; k < nk; k++) s -= h[k] * V[i + k * ldv];
  w[i] = s;
}

// v = w / sqrt(nrm2[0])
__global__ void gm_scale(int64_t len, const double* __restrict__ w, const double* __restrict__ nrm2,
                         double* __restrict__ v) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < len) v[i] = w[i] / sqrt(nrm2[0]);
}

// x += sum_k y[k] Z_k
__global__ void gm_update(int64_t len, int nk, const double* __restrict__ Z, int64_t ldz, const double* __restrict__ y,
                          double* __restrict__ x) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  double s = 0.0;
  for (int k = 0; k < nk; k++) s += y[k] * Z[i + k * ldz];
  x[i] += s;
}

// w = [u; 0] (length n) from u (length P)
__global__ void gm_u0(int64_t P, int64_t n, const double* __restrict__ u, double* __restrict__ w) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) w[i] = i < P ? u[i] : 0.0;
}

// a1 = -w (then + M f by the symmetric product); a2 = f_P + Lw_P
__global__ void gm_neg(int64_t n, const double* __restrict__ w, double* __restrict__ a) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = -w[i];
}
__global__ void gm_a2(int64_t P, const double* __restrict__ f, const double* __restrict__ Lw, double* __restrict__ a2) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P) a2[i] = f[i] + Lw[i];
}

// FP32 vector to FP64
__global__ void gm_f2d(int64_t n, const float* __restrict__ x, double* __restrict__ y) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = (double)x[i];
}

// sum of squares of v[0:len] into out[0] (one block)
__global__ void gm_nrm2(int64_t len, const double* __restrict__ v, double* __restrict__ out) {
  pdl_enter();
  __shared__ double red[256];
  double a = 0.0;
  for (int64_t i = threadIdx.x; i < len; i += 256) a += v[i] * v[i];
  red[threadIdx.x] = a;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

}  // namespace

// The mixed step's solve on M's planes; lub: the sparse FP64 lubrication
// operator (R_lub - R_2B in the grand layout) or null.
// rpp_out (optional): stop once RPP32 = A^-1 + rfu is formed and copy it
// there (6nn x 6nn, ld rpp_ld, full symmetric storage, FP32).
int rsd_mixed_solve(rsd_ctx* ctx, int nn, double* M, int64_t ld, const rsd_lub_sparse* lub, const rsd_step_params* p,
                    const double* ein, const double* Fe, double* U_par, double* S_hyd, rsd_step_info* info, float* rpp_out,
                    int64_t rpp_ld) {
  cudaStream_t s = ctx->stream;
  const int64_t N = nn, n = 11 * N, P = 6 * N, Q = 5 * N;
  mixed_dims d;
  d.P = P;
  d.Q = Q;
  d.n = n;
  // An exported RPP32 carries the rounding of its TF32 factors (1e-4), which
  // moves with the blocks' places: it is formed without the padding, so that
  // the training data of the learned preconditioner stay what they are.
  d.Qp = rpp_out ? Q : (Q + 127) / 128 * 128;
  d.Pp = rpp_out ? P : (P + 3) / 4 * 4;
  d.np = d.Qp + d.Pp;
  const int have_fe = Fe != nullptr;
  const int nr = have_fe ? 2 : 1;
  const double tol = p->tol > 0 ? p->tol : 1e-12;
  const int maxit = p->max_iter > 0 ? p->max_iter : 50;
  // M as FP32 planes hi + lo in the buffer of the FP64 matrix (rsd_ewald_assemble)
  const float* Mh = reinterpret_cast<const float*>(M);
  const float* Ml = Mh + (size_t)ld * n;
  if (ld % 4) return rsd_fail(ctx, RSD_EARG, "mixed solve: the planes' leading dimension must be a multiple of 4");
  const int nbt = (int)((n + SYMV_T - 1) / SYMV_T);
  RSD_TRY(rsd_smem(ctx, symv_planes_part<2>, symv_smem(2)));
  float2* fs = (float2*)rsd_scratch(ctx, "mixed_fs", sizeof(float2) * (size_t)nr * n);
  double* gpart = (double*)rsd_scratch(ctx, "mixed_symv_part", sizeof(double) * 2 * 2 * (size_t)nbt * nbt * SYMV_T);
  if (!fs || !gpart) return RSD_ENOMEM;
  float* M32 = (float*)rsd_scratch(ctx, "mixed_M32", sizeof(float) * d.np * d.np);
  float* A32 = (float*)rsd_scratch(ctx, "mixed_A32", sizeof(float) * d.Pp * d.Pp);
  const size_t nvec = (size_t)nr * (5 * n + 2 * P);
  double* V = (double*)rsd_scratch(ctx, "mixed_vec", sizeof(double) * nvec);
  float* V32 = (float*)rsd_scratch(ctx, "mixed_vec32", sizeof(float) * (size_t)nr * (2 * d.np + 2 * d.Pp));
  if (!M32 || !A32 || !V || !V32) return RSD_ENOMEM;
  double *f = V, *U = f + nr * n, *w = U + nr * P, *r1 = w + nr * n, *Lw = r1 + nr * n, *r2 = Lw + nr * n,
         *y = r2 + nr * P, *nrm = rsd_sums(ctx->d_info);
  float *t32 = V32, *x32 = t32 + nr * d.np, *u32 = x32 + nr * d.np, *du32 = u32 + nr * d.Pp;
  // Status words of the factorisations, read once with the first residual (a
  // failed factor leaves values that nothing branches on): info and timeout
  // of the factor of M', timeout of the inverse, info and timeout of the
  // factor of RPP, timeouts of the block-scaled factors; word 8 is the
  // sweeps' (rsd_uhat_error_flag).
  int* st = ctx->d_info + 16;
  RSD_CUDA(ctx, cudaMemsetAsync(st, 0, sizeof(int) * 9, s));
  info->n_contact = 0;
  // FP32 factor of M' (stresslets first)
  {
    const unsigned nt = (unsigned)((d.np + 31) / 32);
    pdl_launch(convert_perm_half, dim3(nt, nt), dim3(32, 8), 0, s, nn, d, Mh, ld, M32);
  }
  // Tensor-core precision per factor.  The refinement contracts by about the
  // preconditioner's relative error times the condition number it meets:
  // cond(M') is moderate, so TF32 (2^-11) suffices for the factor of M' and
  // for the inverse A^-1 (at N = 2048, phi = 0.5: 7 iterations instead of 6
  // with 3xTF32 there, for half the inverse's time); the factor of RPP meets
  // cond(RPP), which grows like the inverse lubrication gap, and uses 3xTF32
  // (about 2^-21, close to FP32; TF32 there takes ~17 iterations).
  int inf = 0;
  RSD_TRY(rsd_potrf_upper_t<float>(ctx, (int)d.np, M32, d.np, &inf, "m32", ctx->use_tc == 3 ? 3 : 1, st,
                                   rpp_out ? RSD_FACTOR_RPP : RSD_FACTOR_STEP));
  const float* W128 = rsd_potrf_inverses_s(ctx, (int)d.np, "m32");
  float* W_m = nullptr;
  if (!rpp_out) RSD_TRY(rsd_wide_inverses_s(ctx, (int)d.np, M32, d.np, "m32", W128, &W_m));
  // block-scaled factors for one-launch-per-block refinement solves
  rsd_uhat uh_m, uh_r;
  const bool use_uh = ctx->use_tc && !rpp_out;
  if (use_uh) RSD_TRY(rsd_uhat_build(ctx, (int)d.np, M32, d.np, W_m, "m32", &uh_m, st + 5));
  // A^-1 from the trailing factor block, then RPP32 = A^-1 + rfu and its factor
  pdl_launch(copy_block_f, nblk(d.Pp * d.Pp), 256, 0, s, d.Pp, d.Pp, M32 + d.Qp * (d.np + 1), d.np, A32, d.Pp);
  RSD_TRY(rsd_potri_upper_t<float>(ctx, (int)d.Pp, A32, d.Pp, "a32", ctx->use_tc == 3 ? 3 : 1,
                                   rpp_out ? nullptr : W128 + (size_t)(d.Qp / 128) * 128 * 128, st + 2));
  RSD_TRY(rsd_mirror_upper_t<float>(ctx, (int)d.Pp, A32, d.Pp));
  if (lub) RSD_TRY(rsd_lub_add_pp_f32(ctx, lub, A32, d.Pp));
  if (!rpp_out) RSD_TRY(rsd_potrf_upper_t<float>(ctx, (int)d.Pp, A32, d.Pp, &inf, "rpp32", 3, st + 3));
  float* W_r = nullptr;
  if (!rpp_out)
    RSD_TRY(rsd_wide_inverses_s(ctx, (int)d.Pp, A32, d.Pp, "rpp32", rsd_potrf_inverses_s(ctx, (int)d.Pp, "rpp32"), &W_r));
  if (use_uh) RSD_TRY(rsd_uhat_build(ctx, (int)d.Pp, A32, d.Pp, W_r, "rpp32", &uh_r, st + 6));
  // the status words, once the stream has been waited for
  auto status = [&]() -> int {
    const int* h = ctx->h_info + 16;
    info->n_contact = lub ? ctx->h_info[RSD_INFO_CONTACTS] : 0;
    if (h[1]) return rsd_fail(ctx, RSD_ETIMEOUT, "potrf: tensor-core update timed out (code %d)", h[1]);
    if (h[0]) {  // in [Q, P] order without the padding
      info->info = h[0] > d.Qp ? h[0] - (int)(d.Qp - d.Q) : h[0];
      return rsd_fail(ctx, info->info, "FP32 factor of the grand mobility: leading minor %d not positive", info->info);
    }
    if (h[2]) return rsd_fail(ctx, RSD_ETIMEOUT, "potri: tensor-core GEMM timed out (code %d)", h[2]);
    if (h[4]) return rsd_fail(ctx, RSD_ETIMEOUT, "potrf: tensor-core update timed out (code %d)", h[4]);
    if (h[3]) {
      info->info = h[3];
      return rsd_fail(ctx, h[3], "FP32 factor of RPP: leading minor %d not positive", h[3]);
    }
    if (h[5] || h[6]) return rsd_fail(ctx, RSD_ETIMEOUT, "uhat: tensor-core GEMM timed out");
    return RSD_OK;
  };
  // and, in the same copy, the sweeps' error flag and the residual's sums
  const size_t nsum = 2 * (size_t)nr * IT_BLOCKS;
  double* hn = rsd_sums(ctx->h_info);
  auto read_status = [&]() -> int {
    RSD_CUDA(ctx, cudaMemcpyAsync(ctx->h_info + 16, st, sizeof(int) * (RSD_INFO_WORDS - 16) + sizeof(double) * nsum,
                                  cudaMemcpyDeviceToHost, s));
    RSD_CUDA(ctx, cudaStreamSynchronize(s));
    return status();
  };
  if (rpp_out) {
    RSD_CUDA(ctx, cudaMemcpy2DAsync(rpp_out, sizeof(float) * rpp_ld, A32, sizeof(float) * d.Pp, sizeof(float) * P, P,
                                    cudaMemcpyDeviceToDevice, s));
    return read_status();
  }
  // the solves with the two factors: X (overwritten) -> Y
  auto solve_m = [&](float* X, int cols, float* Y, int zero_lead) -> int {
    if (use_uh) return rsd_uhat_solve(ctx, &uh_m, X, d.np, cols, Y, zero_lead);
    return rsd_potrs_wide_s(ctx, (int)d.np, M32, d.np, W_m, X, d.np, cols, Y);
  };
  auto solve_r = [&](float* X, int cols, float* Y) -> int {
    if (use_uh) return rsd_uhat_solve(ctx, &uh_r, X, d.Pp, cols, Y);
    return rsd_potrs_wide_s(ctx, (int)d.Pp, A32, d.Pp, W_r, X, d.Pp, cols, Y);
  };
  // refinement
  const int* tri_err = rsd_uhat_error_flag(ctx);
  // A solve is accepted within the stagnation band of the tolerance, or where its
  // residual is no more than the rounding of its own terms: with a gap of 1e-8
  // L w cancels from 1e8 times the velocities, and no velocities held in FP64
  // leave less of it.
  const double accept = 100.0 * tol;
  // relative residual of column c that the rounding of r2 alone can make up (w
  // and f of that column as they are): the velocities' 2^-53 times |L||w|, about
  // as much from its sum and the terms beside it, and twice that for safety
  auto rounding = [&](int c, double bn, double* out) -> int {
    double* La = (double*)rsd_scratch(ctx, "mixed_la", sizeof(double) * (size_t)(n + IT_BLOCKS));
    if (!La) return RSD_ENOMEM;
    double part[IT_BLOCKS], s2 = 0.0;
    if (lub)
      RSD_TRY(rsd_lub_absmv(ctx, lub, w + (size_t)c * n, La));
    else
      RSD_CUDA(ctx, cudaMemsetAsync(La, 0, sizeof(double) * n, s));
    pdl_launch(it_scale, IT_BLOCKS, 256, 0, s, P, have_fe && c == 0 ? Fe : nullptr, f + (size_t)c * n, La, La + n);
    RSD_CUDA(ctx, cudaMemcpyAsync(part, La + n, sizeof part, cudaMemcpyDeviceToHost, s));
    RSD_CUDA(ctx, cudaStreamSynchronize(s));
    for (int k = 0; k < IT_BLOCKS; k++) s2 += part[k];
    *out = 4.0 * 0x1p-53 * sqrt(s2) / bn;
    return RSD_OK;
  };
  // Right-preconditioned flexible GMRES(m) per right-hand side, FP64
  // residuals; the preconditioner is the stationary iteration's correction.
  // Starts from zero; gm_maxit bounds the iterations over all right-hand
  // sides; returns the iterations, the worst relative residual, and whether
  // every column is accepted.
  auto run_gmres = [&](int gm_maxit, int* its_out, double* res_out, bool* ok) -> int {
    const int m = ctx->gmres_restart > 0 ? ctx->gmres_restart : 30;
    const int64_t len = n + P;
    double* KV = (double*)rsd_scratch(ctx, "gm_basis", sizeof(double) * (size_t)(2 * m + 1) * len + 8 * 64);
    if (!KV) return RSD_ENOMEM;
    double *Vb = KV, *Zb = Vb + (size_t)(m + 1) * len, *dn = Zb + (size_t)m * len;
    double* hacc = (double*)rsd_scratch(ctx, "gm_hacc", sizeof(double) * 64);
    double* hbuf = (double*)rsd_scratch(ctx, "gm_hbuf", sizeof(double) * 64);
    double* Lz = (double*)rsd_scratch(ctx, "gm_lz", sizeof(double) * (size_t)n);
    if (!hacc || !hbuf || !Lz) return RSD_ENOMEM;
    RSD_CUDA(ctx, cudaMemsetAsync(f, 0, sizeof(double) * nr * n, s));
    RSD_CUDA(ctx, cudaMemsetAsync(U, 0, sizeof(double) * nr * P, s));
    double* dv = (double*)rsd_scratch(ctx, "gm_dv", sizeof(double) * (size_t)n);
    if (!dv) return RSD_ENOMEM;
    // the product M v (FP64 v of length n, planes in double-single) into out (added)
    auto symv_add = [&](const double* v, double* out) -> int {
      pdl_launch(to_dsf_vec, nblk(n), 256, 0, s, n, v, fs);
      double* pcol = gpart + (size_t)nbt * nbt * SYMV_T;
      pdl_launch(symv_planes_part<1>, dim3(nbt, nbt), 256, symv_smem(1), s, nn, (int)n, Mh, Ml, ld, fs, nbt, gpart, pcol);
      pdl_launch(symv_planes_reduce, (unsigned)((n + 255) / 256), 256, 0, s, (int)n, 1, nbt, gpart, pcol, 1.0, out, n);
      return RSD_OK;
    };
    // residual of column c: (r1, r2) = b - A x into out (length n + P);
    // Lw (column c) keeps L [U; -EIN] for the stresslet output
    auto residual = [&](int c, double* out) -> int {
      double *fc = f + (size_t)c * n, *Uc = U + (size_t)c * P, *wc = w + (size_t)c * n, *Lc = Lw + (size_t)c * n;
      pdl_launch(build_w, nblk(n), 256, 0, s, P, Q, 1, Uc, ein, wc);
      pdl_launch(gm_neg, nblk(n), 256, 0, s, n, wc, out);
      RSD_TRY(symv_add(fc, out));  // out = M f - w
      pdl_launch(gm_neg, nblk(n), 256, 0, s, n, out, out);  // r1 = w - M f
      if (lub) {
        RSD_TRY(rsd_lub_spmv(ctx, lub, 1, wc, n, Lc, n));
      } else {
        RSD_CUDA(ctx, cudaMemsetAsync(Lc, 0, sizeof(double) * n, s));
      }
      pdl_launch(build_r2, nblk(P), 256, 0, s, P, n, 1, Fe, have_fe && c == 0, fc, Lc, out + n);
      return RSD_OK;
    };
    // z = P v (v, z of length n + P)
    auto precond = [&](const double* v, double* z) -> int {
      pdl_launch(to32_perm, nblk(d.np), 256, 0, s, d, v, t32);
      RSD_TRY(solve_m(t32, 1, x32, 0));
      pdl_launch(it_velocity, nblk(d.np), 256, 0, s, d, 1, x32, v + n, z, u32);  // y = M^-1 v1
      RSD_TRY(solve_r(u32, 1, du32));
      pdl_launch(it_force, nblk(d.np), 256, 0, s, d, 1, du32, t32);
      RSD_TRY(solve_m(t32, 1, x32, (int)d.Qp));
      pdl_launch(from32_add, nblk(d.np), 256, 0, s, d, x32, z);          // df
      pdl_launch(gm_f2d, nblk(P), 256, 0, s, P, du32, z + n);             // dU
      return RSD_OK;
    };
    // a = A z
    auto apply_a = [&](const double* z, double* a) -> int {
      pdl_launch(gm_u0, nblk(n), 256, 0, s, P, n, z + n, dv);  // [zU; 0]
      pdl_launch(gm_neg, nblk(n), 256, 0, s, n, dv, a);
      RSD_TRY(symv_add(z, a));  // M zf - [zU; 0]
      if (lub) {
        RSD_TRY(rsd_lub_spmv(ctx, lub, 1, dv, n, Lz, n));
        pdl_launch(gm_a2, nblk(P), 256, 0, s, P, z, Lz, a + n);
      } else {
        RSD_CUDA(ctx, cudaMemcpyAsync(a + n, z, sizeof(double) * P, cudaMemcpyDeviceToDevice, s));
      }
      return RSD_OK;
    };
    // |b_c|: b = ([0; -EIN], Fe_c)
    std::vector<double> bnorm(nr);
    {
      pdl_launch(it_residual, dim3(IT_BLOCKS, nr), 256, 0, s, d, r1, ein, Fe, have_fe, f, Lw, r2, t32, nrm);  // b part only is used
      RSD_TRY(read_status());
      for (int c = 0; c < nr; c++) {
        double b2 = 0.0;
        for (int k = 0; k < IT_BLOCKS; k++) b2 += hn[2 * (c * IT_BLOCKS + k) + 1];
        bnorm[c] = b2 > 0 ? sqrt(b2) : 1.0;
      }
    }
    int total_it = 0;
    double worst = 0.0;
    std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), g(m + 1), yv(m), hh(m + 2);
    *ok = true;
    for (int c = 0; c < nr; c++) {
      double rel = 0.0, last = 0.0, floor = 0.0;
      for (int cycle = 0;; cycle++) {
        RSD_TRY(residual(c, Vb));
        pdl_launch(gm_nrm2, 1, 256, 0, s, len, Vb, dn);
        double beta2 = 0.0;
        int herr = 0;
        RSD_CUDA(ctx, cudaMemcpyAsync(&beta2, dn, sizeof(double), cudaMemcpyDeviceToHost, s));
        RSD_CUDA(ctx, cudaMemcpyAsync(&herr, tri_err, sizeof(int), cudaMemcpyDeviceToHost, s));
        RSD_CUDA(ctx, cudaStreamSynchronize(s));
        if (herr) return rsd_fail(ctx, RSD_ETIMEOUT, "refinement: a triangular sweep's wait timed out");
        const double beta = sqrt(beta2);
        rel = beta / bnorm[c];
        if (!std::isfinite(rel)) return rsd_fail(ctx, RSD_ENAN, "refinement residual is not finite");
        if (rel <= tol) break;
        const bool spent = total_it >= gm_maxit;
        if (spent || (cycle > 0 && rel > 0.5 * last)) RSD_TRY(rounding(c, bnorm[c], &floor));
        if (spent || rel <= floor) break;
        last = rel;
        pdl_launch(gm_scale, nblk(len), 256, 0, s, len, Vb, dn, Vb);
        std::fill(g.begin(), g.end(), 0.0);
        g[0] = beta;
        int j = 0;
        for (; j < m && total_it < gm_maxit; j++) {
          double* vj = Vb + (size_t)j * len;
          double* zj = Zb + (size_t)j * len;
          double* vn = Vb + (size_t)(j + 1) * len;
          RSD_TRY(precond(vj, zj));
          RSD_TRY(apply_a(zj, vn));
          total_it++;
          // classical Gram-Schmidt, twice
          RSD_CUDA(ctx, cudaMemsetAsync(hacc, 0, sizeof(double) * (j + 1), s));
          for (int pass = 0; pass < 2; pass++) {
            pdl_launch(gm_dots, j + 1, 256, 0, s, len, j + 1, Vb, len, vn, hbuf);
            pdl_launch(gm_orth, nblk(len), 256, 0, s, len, j + 1, Vb, len, hbuf, vn, hacc);
          }
          pdl_launch(gm_nrm2, 1, 256, 0, s, len, vn, dn);
          RSD_CUDA(ctx, cudaMemcpyAsync(hh.data(), hacc, sizeof(double) * (j + 1), cudaMemcpyDeviceToHost, s));
          RSD_CUDA(ctx, cudaMemcpyAsync(hh.data() + j + 1, dn, sizeof(double), cudaMemcpyDeviceToHost, s));
          RSD_CUDA(ctx, cudaStreamSynchronize(s));
          const double hn = sqrt(hh[j + 1]);
          if (hn > 0.0) {
            pdl_launch(gm_scale, nblk(len), 256, 0, s, len, vn, dn, vn);
          }
          // Givens rotations on column j of H
          double* Hj = H.data() + (size_t)j * (m + 1);
          for (int i = 0; i <= j; i++) Hj[i] = hh[i];
          Hj[j + 1] = hn;
          for (int i = 0; i < j; i++) {
            const double t = cs[i] * Hj[i] + sn[i] * Hj[i + 1];
            Hj[i + 1] = -sn[i] * Hj[i] + cs[i] * Hj[i + 1];
            Hj[i] = t;
          }
          const double den = std::hypot(Hj[j], Hj[j + 1]);
          cs[j] = den > 0 ? Hj[j] / den : 1.0;
          sn[j] = den > 0 ? Hj[j + 1] / den : 0.0;
          Hj[j] = den;
          Hj[j + 1] = 0.0;
          g[j + 1] = -sn[j] * g[j];
          g[j] = cs[j] * g[j];
          if (std::fabs(g[j + 1]) <= 0.5 * tol * bnorm[c] || hn == 0.0) {
            j++;
            break;
          }
        }
        // y = H^-1 g (upper triangular, j x j), x += Z y
        for (int i = j - 1; i >= 0; i--) {
          double t = g[i];
          for (int k = i + 1; k < j; k++) t -= H[(size_t)k * (m + 1) + i] * yv[k];
          yv[i] = t / H[(size_t)i * (m + 1) + i];
        }
        RSD_CUDA(ctx, cudaMemcpyAsync(hbuf, yv.data(), sizeof(double) * j, cudaMemcpyHostToDevice, s));
        // x = (f_c, U_c) is not contiguous: update the two parts
        pdl_launch(gm_update, nblk(n), 256, 0, s, n, j, Zb, len, hbuf, f + (size_t)c * n);
        pdl_launch(gm_update, nblk(P), 256, 0, s, P, j, Zb + n, len, hbuf, U + (size_t)c * P);
      }
      worst = fmax(worst, rel);
      *ok = *ok && rel <= fmax(accept, floor);
    }
    *its_out = total_it;
    *res_out = worst;
    return RSD_OK;
  };
  cudaEventRecord(ctx->ev[7], s);
  bool ok = false;
  if (ctx->refine_gmres) {
    int its = 0;
    double res = 0.0;
    RSD_TRY(run_gmres(maxit, &its, &res, &ok));
    pdl_launch(outputs, nblk(P), 256, 0, s, P, Q, nr - 1, f, Lw, U, U_par, S_hyd);
    RSD_CUDA(ctx, cudaGetLastError());
    info->iterations = its;
    info->residual = res;
    if (!ok)
      return rsd_fail(ctx, RSD_ENOCONV, "refinement did not converge: residual %.3e after %d iterations", res, its);
    return RSD_OK;
  }
  RSD_CUDA(ctx, cudaMemsetAsync(f, 0, sizeof(double) * nr * (n + P), s));  // and U, behind it
  double worst = 0.0, best_res = INFINITY;
  int it = 0;
  std::vector<double> hist, rel(nr), bn(nr);
  auto accepted = [&]() -> int {
    ok = worst <= accept;
    if (ok || !std::isfinite(worst)) return RSD_OK;
    ok = true;
    for (int c = 0; c < nr && ok; c++) {
      double floor = 0.0;
      if (rel[c] > accept) RSD_TRY(rounding(c, bn[c], &floor));
      ok = rel[c] <= fmax(accept, floor);
    }
    return RSD_OK;
  };
  for (;; it++) {
    pdl_launch(it_begin, nblk(n * nr), 256, 0, s, P, Q, nr, U, ein, f, w, r1, fs);
    // r1 -= M f, double-single products of the two planes, both right-hand
    // sides in one pass over the stored half of M
    double* pcol = gpart + (size_t)nbt * nbt * SYMV_T * nr;
    if (nr == 2) {
      pdl_launch(symv_planes_part<2>, dim3(nbt, nbt), 256, symv_smem(2), s, nn, (int)n, Mh, Ml, ld, fs, nbt, gpart, pcol);
    } else {
      pdl_launch(symv_planes_part<1>, dim3(nbt, nbt), 256, symv_smem(1), s, nn, (int)n, Mh, Ml, ld, fs, nbt, gpart, pcol);
    }
    pdl_launch(symv_planes_reduce, (unsigned)((n + 255) / 256), 256, 0, s, (int)n, nr, nbt, gpart, pcol, -1.0, r1, n);
    if (lub) {
      RSD_TRY(rsd_lub_spmv(ctx, lub, nr, w, n, Lw, n));
    } else {
      RSD_CUDA(ctx, cudaMemsetAsync(Lw, 0, sizeof(double) * nr * n, s));
    }
    pdl_launch(it_residual, dim3(IT_BLOCKS, nr), 256, 0, s, d, r1, ein, Fe, have_fe, f, Lw, r2, t32, nrm);
    RSD_TRY(read_status());
    if (ctx->h_info[24]) return rsd_fail(ctx, RSD_ETIMEOUT, "refinement: a triangular sweep's wait timed out");
    worst = 0.0;
    for (int c = 0; c < nr; c++) {
      double a2 = 0.0, b2 = 0.0;
      for (int k = 0; k < IT_BLOCKS; k++) {
        a2 += hn[2 * (c * IT_BLOCKS + k)];
        b2 += hn[2 * (c * IT_BLOCKS + k) + 1];
      }
      bn[c] = sqrt(b2) > 0 ? sqrt(b2) : 1.0;
      rel[c] = sqrt(a2) / bn[c];
      worst = std::isfinite(rel[c]) ? fmax(worst, rel[c]) : INFINITY;
    }
    if (worst <= tol || it >= maxit) break;
    // Divergence: FP32 factors too far from the FP64 system (a pair so close
    // that cond(RPP) times the factors' precision exceeds one) make the
    // stationary iteration grow; the flexible GMRES below takes over.
    if (!std::isfinite(worst) || (it >= 2 && worst > 1e3 * best_res)) break;
    best_res = fmin(best_res, worst);
    // Stagnation: the FP64 residual of a stiff system (many near-contact
    // pairs: forces ~1/gap times the velocities) has a floor of about the
    // residual arithmetic's rounding times |M||f| / |b|, which can sit just
    // above tol.  Within 100 tol, or at that floor, an iteration that does not
    // halve the best of the previous two ends the refinement (the solution
    // does not improve further); the reported residual is the one reached.
    hist.push_back(worst);
    if (it >= 2 && worst > 0.5 * fmin(hist[it - 1], hist[it - 2])) {
      RSD_TRY(accepted());
      if (ok) break;
    }
    RSD_TRY(solve_m(t32, nr, x32, 0));  // y = M^-1 r1
    pdl_launch(it_velocity, nblk(d.np * nr), 256, 0, s, d, nr, x32, r2, y, u32);
    RSD_TRY(solve_r(u32, nr, du32));    // dU = RPP^-1 (r2 - y_P)
    pdl_launch(it_force, nblk(d.np * nr), 256, 0, s, d, nr, du32, t32);
    RSD_TRY(solve_m(t32, nr, x32, (int)d.Qp));
    pdl_launch(it_update, nblk(d.np * nr), 256, 0, s, d, nr, x32, y, du32, f, U);  // df = y + M^-1 [dU; 0]
  }
  RSD_TRY(accepted());
  if (!ok) {
    // diverged or stalled above the band: flexible GMRES from zero over the
    // same corrections, which converges where a few modes of the FP32
    // factors are poor
    int its = 0;
    double res = 0.0;
    RSD_TRY(run_gmres(std::max(3 * maxit, 100), &its, &res, &ok));
    it += its;
    worst = res;
    info->fallback = 1;
  }
  pdl_launch(outputs, nblk(P), 256, 0, s, P, Q, nr - 1, f, Lw, U, U_par, S_hyd);
  RSD_CUDA(ctx, cudaGetLastError());
  info->iterations = it;
  info->residual = worst;
  if (!ok)
    return rsd_fail(ctx, RSD_ENOCONV, "refinement did not converge: residual %.3e after %d iterations", worst, it);
  return RSD_OK;
}
