// FP64 grand resistance without the full inverse.  STEPPER_NOGmres
// (src/stepper.f90:348-410) inverts the whole grand mobility (MATREV) but
// needs R_inf = M^-1 only as RPP and as products of RPQ and RQQ with a few
// vectors.  With the stresslets ordered first, M' = [M_QQ M_QP; M_PQ M_PP] =
// U'^T U':
//   (M^-1)_PP      = A^-1 = U_PP^-1 U_PP^-T, A the Schur complement of M_QQ
//   (M^-1)_PQ e    = -A^-1 U_QP^T z,               z = U_QQ^-T e
//   (M^-1)_QP y    = -U_QQ^-1 U_QP A^-1 y
//   (M^-1)_QQ e    = U_QQ^-1 (z + U_QP A^-1 U_QP^T z)
// which takes n^3/3 + 2 (6N)^3/3 = 588 N^3 multiply-adds' worth of flops
// instead of n^3 = 1331 N^3 (n = 11 N).  Q is padded with the identity to a
// multiple of the factorisation's block, so that U_PP's diagonal blocks are
// blocks of U'.
#include <cuda_runtime.h>

#include "pdl.cuh"
#include "rsd_internal.cuh"

template <typename T>
int rsd_gemv(rsd_ctx* ctx, int trans, int m, int k, T alpha, const T* A, int64_t lda, const T* X, int64_t ldx,
             int nrhs, T beta, T* y, int64_t ldy);
int rsd_potri64(rsd_ctx* ctx, int n, double* d_A, int64_t lda, const rsd_factor64& f);
int rsd_potri64_space(rsd_ctx* ctx, int n);
int rsd_potrf64_factor(rsd_ctx* ctx, int n, const char* tag, rsd_factor64* f);
int rsd_trsv64_fwd(rsd_ctx* ctx, int n, const double* U, int64_t ldu, const double* W, double* X, double* Y,
                   int64_t ldx, int nrhs);
int rsd_trsv64_bwd(rsd_ctx* ctx, int n, const double* U, int64_t ldu, const double* W, double* Y, double* X,
                   int64_t ldx, int nrhs);

namespace {

constexpr int R64_BLOCK = 64;

// Upper triangle of M' (stresslets first, padded to Qp) from the upper
// triangle of M in the reference's order, 32 x 32 tiles; the QP block is M's
// PQ block transposed through shared memory.
__global__ void permute_qp(int N, int64_t Qp, int64_t np, const double* __restrict__ M, int64_t ld,
                           double* __restrict__ Mp) {
  pdl_enter();
  __shared__ double T[32][33];
  const int64_t I0 = (int64_t)blockIdx.x * 32, J0 = (int64_t)blockIdx.y * 32, P = 6LL * N, Q = 5LL * N;
  if (I0 > J0) return;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const bool qi = I0 < Qp, qj = J0 < Qp;
  if (qi && !qj) {
    for (int k = ty; k < 32; k += 8) {  // T[k][tx] = M(J0 - Qp + tx, P + I0 + k)
      const int64_t p = J0 - Qp + tx, q = I0 + k;
      T[k][tx] = p < P && q < Q ? M[p + (P + q) * ld] : 0.0;
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8)
      if (I0 + tx < np && J0 + k < np) Mp[I0 + tx + (J0 + k) * np] = T[tx][k];
    return;
  }
  for (int k = ty; k < 32; k += 8) {
    const int64_t i = I0 + tx, j = J0 + k;
    if (i >= np || j >= np) continue;
    double v;
    if (qi)
      v = i < Q && j < Q ? M[P + i + (P + j) * ld] : (i == j ? 1.0 : 0.0);
    else
      v = M[i - Qp + (j - Qp) * ld];
    Mp[i + j * np] = v;
  }
}

__global__ void copy_upper64(int64_t n, const double* __restrict__ S, int64_t lds, double* __restrict__ D) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * n) return;
  const int64_t i = t % n, j = t / n;
  if (i <= j) D[t] = S[i + j * lds];
}

// x = [e; 0] of length Qp
__global__ void pad_q(int64_t Q, int64_t Qp, const double* __restrict__ e, double* __restrict__ x) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < Qp) x[i] = i < Q ? e[i] : 0.0;
}

__global__ void axpy64(int64_t n, double a, const double* __restrict__ x, double* __restrict__ y) {
  pdl_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] += a * x[i];
}

// S(i, r) = -X(i, r), i < Q
__global__ void negate_q(int64_t Q, int64_t Qp, int nr, const double* __restrict__ X, double* __restrict__ S) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < Q * nr) S[t] = -X[t % Q + (t / Q) * Qp];
}

inline unsigned blocks(int64_t n) { return (unsigned)((n + 255) / 256); }

}  // namespace

// Factors M' of the grand mobility in M (the upper triangle of the
// reference's order is read) and forms A^-1 in full, twice: the caller adds the
// lubrication to the one in RPP.  Two cases are left to M itself, factored and
// inverted in place like MATREV; h then holds M^-1 in M, and RPP is its PP block:
// - a matrix within rounding of a singular one, which may have a positive
//   definite factor in the one order only;
// - no memory for M' and the rest (2.6 times that of M, which alone fits the GPU
//   up to N ~ 16000).  The full inverse takes 2.3 times the operations: a step of
//   10000 particles 45 s through the Schur complement, 102 s so; of 16000 390 s.
// A positive info is DPOTRF's on M in the reference's order; M is then overwritten.
int rsd_r64_factor(rsd_ctx* ctx, int nn, double* M, int64_t ld, rsd_r64* h, int* info) {
  const int64_t P = 6LL * nn, Q = 5LL * nn;
  h->P = P;
  h->Q = Q;
  h->Qp = (Q + R64_BLOCK - 1) / R64_BLOCK * R64_BLOCK;
  h->np = h->Qp + P;
  const size_t pp = sizeof(double) * (size_t)P * P;
  h->Mp = (double*)rsd_scratch_try(ctx, "r64_Mp", sizeof(double) * (size_t)h->np * h->np);
  h->Ai = h->Mp ? (double*)rsd_scratch_try(ctx, "r64_Ai", pp) : nullptr;
  h->RPP = h->Ai ? (double*)rsd_scratch_try(ctx, "r64_RPP", pp) : nullptr;
  cudaStream_t s = ctx->stream;
  int inf = 1;
  if (h->RPP && rsd_potri64_space(ctx, (int)P)) {
    const unsigned nt = (unsigned)((h->np + 31) / 32);
    pdl_launch(permute_qp, dim3(nt, nt), dim3(32, 8), 0, s, nn, h->Qp, h->np, M, ld, h->Mp);
    RSD_TRY(rsd_potrf_upper_tag(ctx, (int)h->np, h->Mp, h->np, &inf, "mob"));
  } else {
    for (const char* name : {"r64_Mp", "r64_Ai", "r64_RPP"}) rsd_scratch_free(ctx, name);
  }
  if (inf) {
    RSD_TRY(rsd_potrf_upper_tag(ctx, (int)(P + Q), M, ld, info, "mob"));
    if (*info) return RSD_OK;
    RSD_TRY(rsd_potri_upper_tag(ctx, (int)(P + Q), M, ld, "mob"));
    RSD_TRY(rsd_mirror_upper(ctx, (int)(P + Q), M, ld));
    h->R = h->RPP = M;
    h->ldr = h->ldp = ld;
    return RSD_OK;
  }
  *info = 0;
  RSD_TRY(rsd_potrf64_factor(ctx, (int)h->np, "mob", &h->f));
  pdl_launch(copy_upper64, blocks(P * P), 256, 0, s, P, h->Mp + h->Qp * (h->np + 1), h->np, h->Ai);
  const rsd_factor64 fp{h->f.W + (size_t)(h->Qp / R64_BLOCK) * R64_BLOCK * R64_BLOCK, h->f.dexp + h->Qp};
  RSD_TRY(rsd_potri64(ctx, (int)P, h->Ai, P, fp));
  RSD_TRY(rsd_mirror_upper(ctx, (int)P, h->Ai, P));
  h->ldp = P;
  RSD_CUDA(ctx, cudaMemcpyAsync(h->RPP, h->Ai, pp, cudaMemcpyDeviceToDevice, s));
  return RSD_OK;
}

// f0 = (M^-1)_PQ ein (length P); z = U_QQ^-T ein (length Qp) is kept in h
int rsd_r64_pq(rsd_ctx* ctx, rsd_r64* h, const double* ein, double* f0) {
  if (h->R) {
    h->ein = ein;
    return rsd_gemv<double>(ctx, 0, (int)h->P, (int)h->Q, 1.0, h->R + h->P * h->ldr, h->ldr, ein, h->Q, 1, 0.0, f0, h->P);
  }
  double* w = (double*)rsd_scratch(ctx, "r64_z", sizeof(double) * (size_t)(2 * h->Qp + h->P));
  if (!w) return RSD_ENOMEM;
  h->z = w;
  double *x = w + h->Qp, *v = x + h->Qp;
  pdl_launch(pad_q, blocks(h->Qp), 256, 0, ctx->stream, h->Q, h->Qp, ein, x);
  RSD_TRY(rsd_trsv64_fwd(ctx, (int)h->Qp, h->Mp, h->np, h->f.W, x, h->z, h->Qp, 1));
  RSD_TRY(rsd_gemv<double>(ctx, 1, (int)h->P, (int)h->Qp, 1.0, h->Mp + h->Qp * h->np, h->np, h->z, h->Qp, 1, 0.0, v,
                           h->P));
  return rsd_gemv<double>(ctx, 1, (int)h->P, (int)h->P, -1.0, h->Ai, h->P, v, h->P, 1, 0.0, f0, h->P);
}

// S(:, 0) = (M^-1)_QP Y(:, 0) - (M^-1)_QQ ein, S(:, r) = (M^-1)_QP Y(:, r)
// for r > 0 (ein and f0 of rsd_r64_pq, unchanged since); Y: P x nr, S: Q x nr, nr <= 4
int rsd_r64_stresslet(rsd_ctx* ctx, rsd_r64* h, const double* Y, int nr, const double* f0, double* S) {
  if (h->R) {
    const int P = (int)h->P, Q = (int)h->Q;
    RSD_TRY(rsd_gemv<double>(ctx, 1, Q, P, 1.0, h->R + h->P * h->ldr, h->ldr, Y, P, nr, 0.0, S, Q));
    return rsd_gemv<double>(ctx, 0, Q, Q, -1.0, h->R + h->P * (h->ldr + 1), h->ldr, h->ein, Q, 1, 1.0, S, Q);
  }
  double* w = (double*)rsd_scratch(ctx, "r64_s", sizeof(double) * (size_t)nr * (h->P + 2 * h->Qp));
  if (!w) return RSD_ENOMEM;
  cudaStream_t s = ctx->stream;
  double *u = w + nr * h->P, *x = u + nr * h->Qp;
  RSD_TRY(rsd_gemv<double>(ctx, 1, (int)h->P, (int)h->P, 1.0, h->Ai, h->P, Y, h->P, nr, 0.0, w, h->P));
  pdl_launch(axpy64, blocks(h->P), 256, 0, s, h->P, -1.0, f0, w);
  RSD_TRY(rsd_gemv<double>(ctx, 0, (int)h->Qp, (int)h->P, 1.0, h->Mp + h->Qp * h->np, h->np, w, h->P, nr, 0.0, u,
                           h->Qp));
  pdl_launch(axpy64, blocks(h->Qp), 256, 0, s, h->Qp, 1.0, h->z, u);
  RSD_TRY(rsd_trsv64_bwd(ctx, (int)h->Qp, h->Mp, h->np, h->f.W, u, x, h->Qp, nr));
  pdl_launch(negate_q, blocks(h->Q * nr), 256, 0, s, h->Q, h->Qp, nr, x, S);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}
