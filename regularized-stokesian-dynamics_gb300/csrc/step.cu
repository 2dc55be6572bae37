// The fused step (STEPPER_Stokesian, src/stepper.f90:33-156) on the device:
// lattice -> grand mobility -> R_inf = M^-1 -> R = R_inf + R_lub -> RPP
// factorisation and solves -> velocities, stresslets -> explicit Euler step
// with the Lees-Edwards wrap -> relative viscosity.  Everything stays in HBM;
// the host sees only the lattice (a few scalars) and the outputs it asks for.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "pdl.cuh"
#include "rsd_internal.cuh"

namespace {

__global__ void axpy_block_k(int64_t rows, int64_t cols, double alpha, const double* __restrict__ B, int64_t ldb,
                             double* __restrict__ A, int64_t lda) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= rows * cols) return;
  const int64_t i = t % rows, j = t / rows;
  A[i + j * lda] += alpha * B[i + j * ldb];
}

struct ein5 {
  double v[5];
};
// EIN of every particle, and Fe (zero without d_Fe)
__global__ void fill_inputs(int nn, ein5 e, const double* __restrict__ d_Fe, double* __restrict__ ein,
                            double* __restrict__ Fe) {
  pdl_enter();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 5 * nn) ein[t] = e.v[t % 5];
  if (t < 6 * nn) Fe[t] = d_Fe ? d_Fe[t] : 0.0;
}

// averageU (src/matrices.f90:230-253): U_ave = sum_i (APP F)(3i) / N with
// F(3j) = 6 pi mu_f radii_test; out[0] accumulates sum_ij APP(3i,3j)
// Mh, Ml: the mixed form's M as FP32 planes (hi + lo, the half with row
// particle <= column particle stored); null for FP64 M
__global__ void sum_app_xx(int nn, const double* __restrict__ M, const float* __restrict__ Mh,
                           const float* __restrict__ Ml, int64_t ld, double* __restrict__ out) {
  pdl_enter();
  __shared__ double red[256];
  double s = 0.0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (int64_t)nn * nn;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % nn), j = (int)(t / nn);
    const int64_t o = 3 * i + (int64_t)(3 * j) * ld;
    const int64_t os = 3 * min(i, j) + (int64_t)(3 * max(i, j)) * ld;  // the stored half of the planes
    s += Mh ? (double)Mh[os] + (double)Ml[os] : M[o];
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

struct bg_flow {
  double UOE[9];  // omegaT + Eij (calc_uo_bg, csd_post.f90:507)
  double omega[3];
  double LB[3];
  double T, dt, gamma;
};

__device__ inline void period_correction(double R[3], const bg_flow& f) {
  // PERIOD_CORRECTION (csd_post.f90:65-102), steady shear
  const double lsh = f.LB[2] * f.gamma * f.T;
  if (R[2] > f.LB[2]) {
    R[2] = R[2] - f.LB[2];
    R[0] = fmod(R[0] - lsh, f.LB[0]);
  }
  if (R[2] < 0) {
    R[2] = R[2] + f.LB[2];
    R[0] = fmod(R[0] + lsh, f.LB[0]);
  }
  if (R[0] > f.LB[0])
    R[0] = R[0] - f.LB[0];
  else if (R[0] < 0)
    R[0] = R[0] + f.LB[0];
  if (R[1] > f.LB[1])
    R[1] = R[1] - f.LB[1];
  else if (R[1] < 0)
    R[1] = R[1] + f.LB[1];
}

// STEPPER_conf (stepper.f90:160-227) for the plain-particle case: U_pos =
// U_par + uo_bg(x); x += dt U_pos for i < nn - nb; LE wrap; U_pos recomputed
// with the wrapped positions.
__global__ void euler_update(int nn, int nb, bg_flow f, const double* __restrict__ U_par, double* __restrict__ conf,
                             double* __restrict__ U_pos) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  double x[3] = {conf[3 * i], conf[3 * i + 1], conf[3 * i + 2]};
  double up[3];
  for (int r = 0; r < 3; r++)
    up[r] = U_par[3 * i + r] + (f.UOE[r] * x[0] + f.UOE[r + 3] * x[1] + f.UOE[r + 6] * x[2]);
  if (i < nn - nb)
    for (int r = 0; r < 3; r++) x[r] = x[r] + f.dt * up[r];
  period_correction(x, f);
  for (int r = 0; r < 3; r++) {
    conf[3 * i + r] = x[r];
    U_pos[3 * i + r] = U_par[3 * i + r] + (f.UOE[r] * x[0] + f.UOE[r + 3] * x[1] + f.UOE[r + 6] * x[2]);
    U_pos[3 * nn + 3 * i + r] = U_par[3 * nn + 3 * i + r] + f.omega[r];
  }
}

// yetamu_solve (csd_post.f90:313-367): the three stresslet sums over
// S(5i+3) / (-2 EIN(5i+3))
__global__ void yeta_sums(int nn, const double* __restrict__ Sh, const double* __restrict__ Sfp,
                          const double* __restrict__ Sb, const double* __restrict__ ein, double* __restrict__ out) {
  pdl_enter();
  __shared__ double r0[256], r1[256], r2[256];
  double a = 0, b = 0, c = 0;
  for (int i = threadIdx.x; i < nn; i += blockDim.x) {
    const double d = -2.0 * ein[5 * i + 3];
    const double fp = Sfp ? Sfp[5 * i + 3] : 0.0, bb = Sb ? Sb[5 * i + 3] : 0.0;
    a += (fp + Sh[5 * i + 3] + bb) / d;
    b += bb / d;
    c += fp / d;
  }
  r0[threadIdx.x] = a;
  r1[threadIdx.x] = b;
  r2[threadIdx.x] = c;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (threadIdx.x < d) {
      r0[threadIdx.x] += r0[threadIdx.x + d];
      r1[threadIdx.x] += r1[threadIdx.x + d];
      r2[threadIdx.x] += r2[threadIdx.x + d];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = r0[0];
    out[1] = r1[0];
    out[2] = r2[0];
  }
}

__global__ void nan_check(int64_t n, const double* __restrict__ v, int* __restrict__ flag) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n && !isfinite(v[t])) atomicExch(flag, 1);
}

}  // namespace

int rsd_axpy_block(rsd_ctx* ctx, int64_t rows, int64_t cols, const double* B, int64_t ldb, double* A, int64_t lda,
                   double alpha) {
  const int64_t tot = rows * cols;
  if (tot <= 0) return RSD_OK;
  pdl_launch(axpy_block_k, (unsigned)((tot + 255) / 256), 256, 0, ctx->stream, rows, cols, alpha, B, ldb, A, lda);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// INIT_u_bg (csd_post.f90:442-479) with EI_bg = 0 on input and steady shear:
// Eij(1,3) = Eij(3,1) = gamma/2, omega_bg = (0, gamma/2, 0).
static void background(double gamma, double Eij[9], double omega[3], double UOE[9]) {
  memset(Eij, 0, 9 * sizeof(double));
  Eij[0 + 3 * 2] = Eij[2 + 3 * 0] = gamma * 0.5;
  omega[0] = 0.0;
  omega[1] = gamma * 0.5;
  omega[2] = 0.0;
  auto eps = [](int i, int j, int k) { return (double)((i - j) * (j - k) * (k - i)) / 2.0; };
  for (int I = 0; I < 3; I++)
    for (int J = 0; J < 3; J++) {
      const double om = eps(J, I, 0) * omega[0] + eps(J, I, 1) * omega[1] + eps(J, I, 2) * omega[2];
      UOE[I + 3 * J] = om + Eij[I + 3 * J];
    }
}

static void ei5_of(const double E[9], double out[5]) {
  const double s2 = 1.0 / sqrt(2.0), s6 = 1.0 / sqrt(6.0), s23 = sqrt(2.0 / 3.0);
  double Y[5][9] = {{0}};
  Y[0][0 + 3 * 1] = Y[0][1 + 3 * 0] = s2;
  Y[1][1 + 3 * 2] = Y[1][2 + 3 * 1] = -s2;
  Y[2][0] = Y[2][4] = -s6;
  Y[2][8] = s23;
  Y[3][0 + 3 * 2] = Y[3][2 + 3 * 0] = -s2;
  Y[4][0] = s2;
  Y[4][4] = -s2;
  for (int m = 0; m < 5; m++) {
    double a = 0.0;
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) a = a + E[i + 3 * j] * Y[m][i + 3 * j];
    out[m] = a;
  }
}

int rsd_mixed_solve(rsd_ctx* ctx, int nn, double* M, int64_t ld, const rsd_lub_sparse* lub, const rsd_step_params* p,
                    const double* ein, const double* Fe, double* U_par, double* S_hyd, rsd_step_info* info, float* rpp_out = nullptr,
                    int64_t rpp_ld = 0);
int rsd_lp_pcg_internal(rsd_ctx* ctx, rsd_lp* net, int mode, int nn, const double* d_pos, const double* d_radii,
                        const rsd_lattice* lat, const double* d_rpp, int64_t ld, int nrhs, const double* d_b,
                        double* d_x, double tol, int maxit, int* iters, double* resid);

// What the host entry point adds to the step: its radii, and its results'
// copy into pinned memory before the step's last wait.
struct step_host {
  const double* radii;
  void* dst;
  const void* src;
  size_t bytes;
};

// The step; with rpp_out it stops once RPP = (M^-1)_PP + rfu is formed and
// copies it there (FP64 for the FP64 form, FP32 for the mixed form).
static int step_impl(rsd_ctx* ctx, const rsd_lubtab* tab, const rsd_step_params* p, double* d_conf,
                     const double* d_radii, const double* d_Fe, double* d_U_pos, double* d_SijN, double yeta_mu[5],
                     rsd_step_info* info, void* rpp_out, int64_t rpp_ld, rsd_lattice* lat_out,
                     const step_host* host = nullptr) {
  if (!ctx || !p || !d_conf || !d_radii || (!rpp_out && (!d_U_pos || !d_SijN)) || p->nn < 1 || p->nb < 0 ||
      p->nb > p->nn || !(p->mu_f > 0) || !(p->ews_err > 0) || (p->use_lub && !tab))
    return rsd_fail(ctx, RSD_EARG, "rsd_stepper_stokesian_dev: bad arguments");
  if (p->precision != RSD_PREC_FP64 && p->precision != RSD_PREC_MIXED)
    return rsd_fail(ctx, RSD_EARG, "unknown precision %d", p->precision);
  RSD_TRY(rsd_set_device(ctx));
  cudaStream_t s = ctx->stream;
  const int nn = p->nn;
  const int64_t n = 11LL * nn, P = 6LL * nn, Q = 5LL * nn;
  rsd_step_info loc{};
  // lattice at the start of the step (STEPPER_Stokesian 54-56)
  rsd_lattice lat{};
  RSD_TRY(rsd_set_lattice_skew(p->T, p->LB, p->gamma, 0, 0.0, 0.0, &lat));
  std::vector<double> radii(host ? 0 : nn);
  const double* h_radii = host ? host->radii : radii.data();
  if (!host) {
    RSD_CUDA(ctx, cudaMemcpyAsync(radii.data(), d_radii, nn * sizeof(double), cudaMemcpyDeviceToHost, s));
    RSD_CUDA(ctx, cudaStreamSynchronize(s));
  }
  RSD_TRY(rsd_calc_lattice_inverse(&lat, p->ews_err, nn, h_radii));
  loc.NR = lat.NR;
  loc.NI = lat.NI;
  loc.phi = lat.phi;
  loc.LV = lat.LV;
  if (lat_out) *lat_out = lat;
  // the mixed form's planes have 16-byte aligned columns
  const int64_t ldm = p->precision == RSD_PREC_MIXED ? (n + 3) / 4 * 4 : n;
  double* M = (double*)rsd_scratch(ctx, "step_M", sizeof(double) * ldm * n);
  double* V = (double*)rsd_scratch(ctx, "step_vec", sizeof(double) * (3 * P + 2 * Q));
  if (!M || !V) return RSD_ENOMEM;
  double* X = V;               // P x 2
  double* Upar = V;            // = X(:,0)
  double* ein = V + 2 * P;     // Q
  double* S = ein + Q;         // Q
  double* Fe = S + Q;          // P
  double Eij[9], omega[3], UOE[9];
  ein5 ei5;
  background(p->gamma, Eij, omega, UOE);
  ei5_of(Eij, ei5.v);
  double* sums = rsd_sums(ctx->d_info);
  double* red = sums + 128;    // 256 partial sums, then yeta's three
  pdl_launch(fill_inputs, (unsigned)((P + 255) / 256), 256, 0, s, nn, ei5, d_Fe, ein, Fe);
  cudaEventRecord(ctx->ev[0], s);
  // The lubrication operator needs positions and radii only: it is built on a
  // side stream beside the mobility's pair sums (~190 us of small kernels and
  // one wait of the host at N = 32, ~310 at 512).
  RSD_TRY(rsd_side_stream(ctx));
  rsd_lub_sparse lub;
  rsd_fork beside{ctx, ctx->side2, ctx->ev_la[2], ctx->ev_la[3]};
  if (p->use_lub) {
    RSD_TRY(beside.fork());
    RSD_TRY(rsd_lub_begin(ctx, beside.side, nn, p->nb, 1, d_conf, d_radii, &lat));
  }
  {
    // grand mobility
    rsd_range r("rsd_assembly");
    RSD_TRY(rsd_ewald_assemble(ctx, nn, d_conf, d_radii, &lat, p->mu_f, p->precision, h_radii, M, ldm, rpp_out != nullptr));
    if (p->use_lub)
      RSD_TRY(rsd_lub_build_sparse(ctx, beside.side, tab, nn, p->nb, 1, d_conf, d_radii, &lat, p->mu_f, &lub));
    if (ctx->correction_method) {  // overlap corrections (per_GRPY_YZD.f90:98-116)
      int nov = 0;
      RSD_TRY(rsd_count_overlaps(ctx, nn, d_conf, d_radii, &lat, &nov));
      RSD_TRY(rsd_overlap_correct(ctx, ctx->correction_method, p->precision, nn, d_conf, d_radii, &lat, p->mu_f, nov,
                                  M, ldm));
    }
  }
  cudaEventRecord(ctx->ev[1], s);
  if (p->use_lub) RSD_TRY(beside.join());
  cudaEventRecord(ctx->ev[2], s);
  // averageU on APP before it is overwritten
  const bool planes = p->precision == RSD_PREC_MIXED;
  const float* Mh = planes ? reinterpret_cast<const float*>(M) : nullptr;
  pdl_launch(sum_app_xx, 256, 256, 0, s, nn, M, Mh, planes ? Mh + (size_t)ldm * n : nullptr, ldm, red);
  int info_m = 0;
  if (p->precision == RSD_PREC_FP64) {
    // MobToResist_FTS: R_inf = M^-1 through the Schur complement (resist64.cu)
    rsd_r64 h;
    RSD_TRY(rsd_r64_factor(ctx, nn, M, n, &h, &info_m));
    if (info_m) {
      loc.info = info_m;
      if (info) *info = loc;
      return info_m;
    }
    // arrangResist: RPP = (R_inf)_PP + rfu; the products with rfe and rse
    // come from the sparse lubrication operator (the factor has waited for it)
    if (p->use_lub) loc.n_contact = ctx->h_info[RSD_INFO_CONTACTS];
    double* RPP = h.RPP;
    const int64_t ldp = h.ldp;
    double* f0 = (double*)rsd_scratch(ctx, "step_f0", sizeof(double) * (P + 3 * n));
    if (!f0) return RSD_ENOMEM;
    if (p->use_lub) RSD_TRY(rsd_lub_add_pp_f64(ctx, &lub, RPP, ldp));
    if (rpp_out) {
      RSD_CUDA(ctx, cudaMemcpy2DAsync(rpp_out, sizeof(double) * rpp_ld, RPP, sizeof(double) * ldp, sizeof(double) * P, P,
                                      cudaMemcpyDeviceToDevice, s));
      RSD_CUDA(ctx, cudaStreamSynchronize(s));
      if (info) *info = loc;
      return RSD_OK;
    }
    // RHS [Fe + RPQ EIN, RPQ EIN], RPQ EIN = f0 + rfe EIN
    double *w = f0 + P, *Lw = w + n;  // w = [0; EIN], then [X2; -EIN]; Lw = L w
    RSD_TRY(rsd_r64_pq(ctx, &h, ein, f0));
    RSD_CUDA(ctx, cudaMemcpyAsync(X + P, f0, sizeof(double) * P, cudaMemcpyDeviceToDevice, s));
    if (p->use_lub) {
      RSD_CUDA(ctx, cudaMemsetAsync(w, 0, sizeof(double) * P, s));
      RSD_CUDA(ctx, cudaMemcpyAsync(w + P, ein, sizeof(double) * Q, cudaMemcpyDeviceToDevice, s));
      RSD_TRY(rsd_lub_spmv(ctx, &lub, 1, w, n, Lw, n));
      RSD_TRY(rsd_axpy_block(ctx, P, 1, Lw, P, X + P, P));
    }
    RSD_CUDA(ctx, cudaMemcpyAsync(X, Fe, sizeof(double) * P, cudaMemcpyDeviceToDevice, s));
    RSD_TRY(rsd_axpy_block(ctx, P, 1, X + P, P, X, P));
    bool solved = false;
    if (ctx->rpp_mode != RSD_PC_NONE) {
      // PCG on RPP with the chosen preconditioner; the factorisation stays
      // the fallback when it does not reach the tolerance
      double* B = (double*)rsd_scratch(ctx, "step_rhs", sizeof(double) * 2 * P);
      if (!B) return RSD_ENOMEM;
      RSD_CUDA(ctx, cudaMemcpyAsync(B, X, sizeof(double) * 2 * P, cudaMemcpyDeviceToDevice, s));
      const double tol = ctx->rpp_tol > 0 ? ctx->rpp_tol : 1e-12;
      int it = 0;
      double res = 0.0;
      RSD_TRY(rsd_lp_pcg_internal(ctx, (rsd_lp*)ctx->rpp_net, ctx->rpp_mode, nn, d_conf, d_radii, &lat, RPP, ldp, 2, B, X,
                                  tol, ctx->rpp_maxit > 0 ? ctx->rpp_maxit : 1000, &it, &res));
      loc.rpp_iterations = it;
      if (res <= tol) {
        solved = true;
      } else {
        loc.rpp_iterations = -it;  // did not converge: factorisation below
        RSD_CUDA(ctx, cudaMemcpyAsync(X, B, sizeof(double) * 2 * P, cudaMemcpyDeviceToDevice, s));
      }
    }
    if (!solved) {
      int info_r = 0;
      RSD_TRY(rsd_potrf_upper_tag(ctx, (int)P, RPP, ldp, &info_r, "rpp"));
      if (info_r) {
        loc.info = info_r;
        if (info) *info = loc;
        return info_r;
      }
      RSD_TRY(rsd_potrs_upper_tag(ctx, (int)P, RPP, ldp, X, P, 2, "rpp"));
    }
    // SijN_hyd = RPQ^T RPP^-1 RPQ EIN - RQQ EIN
    RSD_TRY(rsd_r64_stresslet(ctx, &h, X + P, 1, f0, S));
    if (p->use_lub) {
      RSD_CUDA(ctx, cudaMemcpyAsync(w, X + P, sizeof(double) * P, cudaMemcpyDeviceToDevice, s));
      RSD_CUDA(ctx, cudaMemsetAsync(w + P, 0, sizeof(double) * Q, s));
      RSD_TRY(rsd_axpy_block(ctx, Q, 1, ein, Q, w + P, Q, -1.0));
      RSD_TRY(rsd_lub_spmv(ctx, &lub, 1, w, n, Lw, n));
      RSD_TRY(rsd_axpy_block(ctx, Q, 1, Lw + P, Q, S, Q));
    }
    RSD_CUDA(ctx, cudaGetLastError());
  } else {
    {
      rsd_range r("rsd_solve");
      const int rc = rsd_mixed_solve(ctx, nn, M, ldm, p->use_lub ? &lub : nullptr, p, ein, d_Fe ? Fe : nullptr, Upar, S,
                                     &loc, (float*)rpp_out, rpp_ld);
      if (rc != RSD_OK) {
        if (info) *info = loc;
        return rc;
      }
    }
    if (rpp_out) {
      RSD_CUDA(ctx, cudaStreamSynchronize(s));
      if (info) *info = loc;
      return RSD_OK;
    }
    cudaEventRecord(ctx->ev[3], s);
  }
  // velocities, Euler step, LE wrap
  bg_flow f{};
  memcpy(f.UOE, UOE, sizeof UOE);
  memcpy(f.omega, omega, sizeof omega);
  memcpy(f.LB, p->LB, sizeof f.LB);
  f.T = p->T;
  f.dt = p->dt;
  f.gamma = p->gamma;
  pdl_launch(euler_update, (nn + 127) / 128, 128, 0, s, nn, p->nb, f, Upar, d_conf, d_U_pos);
  RSD_CUDA(ctx, cudaMemcpyAsync(d_SijN, S, sizeof(double) * Q, cudaMemcpyDeviceToDevice, s));
  pdl_launch(yeta_sums, 1, 256, 0, s, nn, S, nullptr, nullptr, ein, red + 256);
  int* flag = ctx->d_info + 8;
  RSD_CUDA(ctx, cudaMemsetAsync(flag, 0, sizeof(int), s));
  pdl_launch(nan_check, (unsigned)((6 * nn + 255) / 256), 256, 0, s, 6LL * nn, d_U_pos, flag);
  cudaEventRecord(ctx->ev[5], s);
  // one copy for the status words and the sums, one for a host caller's results
  RSD_CUDA(ctx, cudaMemcpyAsync(ctx->h_info, ctx->d_info, RSD_INFO_BYTES, cudaMemcpyDeviceToHost, s));
  if (host)
    RSD_CUDA(ctx, cudaMemcpyAsync(host->dst, host->src, host->bytes, cudaMemcpyDeviceToHost, s));
  RSD_CUDA(ctx, cudaStreamSynchronize(s));
  const double* hred = rsd_sums(ctx->h_info) + 128;
  const double* ys = hred + 256;
  float t01, t12, t25, t73 = 0.f;  // event 7: factors done, 3: refinement done
  cudaEventElapsedTime(&t01, ctx->ev[0], ctx->ev[1]);
  cudaEventElapsedTime(&t12, ctx->ev[1], ctx->ev[2]);
  cudaEventElapsedTime(&t25, ctx->ev[2], ctx->ev[5]);
  if (p->precision == RSD_PREC_MIXED) cudaEventElapsedTime(&t73, ctx->ev[7], ctx->ev[3]);
  ctx->phase_ms[0] = t01;
  ctx->phase_ms[1] = t12;
  ctx->phase_ms[2] = t25;
  ctx->phase_ms[3] = t73;
  double sxx = 0.0;
  for (int b = 0; b < 256; b++) sxx += hred[b];
  const double f6 = 6.0 * RSD_PI * p->mu_f * 1.0;  // radii_test = 1 after non-dimensionalisation
  const double U_ave = sxx * f6 / nn;
  if (yeta_mu) {
    yeta_mu[0] = ys[0] / lat.LV / p->mu_f;
    yeta_mu[1] = lat.phi;
    yeta_mu[2] = 1.0 / U_ave;
    yeta_mu[3] = ys[1] / lat.LV / p->mu_f;
    yeta_mu[4] = ys[2] / lat.LV / p->mu_f;
  }
  if (info) *info = loc;
  if (ctx->h_info[8]) return rsd_fail(ctx, RSD_ENAN, "non-finite velocity (main.f90:223 NaN check)");
  return RSD_OK;
}

extern "C" int rsd_stepper_stokesian_dev(rsd_ctx* ctx, const rsd_lubtab* tab, const rsd_step_params* p,
                                         double* d_conf, const double* d_radii, const double* d_Fe, double* d_U_pos,
                                         double* d_SijN, double yeta_mu[5], rsd_step_info* info) {
  return step_impl(ctx, tab, p, d_conf, d_radii, d_Fe, d_U_pos, d_SijN, yeta_mu, info, nullptr, 0, nullptr);
}

extern "C" int rsd_resistance_pp_dev(rsd_ctx* ctx, const rsd_lubtab* tab, const rsd_step_params* p,
                                     const double* d_conf, const double* d_radii, void* d_rpp, int64_t ld,
                                     rsd_lattice* lat) {
  if (!ctx || !p || !d_rpp || ld < 6LL * p->nn) return rsd_fail(ctx, RSD_EARG, "rsd_resistance_pp_dev: bad arguments");
  rsd_step_info info{};
  return step_impl(ctx, tab, p, const_cast<double*>(d_conf), d_radii, nullptr, nullptr, nullptr, nullptr, &info, d_rpp,
                   ld, lat);
}

extern "C" int rsd_stepper_stokesian(rsd_ctx* ctx, const rsd_lubtab* tab, const rsd_step_params* p, double* conf,
                                     const double* radii, const double* Fe, double* U_pos, double* SijN,
                                     double yeta_mu[5], rsd_step_info* info) {
  if (!ctx || !p || !conf || !radii || !U_pos || !SijN || p->nn < 1)
    return rsd_fail(ctx, RSD_EARG, "rsd_stepper_stokesian: bad arguments");
  RSD_TRY(rsd_set_device(ctx));
  const int nn = p->nn;
  for (int i = 0; i < 3 * nn; i++)
    if (!std::isfinite(conf[i])) return rsd_fail(ctx, RSD_ENAN, "non-finite position");
  // device [U 6nn | S 5nn | conf 3nn | radii nn | Fe 6nn]: one copy in, one out
  cudaStream_t s = ctx->stream;
  const size_t n1 = (size_t)nn, in = (Fe ? 10 : 4) * n1, out = 14 * n1;
  double* d = (double*)rsd_scratch(ctx, "io_step", sizeof(double) * 21 * n1);
  if (!d) return RSD_ENOMEM;
  RSD_CUDA(ctx, cudaStreamSynchronize(s));  // an earlier call that failed may still use the staging
  double* h = (double*)rsd_pinned(ctx, sizeof(double) * 21 * n1);
  if (!h) return RSD_ENOMEM;
  double *dc = d + 11 * n1, *dr = dc + 3 * n1, *df = Fe ? dr + n1 : nullptr, *hc = h + 11 * n1;
  memcpy(hc, conf, sizeof(double) * 3 * n1);
  memcpy(hc + 3 * n1, radii, sizeof(double) * n1);
  if (Fe) memcpy(hc + 4 * n1, Fe, sizeof(double) * 6 * n1);
  RSD_CUDA(ctx, cudaMemcpyAsync(dc, hc, sizeof(double) * in, cudaMemcpyHostToDevice, s));
  const step_host host{radii, h, d, sizeof(double) * out};
  const int rc = step_impl(ctx, tab, p, dc, dr, df, d, d + 6 * n1, yeta_mu, info, nullptr, 0, nullptr, &host);
  if (rc != RSD_OK) return rc;
  memcpy(U_pos, h, sizeof(double) * 6 * n1);
  memcpy(SijN, h + 6 * n1, sizeof(double) * 5 * n1);
  memcpy(conf, hc, sizeof(double) * 3 * n1);
  return RSD_OK;
}
